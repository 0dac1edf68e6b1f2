"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is one scene and one call on it through the public Python package (``cn_physics``):

* ``soft``    -- XPBD tissue blocks (edges + tets) in a ``Solver``: small, ordinary and large, with
                 ground and tool contacts, under the gather and the Gauss-Seidel schedule;
* ``fluid``   -- PBF dam breaks in a ``Solver``: small, ragged with every fluid term, and 1M particles;
* ``cloth``   -- a sheet held at two corners (edges + dihedrals) over the ground;
* ``mixed``   -- the surgical scene: tissue, cloth, strands, fluid, tool, contacts between them, and
                 the render passes;
* ``rigid``   -- a pile of dynamic bodies with proxy-particle tools;
* ``batch``   -- a pool of tissue scenes stepped together for some ticks with a tool target per tick,
                 then read back;
* ``rollout`` -- the differentiable rollout, forward and backward.

A ``Solver`` pass starts an episode from the state the case made (device copies into the exported
buffers, as an environment's reset does) and steps it ``frames`` frames.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch
import torch.utils.checkpoint

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "cressim-neo_b200"))

import cn_physics  # noqa: E402
from cn_physics import Batch, Solver, World, batch_desc, diff, scenes, serving, solver_desc  # noqa: E402

GATHER, GAUSS_SEIDEL = 0, 2


def listed():
    return [
        # the smallest call: one soft cube of 216 particles dropped on the ground, one frame
        {"name": "soft_small_drop", "kind": "soft", "nx": 6, "ny": 6, "nz": 6, "spacing": 0.1, "pinned": False,
         "tool": False, "schedule": GATHER, "substeps": 4, "iterations": 20, "frames": 1},
        # the plain XPBD cube: 16,875 tets, bottom face pinned
        {"name": "soft_cube", "kind": "soft", "nx": 16, "ny": 16, "nz": 16, "spacing": 0.0625, "pinned": True,
         "tool": False, "schedule": GATHER, "substeps": 10, "iterations": 20, "frames": 1},
        # a large tissue (the surgical scene's block, odd sides) pressed by a kinematic capsule
        {"name": "soft_tissue_tool", "kind": "soft", "nx": 61, "ny": 29, "nz": 57, "spacing": 0.02, "pinned": True,
         "tool": True, "schedule": GATHER, "substeps": 4, "iterations": 20, "frames": 1},
        # the coloured Gauss-Seidel schedule, used where the Jacobi update would need more damping
        {"name": "soft_gauss_seidel", "kind": "soft", "nx": 10, "ny": 9, "nz": 11, "spacing": 0.0625, "pinned": True,
         "tool": False, "schedule": GAUSS_SEIDEL, "substeps": 4, "iterations": 10, "frames": 1},
        # a small fluid block: 3,072 particles
        {"name": "fluid_small", "kind": "fluid", "nx": 16, "ny": 12, "nz": 16, "extras": False, "substeps": 2,
         "iterations": 4, "frames": 1},
        # an ordinary fluid with odd sides and every term: cohesion, surface tension, vorticity
        {"name": "fluid_ragged_terms", "kind": "fluid", "nx": 61, "ny": 37, "nz": 53, "extras": True, "substeps": 2,
         "iterations": 4, "frames": 1},
        # the headline dam break: 1,048,576 particles
        {"name": "fluid_dam_break", "kind": "fluid", "nx": 128, "ny": 64, "nz": 128, "extras": False, "substeps": 2,
         "iterations": 4, "frames": 1},
        # a cloth sheet held at two corners over the ground
        {"name": "cloth_sheet", "kind": "cloth", "nx": 129, "ny": 97, "substeps": 4, "iterations": 20, "frames": 1},
        # the mixed surgical scene with its render passes, at its benchmark sizes, two substeps
        {"name": "mixed_surgical", "kind": "mixed", "tissue": 60, "cloth": 256, "strands": 64, "fluid": 64, "substeps": 2,
         "iterations": 20, "frames": 1},
        # 4,096 dynamic bodies in a touching pile, four proxy-particle tools above it
        {"name": "rigid_pile", "kind": "rigid", "layers": 4, "side": 32, "tools": 4, "substeps": 4, "iterations": 10,
         "frames": 1},
        # a pool of tissue scenes (2K to 60K tets each) stepped together: requests of 8 frames
        {"name": "batch_pool", "kind": "batch", "scenes": 96, "least": 2000, "most": 60000, "substeps": 1,
         "iterations": 20, "frames": 8},
        # the differentiable rollout of a 47,385-tet block, forward and adjoint
        {"name": "rollout_grad", "kind": "rollout", "nx": 28, "ny": 14, "nz": 28, "substeps": 8, "iterations": 20,
         "checkpoint": 4},
    ]


def draw(rng):
    """One more case of the same ranges."""
    def lattice(least, most):
        """Three sides whose product is spread over its logarithm."""
        n = math.exp(rng.uniform(math.log(least), math.log(most)))
        a = [rng.uniform(0.7, 1.5) for _ in range(3)]
        f = (n / (a[0] * a[1] * a[2])) ** (1.0 / 3.0)
        return [max(3, int(round(f * r))) for r in a]

    kind = rng.choice(["soft", "soft", "soft", "fluid", "fluid", "cloth", "batch", "rollout", "rigid", "mixed"])
    if kind == "soft":
        gs = rng.random() < 0.25
        nx, ny, nz = lattice(200, 2000 if gs else 110000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "spacing": rng.choice([0.02, 0.0625, 0.1]),
                "pinned": gs or rng.random() < 0.7, "tool": not gs and rng.random() < 0.4,
                "schedule": GAUSS_SEIDEL if gs else GATHER, "substeps": rng.choice([1, 2, 4, 8]),
                "iterations": rng.choice([5, 10, 20]), "frames": 1}
    if kind == "fluid":
        nx, ny, nz = lattice(2000, 900000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "extras": rng.random() < 0.4, "substeps": rng.choice([1, 2]),
                "iterations": rng.choice([2, 3, 4]), "frames": 1}
    if kind == "cloth":
        n = math.exp(rng.uniform(math.log(200), math.log(65536)))
        r = rng.uniform(0.6, 1.6)
        return {"kind": kind, "nx": max(4, int(math.sqrt(n * r))), "ny": max(4, int(math.sqrt(n / r))),
                "substeps": rng.choice([1, 2, 4]), "iterations": rng.choice([10, 20]), "frames": 1}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(8, 64), "least": 1000, "most": rng.choice([8000, 30000, 60000]),
                "substeps": rng.choice([1, 2]), "iterations": rng.choice([10, 20]), "frames": rng.randint(2, 6)}
    if kind == "rollout":
        nx, ny, nz = lattice(500, 9000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "substeps": rng.choice([4, 8]),
                "iterations": rng.choice([5, 10, 20]), "checkpoint": rng.choice([1, 2, 4])}
    if kind == "rigid":
        return {"kind": kind, "layers": rng.randint(1, 4), "side": rng.randint(4, 30), "tools": rng.randint(0, 4),
                "substeps": rng.choice([1, 2, 4]), "iterations": rng.choice([4, 10]), "frames": 1}
    return {"kind": kind, "tissue": rng.randint(8, 50), "cloth": rng.randint(16, 200), "strands": rng.randint(2, 48),
            "fluid": rng.randint(8, 56), "substeps": rng.choice([1, 2]), "iterations": rng.choice([8, 20]), "frames": 1}


# ------------------------------------------------------------------------------------------------
# worlds
# ------------------------------------------------------------------------------------------------
def _soft_world(case, seed):
    """A regular-grid block over the ground: resting with its bottom face pinned, or dropped."""
    w = World()
    n = [case["nx"], case["ny"], case["nz"]]
    sp = case["spacing"]
    size = [(k - 1.25) * sp for k in n]
    r = 0.4 * sp
    pinned = [x * n[1] * n[2] + z for x in range(n[0]) for z in range(n[2])] if case["pinned"] else []
    w.add_soft_body_grid(tuple(size), sp, position=(0.0, size[1] * 0.5 + r + (0.0 if case["pinned"] else 0.003), 0.0),
                         radius=r, edge_compliance=1e-5, volume_compliance=1e-6, static_particles=pinned, friction=0.3)
    scenes.ground(w)
    tool = None
    if case["tool"]:
        tool = w.add_rigid_body("kinematic", position=_tool_pose(case, 0))
        w.add_collider(tool, "capsule", (TOOL_RADIUS, TOOL_HALF), local_orientation=TOOL_TURN, friction=0.2)
    w.soa()
    rng = np.random.default_rng(seed)
    x = w.positions()
    free = x[:, 3] > 0
    x[free, :3] += rng.uniform(-0.02 * sp, 0.02 * sp, (int(free.sum()), 3)).astype(np.float32)
    v = w.velocities()
    v[free, :3] = rng.normal(0.0, 0.02, (int(free.sum()), 3)).astype(np.float32)
    if not case["pinned"]:
        v[free, 1] -= np.float32(0.5)
    return w, tool


TOOL_RADIUS, TOOL_HALF = 0.02, 0.1
TOOL_TURN = (0.0, 0.0, 0.7071068, 0.7071068)


def _tool_pose(case, frame):
    """Hovering 5 mm over the block, then 5 mm into it and sideways."""
    sp = case["spacing"]
    top = (case["ny"] - 1.25) * sp + 2 * 0.4 * sp
    return (0.0, top + TOOL_RADIUS + 0.005, 0.0) if frame == 0 else (0.004, top + TOOL_RADIUS - 0.005, 0.002)


SPACING = 0.05   # of the fluids


def _fluid_world(case, seed):
    """A fluid block in the corner of a box twice as deep, stirred: jittered positions and a smooth
    velocity field, as a dam break some frames after its release."""
    n = (case["nx"], case["ny"], case["nz"])
    kw = {}
    w = World()
    r = 0.6 * SPACING
    size = tuple(k * SPACING for k in n)
    off = r - 0.5 * SPACING
    if case["extras"]:
        kw = dict(cohesion=0.02, surface_tension=0.5, vorticity=0.3)
    w.add_fluid_grid(size, SPACING, position=tuple(s * 0.5 + off for s in size), radius=r, viscosity=0.01, **kw)
    b = w.add_rigid_body("static")
    for half, centre in _walls(case):
        w.add_collider(b, "box", half, centre)
    w.soa()
    rng = np.random.default_rng(seed)
    x, v = w.positions(), w.velocities()
    x[:, :3] += rng.uniform(-0.1 * SPACING, 0.1 * SPACING, (x.shape[0], 3)).astype(np.float32)
    np.maximum(x[:, :3], np.float32(0.9 * r), out=x[:, :3])
    k = rng.uniform(0.5, 2.0, (3, 3)).astype(np.float32)
    ph = rng.uniform(0.0, 6.28, 3).astype(np.float32)
    v[:, :3] = np.float32(0.3) * np.sin(x[:, :3] @ k + ph)
    v[:, 1] -= np.float32(0.5)
    return w


def _walls(case):
    bx, by, bz = case["nx"] * SPACING, case["ny"] * SPACING * 2, case["nz"] * SPACING * 2
    t = 0.5
    return [((bx * 0.5 + 2 * t, t, bz * 0.5 + 2 * t), (bx * 0.5, -t, bz * 0.5)),
            ((t, by * 0.5 + 2 * t, bz * 0.5 + 2 * t), (-t, by * 0.5, bz * 0.5)),
            ((t, by * 0.5 + 2 * t, bz * 0.5 + 2 * t), (bx + t, by * 0.5, bz * 0.5)),
            ((bx * 0.5 + 2 * t, by * 0.5 + 2 * t, t), (bx * 0.5, by * 0.5, -t)),
            ((bx * 0.5 + 2 * t, by * 0.5 + 2 * t, t), (bx * 0.5, by * 0.5, bz + t))]


def _cloth_world(case, seed):
    w = World()
    nx, ny = case["nx"], case["ny"]
    sp = 0.02
    w.add_cloth_grid((nx, ny), ((nx - 1) * sp, (ny - 1) * sp), position=(0.0, 0.05, 0.0), radius=0.008,
                     structural_compliance=1e-6, bend_compliance=1e-3, static_particles=[0, nx - 1], friction=0.3)
    scenes.ground(w)
    w.soa()
    rng = np.random.default_rng(seed)
    x, v = w.positions(), w.velocities()
    free = x[:, 3] > 0
    # a rippled sheet, parts of it at the ground
    ph = rng.uniform(0.0, 6.28, 2)
    x[free, 1] += (0.045 * np.sin(9.0 * x[free, 0] + ph[0]) * np.cos(7.0 * x[free, 2] + ph[1])).astype(np.float32)
    x[free, :3] += rng.uniform(-1e-4, 1e-4, (int(free.sum()), 3)).astype(np.float32)
    v[free, 1] = np.float32(-0.3)
    return w


def _mixed_world(case, seed):
    """The surgical scene with the cloth lowered onto the tissue and the strands onto the cloth, so that the
    contacts between them are there from the first frame."""
    t = case["tissue"]
    out = scenes.mixed_surgical(tissue=(t, max(4, t // 2), t), cloth=(case["cloth"], case["cloth"]),
                                strands=(case["strands"], 129), fluid=(case["fluid"],) * 3, seed=seed)
    w = out[0]
    x = w.positions()
    top = (max(4, t // 2) - 1) * 0.02
    solid = w.array("kinds") == 0
    strand, cloth = solid & (x[:, 1] > top + 0.1), solid & (abs(x[:, 1] - top - 0.05) < 0.01)
    x[strand, 1] -= np.float32(0.12)
    x[cloth, 1] -= np.float32(0.027)
    return out


def _rigid_world(case, seed):
    """Spheres, capsules and boxes in touching layers, falling slowly; proxy-particle tools just above."""
    rng = np.random.default_rng(seed)
    w = World()
    scenes.ground(w)
    pitch, side = 0.081, case["side"]
    half = (side - 1) * pitch * 0.5
    k = 0
    for ly in range(case["layers"]):
        for ix in range(side):
            for iz in range(side):
                p = [ix * pitch - half, 0.0395 + ly * 0.0795, iz * pitch - half]
                p = tuple(float(c + rng.uniform(-0.002, 0.002)) for c in p)
                b = w.add_rigid_body("dynamic", position=p, mass=0.2, inverse_inertia=(400.0,) * 3)
                shape, params = (("sphere", (0.04,)), ("capsule", (0.03, 0.01)), ("box", (0.04, 0.04, 0.04)))[k % 3]
                w.add_collider(b, shape, params, friction=0.5)
                k += 1
    g = (np.arange(3) - 1.0) * 0.04
    points = np.array([(x, y, z) for x in g for y in g for z in g], np.float32)
    for t in range(case["tools"]):
        p = (-half + (t + 0.5) * 2 * half / case["tools"], 0.055 + case["layers"] * 0.0795, 0.0)
        b = w.add_rigid_body("dynamic", position=p, mass=0.5, inverse_inertia=(800.0,) * 3)
        w.set_rigid_proxy_particles(b, points, 0.02, friction=0.5)
    return w


def _pool(case, seed):
    dims = serving.pool_dims(case["scenes"], case["scenes"], (case["least"], case["most"]))
    return [serving.tissue_scene(d, seed=seed * 1009 + k) for k, d in enumerate(dims)]


def _pool_targets(case, seed, pool):
    """Per frame and scene the tool's position: a walk that presses into the tissue and along it."""
    rng = np.random.default_rng(seed + 77)
    p = np.stack([sc.tool_pose for sc in pool]).astype(np.float32)
    out = []
    for _ in range(case["frames"]):
        p = p + rng.normal(0.0, 0.0005, p.shape).astype(np.float32)
        p[:, 1] -= np.float32(0.001)
        out.append(p)
    return np.stack(out)


def _rollout_world(case, seed):
    """A pinned block whose per-tet compliances carry its stiffness."""
    n = (case["nx"], case["ny"], case["nz"])
    sp = 0.1
    w = World()
    size = tuple((k - 1.25) * sp for k in n)
    pinned = [x * n[1] * n[2] + z for x in range(n[0]) for z in range(n[2])]
    w.add_soft_body_grid(size, sp, position=(0.0, size[1] * 0.5, 0.0), radius=0.4 * sp, edge_compliance=1e-4,
                         volume_compliance=1e-11, static_particles=pinned)
    w.soa()
    rng = np.random.default_rng(seed)
    comp = w.array("tets").view(np.float32)[:, 5]
    comp[:] = (1e-11 * rng.lognormal(0.0, 0.5, comp.shape[0])).astype(np.float32)
    x = w.positions()
    free = x[:, 3] > 0
    x[free, :3] += rng.uniform(-0.002, 0.002, (int(free.sum()), 3)).astype(np.float32)
    v = np.zeros((x.shape[0], 4), np.float32)
    v[free, :3] = rng.normal(0.0, 0.05, (int(free.sum()), 3))
    g = np.zeros((x.shape[0], 4), np.float32)
    surf = diff.lattice_surface(n)
    g[surf, :3] = rng.normal(0.0, 1.0 / math.sqrt(len(surf)), (len(surf), 3))
    return w, comp.copy(), v, g


def _soft_desc(case):
    d = solver_desc(substeps=case["substeps"], default_iterations=case["iterations"], enable_blocking_readback=0)
    return d


DT = 1.0 / 60.0


def _frame_dt(case):
    return 1.0 / 120.0 if case["kind"] == "fluid" else DT


# ------------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        pool = _pool(case, seed)
        desc = serving.serving_solver_desc(case["substeps"], case["iterations"])
        c = [sc.world.counts() for sc in pool]
        b = Batch(batch_desc(desc, memory_budget_bytes=64 << 30, max_scenes=len(pool) + 8,
                             particle_capacity=sum(k["particles"] for k in c) + 4096,
                             edge_capacity=sum(k["edges"] for k in c) + 4096,
                             tet_capacity=sum(k["tets"] for k in c) + 4096))
        ids = [b.add_scene(sc.world) for sc in pool]
        return {"case": case, "batch": b, "ids": ids, "tools": [sc.tool for sc in pool],
                "targets": _pool_targets(case, seed, pool).tolist()}
    if kind == "rollout":
        w, comp, v, g = _rollout_world(case, seed)
        r = diff.Rollout(w, substeps=case["substeps"], iterations=case["iterations"], substep_dt=1.0 / 480.0,
                         checkpoint_interval=case["checkpoint"])
        dev = lambda a: torch.as_tensor(np.array(a), device="cuda")  # noqa: E731
        return {"case": case, "rollout": r, "g": dev(g), "comp": dev(comp).requires_grad_(),
                "v": dev(v).requires_grad_(), "x": dev(w.positions()).requires_grad_()}
    tool = None
    if kind == "soft":
        w, tool = _soft_world(case, seed)
        desc = _soft_desc(case)
        desc.soft.xpbd_schedule = case["schedule"]
    elif kind == "fluid":
        w = _fluid_world(case, seed)
        desc = solver_desc(substeps=case["substeps"], fluid_iterations=case["iterations"], enable_blocking_readback=0)
    elif kind == "cloth":
        w, desc = _cloth_world(case, seed), _soft_desc(case)
    elif kind == "mixed":
        w, _, _, tool = _mixed_world(case, seed)
        desc = _soft_desc(case)
    else:
        w, desc = _rigid_world(case, seed), _soft_desc(case)
        desc.particle_rigid_pairs_per_particle = 16
    s = Solver(desc)
    s.sync_world(w)
    st = {"case": case, "world": w, "solver": s, "tool": tool, "out": {}, "first": {}}
    names = ["positions_inv_mass", "velocities"] if w.counts()["particles"] else []
    if kind == "mixed":
        names += ["strand_segment_states"]
        st["target"] = scenes.tool_path(DT, seed)
    elif tool is not None:
        st["target"] = _tool_pose(case, 1)
    for name in names:
        st["out"][name] = s.export_dlpack(name)
        st["first"][name] = st["out"][name].clone()
    if kind == "mixed":
        for name in ("render_positions", "render_normals", "surface_world_aabbs"):
            st["out"][name] = s.export_dlpack(name)
    for view in st["out"].values():
        view.solver = s     # the views last as long as the solver's buffers
    torch.cuda.synchronize()
    return st


def _stream():
    # the C ABI reads 0 as the solver's own stream; the legacy default stream is named by 1
    return torch.cuda.current_stream().cuda_stream or 1


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        for frame in state["targets"]:
            for i, tool, p in zip(state["ids"], state["tools"], frame):
                b.set_kinematic_target(i, tool, p, TOOL_FLAT)
            b.step(state["ids"], DT)
        got = [b.read_particles(i) for i in state["ids"]]
        return {"x": np.concatenate([g[0] for g in got]), "v": np.concatenate([g[1] for g in got])}
    if kind == "rollout":
        out = diff.XPBDRollout.apply(state["comp"], state["v"], state["x"], state["rollout"])
        gc, gv, gx = torch.autograd.grad(out, (state["comp"], state["v"], state["x"]), state["g"])
        return {"x": out.detach(), "grad_compliance": gc, "grad_v": gv, "grad_x": gx}
    s = state["solver"]
    for name, first in state["first"].items():
        state["out"][name].copy_(first)
    if kind == "rigid":
        s.update_world(state["world"], "rigid_bodies")
    if state["tool"] is not None:
        s.set_kinematic_target(state["tool"], state["target"])
    stream = _stream()
    for _ in range(case["frames"]):
        s.step(_frame_dt(case), stream)
    if kind == "rigid":
        return dict(zip(("position", "rotation", "linear", "angular"), s.read_rigid_bodies()), **state["out"])
    return state["out"]


TOOL_FLAT = (0.0, 0.0, 0.0, 1.0)


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _block_counts(nx, ny, nz):
    """Particles, edges and tets of a regular-grid block (5 tets a cell)."""
    cells = (nx - 1) * (ny - 1) * (nz - 1)
    axis = (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)
    faces = nx * (ny - 1) * (nz - 1) + (nx - 1) * ny * (nz - 1) + (nx - 1) * (ny - 1) * nz
    return nx * ny * nz, axis + faces, 5 * cells


EDGE_FLOPS, TET_FLOPS, DIHEDRAL_FLOPS, GATHER_FLOPS = 40, 170, 200, 3
NEIGHBOURS = 30           # of a fluid particle within the smoothing radius
DENSITY_FLOPS, DELTA_FLOPS = 18, 45


def _soft_work(n, e, t, passes):
    return {"bytes": 64 * n + 16 * e + 24 * t, "flops": passes * (e * (EDGE_FLOPS + 2 * GATHER_FLOPS) +
                                                                  t * (TET_FLOPS + 4 * GATHER_FLOPS))}


def _fluid_work(n, substeps, iterations):
    pairs = n * NEIGHBOURS
    return {"bytes": 64 * n, "flops": substeps * iterations * pairs * (DENSITY_FLOPS + DELTA_FLOPS)}


def work(case):
    kind = case["kind"]
    passes = case["substeps"] * case["iterations"] * case.get("frames", 1)
    if kind == "soft":
        return _soft_work(*_block_counts(case["nx"], case["ny"], case["nz"]), passes)
    if kind == "fluid":
        return _fluid_work(case["nx"] * case["ny"] * case["nz"], case["substeps"], case["iterations"])
    if kind == "cloth":
        n, q = case["nx"] * case["ny"], (case["nx"] - 1) * (case["ny"] - 1)
        return {"bytes": 64 * n + 16 * 3 * q + 24 * 3 * q,
                "flops": passes * 3 * q * (EDGE_FLOPS + DIHEDRAL_FLOPS + 6 * GATHER_FLOPS)}
    if kind == "mixed":
        t, q = case["tissue"], (case["cloth"] - 1) ** 2
        a = _soft_work(*_block_counts(t, max(4, t // 2), t), passes)
        f = _fluid_work(case["fluid"] ** 3, case["substeps"], case["iterations"])
        s = case["strands"] * 128
        return {"bytes": a["bytes"] + f["bytes"] + 64 * case["cloth"] ** 2 + 120 * q + 130 * s,
                "flops": a["flops"] + f["flops"] + passes * (3 * q * (EDGE_FLOPS + DIHEDRAL_FLOPS) + s * 500)}
    if kind == "rigid":
        n = case["layers"] * case["side"] ** 2
        pairs = 10 * n            # a body touches some ten others and the ground
        return {"bytes": 2 * 64 * n + 176 * n, "flops": case["substeps"] * pairs * (400 + case["iterations"] * 4 * 120)}
    if kind == "batch":
        b = {"bytes": 0, "flops": 0}
        for d in serving.pool_dims(case["scenes"], case["scenes"], (case["least"], case["most"])):
            a = _soft_work(*_block_counts(*(k + 1 for k in d)), passes)
            b = {k: b[k] + a[k] for k in b}
        return b
    n, e, t = _block_counts(case["nx"], case["ny"], case["nz"])
    a = _soft_work(n, e, t, passes)
    # forward, and the adjoint with its recomputation: the reverse pass of an operation costs about two
    return {"bytes": 112 * n + 16 * e + 28 * t, "flops": 4 * a["flops"]}


def tolerance(case):
    """About four times the relative error measured against ``exact``: 32-bit sums through tens to hundreds
    of iterations of a nonlinear solve, the velocities being position differences over a substep.  In the
    fluids a pair at the very edge of the smoothing radius, or a particle in an edge of the box, changes a
    neighbour count or a wall by its last bit (measured 0.8 % to 2.6 % of the velocities); in the scenes
    without ``exact`` the contacts do the same and are summed by atomics."""
    return {"soft": {"rel": 2e-3, "max": 0.1}, "fluid": {"rel": 3e-2, "max": 0.99}, "cloth": {"rel": 2e-4, "max": 2e-2},
            "mixed": {"rel": 3e-2, "max": 0.99}, "rigid": {"rel": 3e-2, "max": 0.99}, "batch": {"rel": 1.2e-2, "max": 0.5},
            "rollout": {"rel": 6e-3, "max": 0.2}}[case["kind"]]


# ------------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ------------------------------------------------------------------------------------------------
EPS = 1e-6
SLOP, SOFT_RELAX, MAX_CORR, MIN_FRICTION = 1e-3, 0.95, 0.05, 1e-5
RELAX = float(np.float32(0.2))
GRAVITY = -9.81


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.array(a), device=_dev()).to(dtype)


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _edge_terms(p, w, e, rest, alpha, lam):
    """Corrections of the edges' two particles and the new lambdas."""
    a, b = p[e[:, 0]], p[e[:, 1]]
    wa, wb = w[e[:, 0]], w[e[:, 1]]
    d = b - a
    ln = torch.sqrt(_dot(d, d).clamp_min(1e-300))
    ok = ((wa + wb > EPS) & (_dot(d, d) > EPS) & (wa + wb + alpha > EPS)).to(p.dtype)
    dl = -(ln - rest + alpha * lam) / (wa + wb + alpha).clamp_min(1e-300) * ok
    g = d / ln
    return [-wa * dl * g * RELAX, wb * dl * g * RELAX], lam + dl


def _tet_terms(p, w, t, rest, alpha, lam):
    p0, p1, p2, p3 = (p[t[:, k]] for k in range(4))
    cr = torch.linalg.cross
    sv = _dot(cr(p1 - p0, p2 - p0), p3 - p0) / 6.0
    sg = torch.where(sv >= 0, 1.0, -1.0).to(p.dtype) / 6.0
    g = [cr(p3 - p1, p2 - p1) * sg, cr(p2 - p0, p3 - p0) * sg, cr(p3 - p0, p1 - p0) * sg, cr(p1 - p0, p2 - p0) * sg]
    ws = [w[t[:, k]] for k in range(4)]
    den = sum(wk * _dot(gk, gk) for wk, gk in zip(ws, g)) + alpha
    ok = ((sum(ws) > EPS) & (den > EPS)).to(p.dtype)
    dl = -(sv.abs() - rest + alpha * lam) / den.clamp_min(1e-300) * ok
    return [wk * dl * gk * RELAX for wk, gk in zip(ws, g)], lam + dl


def _dihedral_terms(p, w, h, rest, alpha, lam):
    """h: edge particles 0 and 1, opposite particles 0 and 1."""
    p2, p3, p0, p1 = (p[h[:, k]] for k in range(4))
    cr = torch.linalg.cross
    e = p3 - p2
    el = torch.sqrt(_dot(e, e))
    r0, r1 = cr(p2 - p0, p3 - p0), cr(p3 - p1, p2 - p1)
    s0, s1 = _dot(r0, r0), _dot(r1, r1)
    ok = (el * el > EPS) & (s0 > EPS) & (s1 > EPS)
    q0, q1 = r0 / s0, r1 / s1
    g = [-(_dot(p0 - p3, e) / el * q0 + _dot(p1 - p3, e) / el * q1),
         -(_dot(p2 - p0, e) / el * q0 + _dot(p2 - p1, e) / el * q1), -el * q0, -el * q1]
    n0, n1 = r0 / torch.sqrt(s0), r1 / torch.sqrt(s1)
    c = torch.atan2(_dot(e / el, cr(n0, n1)), _dot(n0, n1).clamp(-1.0, 1.0)) - rest
    c = c - 2 * math.pi * torch.floor((c + math.pi) / (2 * math.pi))
    ws = [w[h[:, k]] for k in range(4)]
    den = sum(wk * _dot(gk, gk) for wk, gk in zip(ws, g)) + alpha
    ok = (ok & (den > EPS)).to(p.dtype)
    dl = torch.nan_to_num(-(c + alpha * lam) / den) * ok
    return [torch.nan_to_num(wk * dl * gk * RELAX) for wk, gk in zip(ws, g)], lam + dl


def _summed(p, w, idx, terms):
    total = torch.zeros_like(p)
    for k, c in enumerate(terms):
        total = total.index_add(0, idx[:, k], c)
    return p + total * (w > EPS)


def _colours(idx, n):
    """Greedy colouring, constraints in order: the lowest colour none of their particles' earlier ones holds."""
    used, out = [0] * n, []
    for c in idx.tolist():
        taken = 0
        for p in c:
            taken |= used[p]
        col = 0
        while taken >> col & 1:
            col += 1
        for p in c:
            used[p] |= 1 << col
        out.append(col)
    out = torch.tensor(out, device=idx.device)
    return [torch.nonzero(out == k).reshape(-1) for k in range(int(out.max()) + 1)] if len(out) else []


def _rotate(q, v):
    qv, qw = q[:3].expand_as(v), q[3]
    t = 2.0 * torch.linalg.cross(qv, v)
    return v + qw * t + torch.linalg.cross(qv, t)


def _body_contact(body, p):
    """Normal, signed distance and surface point of each particle against a body at its predicted pose."""
    if body["shape"] == "box":      # axis-aligned, at rest
        l = p - body["at"]
        he = body["half"]
        cl = torch.minimum(torch.maximum(l, -he), he)
        d = l - cl
        dl = torch.sqrt(_dot(d, d))
        ds = he - l.abs()
        k = ds.argmin(-1, keepdim=True)
        nin = torch.zeros_like(l).scatter(-1, k, torch.where(l >= 0, 1.0, -1.0).to(l.dtype).gather(-1, k))
        out = dl > EPS
        n = torch.where(out, d / dl.clamp_min(1e-300), nin)
        sd = torch.where(out, dl, -ds.gather(-1, k))
        face = torch.where(nin != 0, nin * he, l)
        return n, sd, body["at"] + torch.where(out, cl, face)
    a, seg = body["at"] - body["axis"] * body["half"], 2 * body["axis"] * body["half"]
    t = (_dot(p - a, seg) / _dot(seg, seg)).clamp(0.0, 1.0)
    cl = a + seg * t
    d = p - cl
    ln = torch.sqrt(_dot(d, d))
    n = d / ln.clamp_min(1e-300)
    return n, ln - body["radius"], cl + n * body["radius"]


def _contacts(p, prev, w, radius, friction, bodies):
    """One contact iteration; returns the moved positions and the contacts for the velocity pass."""
    total, kept = torch.zeros_like(p), []
    for body in bodies:
        n, sd, cp = _body_contact(body, p)
        pen = radius - sd
        depth = (pen - SLOP).clamp(0.0, MAX_CORR)
        on = (pen > 0) & (w > EPS)
        act = (on & (depth > 0)).to(p.dtype)
        move = n * depth * SOFT_RELAX
        rel = (body["at"] - body["was"]).expand_as(p) - (p - prev)
        tang = rel - n * _dot(rel, n)
        td = torch.sqrt(_dot(tang, tang)).clamp_min(1e-300)
        mu = torch.sqrt(friction * body["friction"])
        fd = torch.where(td <= mu.clamp(0, 1) * depth, tang, tang * (mu.clamp(0, 1) * depth / td).clamp_max(1.0))
        fd = fd * ((td > MIN_FRICTION) & (depth > EPS)).to(p.dtype)
        total = total + (move + fd * SOFT_RELAX) * act
        kept.append((on, n, body))
    return p + total, kept


def _soft_exact(sc, dt, substeps, iterations, schedule=GATHER):
    """Substeps of the soft families and the contacts. `sc`: x, v (N, 3), w (N, 1), the families as
    (indices, rest, compliance, terms), bodies, and per particle radius, friction."""
    x, v, w = sc["x"], sc["v"], sc["w"]
    h = dt / substeps
    free = (w > EPS).to(x.dtype)
    inv = max(h * h, EPS)
    grav = torch.tensor([0.0, GRAVITY, 0.0], device=x.device, dtype=x.dtype)
    fams = [(i, r, c.clamp_min(0.0) / inv, f) for i, r, c, f in sc["families"]]
    cols = [_colours(f[0], len(x)) for f in fams] if schedule == GAUSS_SEIDEL else None
    for sub in range(substeps):
        def substep(x, v, *alphas):
            bodies = []
            for b in sc.get("bodies", []):
                was = b["from"] if sub == 0 else b["to"]
                bodies.append({**b, "was": was, "at": b["to"], "vel": (b["to"] - was) / max(h, EPS)})
            prev = x
            v = (v + grav * h) * free
            x = x + v * h * free
            lams = [torch.zeros_like(f[1]) for f in fams]
            kept = []
            for _ in range(iterations):
                for k, (idx, rest, _, terms) in enumerate(fams):
                    if cols is None:
                        t, lams[k] = terms(x, w, idx, rest, alphas[k], lams[k])
                        x = _summed(x, w, idx, t)
                    else:
                        for col in cols[k]:
                            t, l = terms(x, w, idx[col], rest[col], alphas[k][col], lams[k][col])
                            lams[k][col] = l
                            x = _summed(x, w, idx[col], t)
                if bodies:
                    x, kept = _contacts(x, prev, w, sc["radius"], sc["friction"], bodies)
            v = (x - prev) / h * free
            for _ in range(iterations if kept else 0):
                total = torch.zeros_like(v)
                for on, n, body in kept:
                    nv = _dot(v - body["vel"], n)
                    total = total + n * (-nv).clamp_min(0.0) * on.to(v.dtype)
                v = v + total
            return x, v
        args = (x, v) + tuple(f[2] for f in fams)
        if any(a.requires_grad for a in args):
            x, v = torch.utils.checkpoint.checkpoint(substep, *args, use_reentrant=False)
        else:
            x, v = substep(*args)
    return x, v


def _families(w, offset=0):
    """The world's constraint records as families in the order of an iteration."""
    out = []
    c = w.counts()
    if c["edges"]:
        e = w.array("edges")
        f = e.view(np.float32)
        out.append((_t(e[:, :2].astype(np.int64) + offset, torch.int64), _t(f[:, 2:3]), _t(f[:, 3:4]), _edge_terms))
    if c["dihedrals"]:
        d = w.array("dihedrals")
        f = d.view(np.float32)
        out.append((_t(d[:, :4].astype(np.int64) + offset, torch.int64), _t(f[:, 4:5]), _t(f[:, 5:6]), _dihedral_terms))
    if c["tets"]:
        t = w.array("tets")
        f = t.view(np.float32)
        out.append((_t(t[:, :4].astype(np.int64) + offset, torch.int64), _t(f[:, 4:5]), _t(f[:, 5:6]), _tet_terms))
    return out


GROUND = {"shape": "box", "from": (0.0, -0.5, 0.0), "to": (0.0, -0.5, 0.0), "half": (50.0, 0.5, 50.0), "friction": 0.5}


def _body(b):
    return {k: (_t(np.asarray(v, np.float32)) if not isinstance(v, (str, torch.Tensor)) else v) for k, v in b.items()}


def _capsule(start, target, radius, half, friction):
    axis = _rotate(_t(np.asarray(TOOL_TURN, np.float32)) / math.sqrt(2 * float(np.float32(0.7071068)) ** 2),
                   _t([[0.0, 1.0, 0.0]]))[0]
    return _body({"shape": "capsule", "from": start, "to": target, "radius": radius, "half": half, "axis": axis,
                  "friction": friction})


def _four(p, w):
    return torch.cat([p, w], 1)


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("soft", "cloth"):
            w, tool = _soft_world(case, seed) if kind == "soft" else (_cloth_world(case, seed), None)
            x, v = _t(w.positions()), _t(w.velocities())
            bodies = [_body(GROUND)]
            if tool is not None:
                bodies.insert(0, _capsule(_tool_pose(case, 0), _tool_pose(case, 1), TOOL_RADIUS, TOOL_HALF, 0.2))
            sc = {"x": x[:, :3], "v": v[:, :3], "w": x[:, 3:], "families": _families(w), "bodies": bodies,
                  "radius": _t(w.array("radii"))[:, None], "friction": _t(np.float32(0.3))}
            p, u = _soft_exact(sc, DT, case["substeps"], case["iterations"], case.get("schedule", GATHER))
            return {"positions_inv_mass": _four(p, sc["w"]), "velocities": _four(u, torch.zeros_like(sc["w"]))}
        if kind == "fluid":
            return _fluid_exact(case, seed)
        if kind == "batch":
            return _batch_exact(case, seed)
    if kind == "rollout":
        w, comp, v, g = _rollout_world(case, seed)
        x = _t(w.positions())
        comp, v, p = _t(comp)[:, None].requires_grad_(), _t(v)[:, :3].requires_grad_(), x[:, :3].clone().requires_grad_()
        fams = _families(w)
        fams[-1] = fams[-1][:2] + (comp,) + fams[-1][3:]
        out, _ = _soft_exact({"x": p, "v": v, "w": x[:, 3:], "families": fams}, case["substeps"] / 480.0, case["substeps"],
                             case["iterations"])
        gc, gv, gx = torch.autograd.grad(out, (comp, v, p), _t(g)[:, :3])
        zero = torch.zeros_like(x[:, 3:])
        return {"x": _four(out.detach(), x[:, 3:]), "grad_compliance": gc[:, 0], "grad_v": _four(gv, zero),
                "grad_x": _four(gx, zero)}
    # thousands of bodies or four families with contacts between them, summed in no fixed order: no
    # short restatement
    return None


def _batch_exact(case, seed):
    """The pool as one scene of disjoint blocks, the tools' poses per particle."""
    pool = _pool(case, seed)
    targets = _pool_targets(case, seed, pool)
    xs, vs, radii, fams, owner = [], [], [], None, []
    n = 0
    for k, sc in enumerate(pool):
        w = sc.world
        xs.append(_t(w.positions()))
        vs.append(_t(w.velocities()))
        radii.append(_t(w.array("radii")))
        owner.append(torch.full((len(xs[-1]),), k, device=_dev()))
        f = _families(w, n)
        fams = [[a] for a in f] if fams is None else [a + [b] for a, b in zip(fams, f)]
        n += len(xs[-1])
    fams = [tuple(torch.cat([a[j] for a in fam]) for j in range(3)) + (fam[0][3],) for fam in fams]
    x, v, owner = torch.cat(xs), torch.cat(vs), torch.cat(owner)
    p, u, w = x[:, :3], v[:, :3], x[:, 3:]
    pose = _t(np.stack([sc.tool_pose for sc in pool]))
    for frame in targets:
        to = _t(frame)
        tool = _capsule((0.0, 0.0, 0.0), (0.0, 0.0, 0.0), serving.TOOL_RADIUS, serving.TOOL_HALF_HEIGHT, 0.2)
        tool.update({"from": pose[owner], "to": to[owner]})
        sc = {"x": p, "v": u, "w": w, "families": fams, "bodies": [tool, _body(GROUND)],
              "radius": torch.cat(radii)[:, None], "friction": _t(np.float32(0.3))}
        p, u = _soft_exact(sc, DT, case["substeps"], case["iterations"])
        pose = to
    return {"x": _four(p, w), "v": _four(u, torch.zeros_like(w))}


def _neighbour_pairs(p, h, reach):
    """All ordered pairs (i, j) within `reach` in a CSR over i: (starts, j)."""
    cell = reach
    g = torch.floor((p - p.min(0).values) / cell).long() + 1
    dims = g.max(0).values + 2
    key = (g[:, 0] * dims[1] + g[:, 1]) * dims[2] + g[:, 2]
    order = torch.argsort(key)
    cells = int(dims.prod())
    start = torch.zeros(cells + 1, device=p.device, dtype=torch.int64)
    start[1:] = torch.cumsum(torch.bincount(key, minlength=cells), 0)
    shifts = [(a * int(dims[1]) + b) * int(dims[2]) + c for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
    near_i, near_j = [], []
    for lo in range(0, len(p), 100_000):
        i = torch.arange(lo, min(len(p), lo + 100_000), device=p.device)
        k = key[i][:, None] + torch.tensor(shifts, device=p.device)[None]
        b, c = start[k].reshape(-1), (start[k + 1] - start[k]).reshape(-1)
        ii = i.repeat_interleave(len(shifts)).repeat_interleave(c)
        at = torch.arange(len(ii), device=p.device) - (torch.cumsum(c, 0) - c).repeat_interleave(c)
        jj = order[b.repeat_interleave(c) + at]
        d = p[ii] - p[jj]
        keep = ((d * d).sum(-1) < reach * reach) & (ii != jj)
        near_i.append(ii[keep].int())
        near_j.append(jj[keep].int())
    i, j = torch.cat(near_i), torch.cat(near_j)
    return i, j


def _wall(p, wall):
    """Normal and signed distance to an axis-aligned box."""
    half, at = (_t(np.asarray(k, np.float32)) for k in wall)
    n, sd, _ = _body_contact({"shape": "box", "at": at, "half": half}, p)
    return n, sd


def _fluid_exact(case, seed):
    w = _fluid_world(case, seed)
    m = w.fluid_materials()[0].astype(np.float64)
    rho0, h, cscale, visc, coh, coh1, coh2, st, vort, gs, cfl = (float(m[k]) for k in (0, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11))
    x = _t(w.positions())
    v = _t(w.velocities())[:, :3]
    iw, x = x[:, 3:], x[:, :3]
    dt = 1.0 / 120.0 / case["substeps"]
    radius = float(np.float32(0.6 * SPACING))
    kw = 15.0 / (math.pi * h ** 3)
    walls = _walls(case)
    solve, ghost_density, ghost_delta = (float(np.float32(k)) for k in (0.7, 0.12, 0.08))
    chunk = 6_000_000

    def over_pairs(i, j, q, f, width, total=None):
        """Sum over the pairs within h of f(i, j, delta, d) at the first of the two."""
        out = torch.zeros((len(q), width), device=q.device, dtype=q.dtype)
        for lo in range(0, len(i), chunk):
            a, b = i[lo:lo + chunk].long(), j[lo:lo + chunk].long()
            d = q[a] - q[b]
            r = torch.sqrt((d * d).sum(-1, keepdim=True))
            keep = (r < h)[:, 0]
            a, b, d, r = a[keep], b[keep], d[keep], r[keep]
            out.index_add_(0, a, f(a, b, d, r))
        return out

    def ghosts(q):
        for wall in walls:
            n, sd = _wall(q, wall)
            g = n * 2.0 * sd
            r = 2.0 * sd
            on = (sd >= 0) & (sd < h) & (r < h)
            yield on.to(q.dtype), g, r

    for _ in range(case["substeps"]):
        prev = x
        v = v + torch.tensor([0.0, GRAVITY, 0.0], device=x.device, dtype=x.dtype) * dt * gs
        x = x + v * dt
        pi, pj = _neighbour_pairs(x, h, 1.4 * h)
        acc = torch.zeros_like(x)
        for it in range(case["iterations"]):
            q = x + acc

            def density(a, b, d, r):
                om = 1.0 - r / h
                grad = torch.where(r > EPS, -2.0 * kw * om / h * d / r.clamp_min(1e-300), 0.0)
                return torch.cat([kw * om * om, grad], 1)
            s = over_pairs(pi, pj, q, density, 4)
            rho, nrm = s[:, :1], s[:, 1:] * st
            for on, _, r in ghosts(q):
                rho = rho + on * kw * (1.0 - r / h) ** 2 * ghost_density
            con = (rho - rho0).clamp_min(0.0) * cscale

            def delta(a, b, d, r):
                nij = d / r.clamp_min(1e-300)
                om = 1.0 - r / h
                out = -0.5 * (con[a] + con[b]) * (-2.0 * kw * om / h) * nij
                if dt * coh > EPS:
                    z = r / h
                    out = out - nij * dt * coh * (coh1 * z ** 3 + coh2 * z * z - 1.0)
                rel = acc[a] - acc[b]
                if dt * visc > EPS:
                    out = out - (1.0 - 1.0 / (1.0 + dt * visc * kw * om * om)) * rel
                if cfl > EPS:
                    pr = _dot(rel, nij)
                    out = out - nij * (pr + cfl).clamp_max(0.0) * 0.5
                if st > EPS:
                    out = out - dt * (nrm[a] - nrm[b])
                on = (r > EPS).to(q.dtype)
                return torch.cat([out * on, on], 1)
            s = over_pairs(pi, pj, q, delta, 4)
            packed = s[:, :3] * solve
            for on, g, r in ghosts(q):
                on = on * (r > EPS)
                packed = packed + ghost_delta * on * con * 2.0 * kw * (1.0 - r / h) / h * g / r.clamp_min(1e-300)
            cur = x + acc + packed / s[:, 3:].clamp_min(1.0)
            for _ in range(2):
                for wall in walls:
                    n, sd = _wall(cur, wall)
                    cur = cur + n * (radius - sd).clamp_min(0.0)
            acc = cur - x
        x = x + acc
        v = (x - prev) / dt
        best = torch.full_like(iw, math.inf)
        bn = torch.zeros_like(x)
        for wall in walls:
            n, sd = _wall(x, wall)
            near = (sd <= radius + 2 * SLOP) & (sd < best)
            best, bn = torch.where(near, sd, best), torch.where(near, n, bn)
        hit = torch.isfinite(best)
        best = torch.where(hit, best, torch.zeros_like(best))
        # the fluid's own friction is zero, so the combined friction is
        u = v - bn * _dot(v, bn).clamp_max(0.0)
        v = torch.where(hit, u, v)
        if vort > EPS:
            q = x
            pi, pj = _neighbour_pairs(q, h, h * 1.01)

            def grad(d, r):
                return torch.where(r > EPS, -2.0 * kw * (1.0 - r / h) / h * d / r.clamp_min(1e-300), 0.0)
            curl = over_pairs(pi, pj, q, lambda a, b, d, r: torch.linalg.cross(v[b] - v[a], grad(d, r)), 3)
            mag = torch.sqrt(_dot(curl, curl))
            g = over_pairs(pi, pj, q, lambda a, b, d, r: mag[b] * grad(d, r), 3)
            gl = torch.sqrt(_dot(g, g))
            f = vort * torch.linalg.cross(g / gl.clamp_min(1e-300), curl)
            v = v + dt * f * ((gl > EPS) & (mag > EPS)).to(x.dtype)
    return {"positions_inv_mass": _four(x, iw), "velocities": _four(v, torch.zeros_like(iw))}
