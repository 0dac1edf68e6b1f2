"""The tiled soft iterations (one CTA per tile: edges, then tets or bends with the contacts) and the
resident coloured iterations (one CTA for a small scene) against the oracle, at the edges of their
ranges.  Both evaluate the oracle's expressions in its order, so states are equal bit for bit; the bends and
dihedrals go through acos / atan2, which the two sides may round apart: 1e-5, as the golden files."""
import numpy as np
import pytest

import cn_oracle
from cn_physics import Solver, World, scenes, solver_desc

pytestmark = pytest.mark.gpu


def _block(n, compliance=1e-6, pinned=True, seed=0):
    w = World()
    sp = 0.1
    size = tuple((k - 1.25) * sp for k in n)
    static = [x * n[1] * n[2] + z for x in range(n[0]) for z in range(n[2])] if pinned else []
    w.add_soft_body_grid(size, sp, position=(0.0, size[1] * 0.5 + 0.04, 0.0), radius=0.04, edge_compliance=1e-5,
                         volume_compliance=compliance, static_particles=static, friction=0.3)
    scenes.ground(w)
    w.soa()
    x = w.positions()
    x[:, :3] += np.random.default_rng(seed).uniform(-2e-3, 2e-3, (len(x), 3)).astype(np.float32) * (x[:, 3:] > 0)
    return w


def _states(w, desc, frames=2, edit=None):
    gpu, ora = Solver(desc), cn_oracle.Oracle(desc, w.soa())
    gpu.sync_world(w)
    for k in range(frames):
        if edit is not None and k == 1:
            edit(gpu, ora)
        gpu.step(1.0 / 60.0)
        ora.step(1.0 / 60.0)
    return gpu.read_particles(), ora.read_particles()


def _equal(a, b):
    for g, o in zip(*(a, b)):
        assert np.array_equal(np.asarray(g).view(np.uint32), np.asarray(o).view(np.uint32)), float(np.abs(g - o).max())


# one tile; a few; the last size of the small range; the first tiled one above it; two waves' partial one
@pytest.mark.parametrize("n", [(2, 2, 2), (5, 4, 3), (16, 12, 16), (18, 18, 19), (27, 21, 23)])
@pytest.mark.parametrize("pinned", [True, False])
def test_tiles_equal_the_oracle(n, pinned):
    w = _block(n, pinned=pinned)
    desc = solver_desc(substeps=2, default_iterations=5, enable_blocking_readback=0)
    _equal(*_states(w, desc))


def test_tiles_are_sized_by_the_particles_in_them():
    # 1,000 particles of tissue have tiles, two launches an iteration, beside 1,400 of fluid and beside 2,688
    # (whose world is of a size that alone would have none)
    launches = []
    for fluid in ((10, 10, 14), (12, 14, 16)):
        w = _block((10, 10, 10))
        size = tuple(0.05 * k for k in fluid)
        w.add_fluid_grid(size, 0.05, position=(5.0, size[1] * 0.5 + 0.01, 0.0), radius=0.03)
        desc = solver_desc(substeps=1, default_iterations=5, enable_blocking_readback=0)
        gpu, ora = Solver(desc), cn_oracle.Oracle(desc, w.soa())
        gpu.sync_world(w)
        gpu.step(1.0 / 60.0)
        ora.step(1.0 / 60.0)
        _equal(gpu.read_particles(), ora.read_particles())
        launches.append(gpu.graph_stats()[0])
    assert launches[0] == launches[1]


def test_tets_without_compliance_keep_their_records():
    # 10 cm tets: the weighted squared gradients (~1e-5) are above the degenerate bound; flattened ones are not
    w = _block((6, 5, 6), compliance=0.0, pinned=False)
    x = w.positions()
    x[x[:, 0] > 0.1, 1] *= np.float32(1e-3)
    desc = solver_desc(substeps=2, default_iterations=4, enable_blocking_readback=0)
    _equal(*_states(w, desc, 3))


def test_disabled_edges_and_a_hub():
    # every particle joined to one: a degree far over the others', and some edges off
    w = _block((6, 6, 6))
    e = w.array("edges")
    e[: len(e) // 3, 0] = 100
    e[::7, 4] = 0
    e[:, 1][e[:, 0] == e[:, 1]] = 101
    desc = solver_desc(substeps=2, default_iterations=4, enable_blocking_readback=0, soft_internal_relaxation=0.02)
    _equal(*_states(w, desc))


def test_edges_alone():
    rng = np.random.default_rng(3)
    w = World()
    w.add_soft_body_meshfree(rng.uniform(0.0, 1.0, (400, 3)), 6, position=(0.0, 0.1, 0.0), radius=0.02, edge_compliance=1e-5)
    scenes.ground(w)
    desc = solver_desc(substeps=2, default_iterations=5, enable_blocking_readback=0)
    _equal(*_states(w, desc))


@pytest.mark.parametrize("resolution", [(7, 5), (90, 80)])
def test_cloth_tiles(resolution):
    w = World()
    w.add_cloth_grid(resolution, (0.02 * resolution[0], 0.02 * resolution[1]), position=(0.0, 0.02, 0.0), radius=0.008,
                     structural_compliance=1e-6, bend_compliance=1e-3, static_particles=[0], friction=0.2)
    scenes.ground(w)
    desc = solver_desc(substeps=2, default_iterations=5, enable_blocking_readback=0)
    for g, o in zip(*_states(w, desc)):
        np.testing.assert_allclose(g, o, rtol=1e-5, atol=1e-5)


# within one CTA; colours larger than its threads; past its shared memory (a launch per colour)
@pytest.mark.parametrize("schedule", [1, 2])
@pytest.mark.parametrize("n, pinned", [((3, 3, 3), False), ((10, 9, 11), True), ((13, 13, 13), True)])
def test_resident_colours_equal_the_oracle(schedule, n, pinned):
    w = _block(n, pinned=pinned)
    desc = solver_desc(substeps=2, default_iterations=3, enable_blocking_readback=0)
    desc.soft.xpbd_schedule = schedule
    _equal(*_states(w, desc))


def test_restitution_after_the_iterations():
    # fast contacts that bounce: the velocity pass keeps its contacts in registers over the iterations
    w = World()
    w.add_soft_body_grid((0.3, 0.3, 0.3), 0.1, position=(0.0, 0.25, 0.0), radius=0.05, edge_compliance=1e-5,
                         volume_compliance=1e-6, restitution=0.6, friction=0.3)
    scenes.ground(w)
    b = w.add_rigid_body("static", position=(0.1, 0.0, 0.0))
    w.add_collider(b, "sphere", (0.1,), restitution=0.5)
    c = w.add_rigid_body("static", position=(-0.1, 0.02, 0.0))
    w.add_collider(c, "capsule", (0.05, 0.05), restitution=0.5)
    w.soa()
    w.velocities()[:, 1] = np.float32(-3.0)
    desc = solver_desc(substeps=2, default_iterations=6, enable_blocking_readback=0)
    _equal(*_states(w, desc, 4))


# a strand and a cloth on the ground within what one CTA does faster than a launch per colour, and over it; a
# launch per colour makes 10 iterations of 6 (20) colours
@pytest.mark.parametrize("schedule", [1, 2])
@pytest.mark.parametrize("kind, n, resident", [("strand", 600, True), ("strand", 2000, False), ("cloth", 30, True),
                                               ("cloth", 40, False)])
def test_resident_colours_stop_where_launches_are_faster(schedule, kind, n, resident):
    w = World()
    if kind == "strand":
        w.add_strand([(0.0, 0.02, 0.02 * k) for k in range(n)], radius=0.01, stretch_shear_compliance=1e-6, bend_compliance=1e-4,
                     twist_compliance=1e-4, static_particles=[0])
    else:
        w.add_cloth_grid((n, n), (0.02 * n, 0.02 * n), position=(0.0, 0.01, 0.0), radius=0.008, structural_compliance=1e-6,
                         bend_compliance=1e-3, static_particles=[0], friction=0.2)
    scenes.ground(w)
    desc = solver_desc(substeps=1, default_iterations=10, enable_blocking_readback=0)
    desc.soft.xpbd_schedule = schedule
    gpu, ora = Solver(desc), cn_oracle.Oracle(desc, w.soa())
    gpu.sync_world(w)
    gpu.step(1.0 / 60.0)
    ora.step(1.0 / 60.0)
    assert (gpu.graph_stats()[0] < 20) == resident
    for g, o in zip(gpu.read_particles(), ora.read_particles()):
        np.testing.assert_allclose(g, o, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("schedule", [1, 2])
def test_resident_colours_with_a_particle_named_twice(schedule):
    w = _block((4, 4, 4), pinned=False)
    w.array("tets")[::5, 3] = w.array("tets")[::5, 1]
    desc = solver_desc(substeps=2, default_iterations=3, enable_blocking_readback=0)
    desc.soft.xpbd_schedule = schedule
    _equal(*_states(w, desc))
