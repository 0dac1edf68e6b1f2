"""The tiled soft iterations (one CTA per tile: edges, then tets or bends with the contacts) and the
resident coloured iterations (one CTA for a small scene) against the oracle, at the edges of their
ranges.  Both evaluate the oracle's expressions in its order, so states are equal bit for bit; the bends and
dihedrals go through acos / atan2, which the two sides may round apart: 1e-5, as the golden files."""
import numpy as np
import pytest

import cn_oracle
from cn_physics import Solver, World, scenes, solver_desc

pytestmark = pytest.mark.gpu


def _block(n, compliance=1e-6, pinned=True, seed=0, sp=0.1):
    w = World()
    size = tuple((k - 1.25) * sp for k in n)
    static = [x * n[1] * n[2] + z for x in range(n[0]) for z in range(n[2])] if pinned else []
    w.add_soft_body_grid(size, sp, position=(0.0, size[1] * 0.5 + 0.04, 0.0), radius=0.4 * sp, edge_compliance=1e-5,
                         volume_compliance=compliance, static_particles=static, friction=0.3)
    scenes.ground(w)
    w.soa()
    x = w.positions()
    x[:, :3] += np.random.default_rng(seed).uniform(-2e-3, 2e-3, (len(x), 3)).astype(np.float32) * (x[:, 3:] > 0)
    return w


def _states(w, desc, frames=2, edit=None):
    """States of the two sides; `edit` changes the world's constraints before the second frame."""
    gpu, ora = Solver(desc), cn_oracle.Oracle(desc, w.soa())
    gpu.sync_world(w)
    for k in range(frames):
        if edit is not None and k == 1:
            edit()
            gpu.update_world(w, "constraints")
            ora.update_constraints(w.soa())
        gpu.step(1.0 / 60.0)
        ora.step(1.0 / 60.0)
    return gpu.read_particles(), ora.read_particles()


def _launches(w, desc):
    """Launches of one iteration, by which the path that runs is told: two on tiles (edges, then tets or bends
    with the contacts), four by family, none in the one CTA of a coloured schedule."""
    count = []
    for iterations in (desc.default_iterations, desc.default_iterations + 1):
        d = type(desc).from_buffer_copy(desc)
        d.default_iterations = iterations
        gpu = Solver(d)
        gpu.sync_world(w)
        gpu.step(1.0 / 60.0)
        count.append(gpu.graph_stats()[0])
    return (count[1] - count[0]) // desc.substeps


def _equal(a, b):
    for g, o in zip(*(a, b)):
        assert np.array_equal(np.asarray(g).view(np.uint32), np.asarray(o).view(np.uint32)), float(np.abs(g - o).max())


# one tile; a few; the last size of the small range (3,072); the sizes without tiles next to it and to the first one
# above (6,144); two waves' partial one
@pytest.mark.parametrize("n, launches", [((2, 2, 2), 2), ((5, 4, 3), 2), ((16, 12, 16), 2), ((11, 14, 20), 4), ((17, 19, 19), 4),
                                         ((16, 16, 24), 2), ((18, 18, 19), 2), ((27, 21, 23), 2)])
@pytest.mark.parametrize("pinned", [True, False])
def test_tiles_equal_the_oracle(n, launches, pinned):
    w = _block(n, pinned=pinned)
    desc = solver_desc(substeps=2, default_iterations=5, enable_blocking_readback=0)
    _equal(*_states(w, desc))
    assert _launches(w, desc) == launches


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


# A tet without compliance whose weighted squared gradients are under the bound (1e-6) keeps its last corrections.
# At 5.2 cm and a particle mass of 1 kg they are 0.8e-6 to 2.2e-6, a median of 1e-6: tets go from one side to the other
# (records cleared after the first frame change the oracle's positions by 4 mm).
@pytest.mark.parametrize("schedule", [0, 1, 2])
def test_tets_without_compliance_keep_their_records(schedule):
    w = _block((6, 5, 6), compliance=0.0, pinned=False, sp=0.052)
    desc = solver_desc(substeps=2, default_iterations=4, enable_blocking_readback=0)
    desc.soft.xpbd_schedule = schedule
    _equal(*_states(w, desc, 3))
    assert _launches(w, desc) == (0 if schedule else 2)


# After a frame every tet loses its compliance, at 4 cm and 1 kg under the bound (3e-7 to 8e-7; 3e-6 of scaled
# compliance before): they keep the corrections of the iteration before the change.  And every third edge is switched.
@pytest.mark.parametrize("schedule", [0, 1, 2])
def test_constraints_changed_between_frames(schedule):
    w = _block((6, 5, 6), compliance=2e-10, pinned=False, sp=0.04)

    def edit():
        w.array("tets").view(np.float32)[:, 5] = 0.0
        e = w.array("edges")
        e[::3, 4] = 1 - e[::3, 4]

    desc = solver_desc(substeps=2, default_iterations=4, enable_blocking_readback=0)
    desc.soft.xpbd_schedule = schedule
    _equal(*_states(w, desc, 3, edit))
    assert _launches(w, desc) == (0 if schedule else 2)


def test_disabled_edges_and_a_hub():
    # every particle joined to one: a degree far over the others', and some edges off
    w = _block((6, 6, 6))
    e = w.array("edges")
    e[: len(e) // 3, 0] = 100
    e[::7, 4] = 0
    e[:, 1][e[:, 0] == e[:, 1]] = 101
    desc = solver_desc(substeps=2, default_iterations=4, enable_blocking_readback=0, soft_internal_relaxation=0.02)
    _equal(*_states(w, desc))
    assert _launches(w, desc) == 2


# a particle with more edges than a tile's records hold: the families' own kernels, gathers of four lanes per particle up
# to 32,768 particles and of one above
@pytest.mark.parametrize("n", [(31, 33, 32), (32, 33, 32)])
def test_families_beside_a_hub_over_the_tiles_limit(n):
    w = _block(n)
    e = w.array("edges")
    e[:1100, 0] = 5000
    e[:, 1][e[:, 0] == e[:, 1]] = 5001
    desc = solver_desc(substeps=1, default_iterations=3, enable_blocking_readback=0, soft_internal_relaxation=0.001)
    _equal(*_states(w, desc))
    assert _launches(w, desc) == 4


def test_edges_alone():
    rng = np.random.default_rng(3)
    w = World()
    w.add_soft_body_meshfree(rng.uniform(0.0, 1.0, (400, 3)), 6, position=(0.0, 0.1, 0.0), radius=0.02, edge_compliance=1e-5)
    scenes.ground(w)
    desc = solver_desc(substeps=2, default_iterations=5, enable_blocking_readback=0)
    _equal(*_states(w, desc))
    assert _launches(w, desc) == 2


@pytest.mark.parametrize("resolution", [(7, 5), (90, 80)])
def test_cloth_tiles(resolution):
    w = World()
    w.add_cloth_grid(resolution, (0.02 * resolution[0], 0.02 * resolution[1]), position=(0.0, 0.02, 0.0), radius=0.008,
                     structural_compliance=1e-6, bend_compliance=1e-3, static_particles=[0], friction=0.2)
    scenes.ground(w)
    desc = solver_desc(substeps=2, default_iterations=5, enable_blocking_readback=0)
    for g, o in zip(*_states(w, desc)):
        np.testing.assert_allclose(g, o, rtol=1e-5, atol=1e-5)
    assert _launches(w, desc) == 2


def test_edges_between_tiles_of_tets_and_of_bends():
    # a tile holds particles with tets or particles with bends: these edges have one end in each
    w = _block((6, 5, 6))
    tissue = len(w.positions())
    w.add_cloth_grid((9, 8), (0.4, 0.35), position=(0.0, 0.8, 0.0), radius=0.008, structural_compliance=1e-6, bend_compliance=1e-3,
                     friction=0.2)
    w.soa()
    e = w.array("edges")
    across = np.arange(0, len(e), 40)
    e[across, 0], e[across, 1] = np.arange(len(across)), tissue + np.arange(len(across)) % 72
    e.view(np.float32)[across, 2] = 0.5
    desc = solver_desc(substeps=2, default_iterations=5, enable_blocking_readback=0)
    for g, o in zip(*_states(w, desc)):
        np.testing.assert_allclose(g, o, rtol=1e-5, atol=1e-5)
    assert _launches(w, desc) == 8      # edges, tets, bends (seven by family); five of the contacts between the two bodies


# within one CTA; colours larger than its threads; past its shared memory (a launch per colour)
@pytest.mark.parametrize("schedule", [1, 2])
@pytest.mark.parametrize("n, pinned, resident", [((3, 3, 3), False, True), ((10, 9, 11), True, True), ((13, 13, 13), True, False)])
def test_resident_colours_equal_the_oracle(schedule, n, pinned, resident):
    w = _block(n, pinned=pinned)
    desc = solver_desc(substeps=2, default_iterations=3, enable_blocking_readback=0)
    desc.soft.xpbd_schedule = schedule
    _equal(*_states(w, desc))
    assert (_launches(w, desc) == 0) == resident


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


# a strand and a cloth on the ground within what one CTA does faster than a launch per colour, and over it
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
    for g, o in zip(*_states(w, desc, 1)):
        np.testing.assert_allclose(g, o, rtol=1e-5, atol=1e-5)
    assert (_launches(w, desc) == 0) == resident


@pytest.mark.parametrize("schedule", [1, 2])
def test_resident_colours_with_a_particle_named_twice(schedule):
    w = _block((4, 4, 4), pinned=False)
    w.array("tets")[::5, 3] = w.array("tets")[::5, 1]
    desc = solver_desc(substeps=2, default_iterations=3, enable_blocking_readback=0)
    desc.soft.xpbd_schedule = schedule
    _equal(*_states(w, desc))


def test_rigid_candidates_in_one_block_and_in_launches():
    # 512 particles take one block against any colliders, 720 against up to sixteen; launches are two more
    count = {}
    for n in ((8, 8, 8), (9, 8, 10)):
        for colliders in (15, 40):
            w = _block(n, pinned=False)
            rng = np.random.default_rng(6)
            for k in range(colliders):
                b = w.add_rigid_body("static", position=tuple(float(c) for c in rng.uniform(-0.4, 0.4, 3)))
                w.add_collider(b, ("sphere", "box")[k % 2], ((0.05,), (0.05, 0.05, 0.05))[k % 2])
            desc = solver_desc(substeps=1, default_iterations=3, enable_blocking_readback=0, particle_rigid_pairs_per_particle=32)
            gpu, ora = Solver(desc), cn_oracle.Oracle(desc, w.soa())
            gpu.sync_world(w)
            gpu.step(1.0 / 60.0)
            ora.step(1.0 / 60.0)
            _equal(gpu.read_particles(), ora.read_particles())
            count[n[0], colliders] = gpu.graph_stats()[0]
    assert count[9, 15] == count[8, 15] and count[9, 40] == count[8, 40] + 2
