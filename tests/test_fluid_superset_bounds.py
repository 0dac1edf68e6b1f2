"""Superset lists where particles move far within a substep: the bound on the moves fails, and the iteration
walks the cells or, with two more to come, builds the superset anew.  Lists and states equal the walk of
every cell in every iteration and the oracle, bit for bit."""
import numpy as np
import pytest

import cn_oracle
from cn_physics import Solver, World, scenes, solver_desc

pytestmark = pytest.mark.gpu


# one particle driven into a wall; a corner of them; a share of the whole block; all.  Eight lanes per particle, and
# one; in the later substeps iterations whose new lists did not last are left out.
@pytest.mark.parametrize("share", ["one", "corner", "some", "all"])
@pytest.mark.parametrize("dims, iterations", [((5, 4, 6), 12), ((21, 13, 17), 4), ((21, 13, 17), 9), ((41, 29, 31), 4),
                                              ((41, 29, 31), 9)])
def test_lists_where_some_particles_move_far(dims, iterations, share):
    box = (0.05 * dims[0], 1.0, 0.1 * dims[2])
    w, desc, dt = scenes.dam_break(nx=dims[0], ny=dims[1], nz=dims[2], box=box)
    desc.fluid_iterations = iterations
    x, v = w.positions(), w.velocities()
    rng = np.random.default_rng(1)
    fast = {"one": np.arange(len(x)) == len(x) // 2, "corner": (x[:, 0] < 0.1) & (x[:, 1] < 0.1),
            "some": rng.random(len(x)) < 0.05, "all": np.ones(len(x), bool)}[share]
    v[fast, :3] = rng.normal(0.0, 6.0, (int(fast.sum()), 3)).astype(np.float32)
    _lists_equal_the_walk_and_the_oracle(w, desc, dt)


# a block of a small smoothing radius, pressed to half its spacing, bursts towards a block at rest of three times
# that radius: 7 to 12 mm an iteration, over the one radius's bound (4 mm), under the other's (12 mm), 30 mm in
# all (a list reaches 25 mm past the radius).  Eight lanes per particle, and one.
@pytest.mark.parametrize("n", [5, 33])
@pytest.mark.parametrize("iterations", [4, 6, 16])
def test_lists_of_fluids_with_different_radii(n, iterations):
    w = World()
    sp, s2 = 0.05, 0.5 * 0.05 / 3.0
    for k, spacing, radius, x in ((n, sp, 0.6 * sp, 0.0), (12, s2, 0.2 * sp, n * sp + 0.1)):
        size = k * spacing
        w.add_fluid_grid((size,) * 3, spacing, position=(x + size * 0.5, n * sp * 0.5 + 0.05, n * sp * 0.5), radius=radius, viscosity=0.0)
    scenes.ground(w)
    desc = solver_desc(substeps=1, fluid_iterations=iterations, enable_blocking_readback=0)
    _lists_equal_the_walk_and_the_oracle(w, desc, 1.0 / 240.0, 1)


def _lists_equal_the_walk_and_the_oracle(w, desc, dt, frames=2):
    soa = w.soa()
    got = []
    for walk in (False, True):
        gpu = Solver(desc)
        gpu.set_debug(keep_fluid_delta=True, walk_cells=walk)
        gpu.sync_world(soa)
        for _ in range(frames):
            gpu.step(dt)
        counts = gpu.debug_read("fluid_neighbor_counts").view(np.uint32)
        lists = gpu.debug_read("fluid_neighbors").view(np.uint32).reshape(-1, 128).copy()
        lists[np.arange(128)[None, :] >= counts[:, None]] = 0
        got.append([counts, lists, *gpu.read_particles()])
    ora = cn_oracle.Oracle(desc, soa)
    ora.set_post_update_neighbors(False)
    for _ in range(frames):
        ora.step(dt)
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for a, b in zip(got[0][2:], ora.read_particles()):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
