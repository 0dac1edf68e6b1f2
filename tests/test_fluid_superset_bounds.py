"""Superset lists where particles move far within a substep: the bound on the moves fails, and the iteration
walks the cells and, with two more to come, builds the superset anew.  Lists and states equal the walk of
every cell in every iteration and the oracle, bit for bit."""
import numpy as np
import pytest

import cn_oracle
from cn_physics import Solver, scenes

pytestmark = pytest.mark.gpu


# one particle driven into a wall; a corner of them; a share of the whole block; all
@pytest.mark.parametrize("share", ["one", "corner", "some", "all"])
@pytest.mark.parametrize("dims, iterations", [((5, 4, 6), 12), ((21, 13, 17), 4), ((21, 13, 17), 9)])
def test_lists_where_some_particles_move_far(dims, iterations, share):
    box = (0.05 * dims[0], 1.0, 0.1 * dims[2])
    w, desc, dt = scenes.dam_break(nx=dims[0], ny=dims[1], nz=dims[2], box=box)
    desc.fluid_iterations = iterations
    x, v = w.positions(), w.velocities()
    rng = np.random.default_rng(1)
    fast = {"one": np.arange(len(x)) == len(x) // 2, "corner": (x[:, 0] < 0.1) & (x[:, 1] < 0.1),
            "some": rng.random(len(x)) < 0.05, "all": np.ones(len(x), bool)}[share]
    v[fast, :3] = rng.normal(0.0, 6.0, (int(fast.sum()), 3)).astype(np.float32)
    soa = w.soa()
    got = []
    for walk in (False, True):
        gpu = Solver(desc)
        gpu.set_debug(keep_fluid_delta=True, walk_cells=walk)
        gpu.sync_world(soa)
        for _ in range(2):
            gpu.step(dt)
        counts = gpu.debug_read("fluid_neighbor_counts").view(np.uint32)
        lists = gpu.debug_read("fluid_neighbors").view(np.uint32).reshape(-1, 128).copy()
        lists[np.arange(128)[None, :] >= counts[:, None]] = 0
        got.append([counts, lists, *gpu.read_particles()])
    ora = cn_oracle.Oracle(desc, soa)
    ora.set_post_update_neighbors(False)
    for _ in range(2):
        ora.step(dt)
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for a, b in zip(got[0][2:], ora.read_particles()):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
