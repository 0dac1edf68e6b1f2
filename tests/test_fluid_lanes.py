"""Fluid kernels with eight lanes per particle and with one, on both sides of the sizes where the one takes over:
each evaluates the oracle's expressions in its order, so states are equal bit for bit."""
import numpy as np
import pytest

import cn_oracle
from cn_physics import Solver, World, scenes, solver_desc

pytestmark = pytest.mark.gpu


# 22,528 fluid particles: eight lanes; 22,568 and 32,768: one for the neighbours; 32,800: one; 1,000 beside 27,000 of
# tissue: eight, most slots of other kinds
@pytest.mark.parametrize("extras", [{}, dict(cohesion=0.02, surface_tension=0.5, vorticity=0.3)])
@pytest.mark.parametrize("dims, tissue", [((22, 32, 32), 0), ((31, 28, 26), 0), ((32, 32, 32), 0), ((25, 32, 41), 0), ((10, 10, 10), 30)])
def test_lanes_equal_the_oracle(dims, tissue, extras):
    w = World()
    sp = 0.05
    size = tuple(n * sp for n in dims)
    w.add_fluid_grid(size, sp, position=(size[0] * 0.5 + 0.005, size[1] * 0.5 + 0.005, size[2] * 0.5), radius=0.6 * sp,
                     viscosity=0.01, **extras)
    if tissue:
        side = (tissue - 1) * 0.1
        w.add_soft_body_grid((side,) * 3, 0.1, position=(10.0, side * 0.5 + 0.04, 0.0), radius=0.04, edge_compliance=1e-5,
                             volume_compliance=1e-6)
    scenes.ground(w)
    soa = w.soa()
    v = w.velocities()
    v[:, :3] = np.random.default_rng(4).normal(0.0, 0.5, (len(v), 3)).astype(np.float32) * (w.positions()[:, 3:] > 0)
    desc = solver_desc(substeps=2, default_iterations=4, enable_blocking_readback=0)
    gpu, ora = Solver(desc), cn_oracle.Oracle(desc, soa)
    gpu.sync_world(soa)
    gpu.step(1.0 / 120.0)
    ora.step(1.0 / 120.0)
    for a, b in zip(gpu.read_particles(), ora.read_particles()):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), float(np.abs(a - b).max())
