"""Node-list and wall kernels where they can go wrong: node counts that fill neither a warp's ten nodes
nor a block, bodies across tile edges (x = 64, y = 16), both walls in one warp, z walls.

FP32 against the FP32 oracle with the strict bound of the parity tests (1e-5 in the scaled metric, four
steps).  The narrow storage modes against FP32 from the same stored state after one step: the
closures then see the same values, and the results differ by the rounding of the store (half an
ulp: 2^-11 of the stored value for FP16 halves, 2^-8 for BF16, velocities and second moments as they
are, rho as its difference from 1) and by FP32 rounding (the strict bound again)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import field_errors

pytestmark = pytest.mark.gpu


def case(name, storage=0):
    from mrlbm_3d_cuda_gb300 import cases
    if name == "channel":  # body across the tile edges
        return cases.cylinder_channel(96, 40, 8, 10, 63.6, 15.8, 0.05, 60.0, storage=storage)
    if name == "periodic":
        return cases.cylinder_channel(72, 48, 4, 13.3, 30.2, 31.9, 0.05, 60.0, periodic_y=True, storage=storage)
    if name == "z walls":
        return cases.cylinder_channel(64, 40, 8, 10, 24.3, 19.7, 0.05, 60.0, periodic_z=False, storage=storage)
    if name == "annulus":
        return cases.annulus(48, 48, 4, 8.0, 20.0, 0.05, 50.0, storage=storage)
    return cases.annulus(80, 80, 8, 9.5, 33.0, 0.05, 50.0, u_outer=-0.02, periodic_z=False, storage=storage)


NAMES = ["channel", "periodic", "z walls", "annulus", "annulus, z walls"]


@pytest.mark.parametrize("name", NAMES)
def test_fp32_matches_oracle(cuda_device, name):
    import oracle
    from mrlbm_3d_cuda_gb300 import Simulation
    from mrlbm_3d_cuda_gb300 import native as N
    desc, steps = case(name), 4
    o = oracle.Oracle(desc, 32)
    o.init(N.INIT_REST, ())
    o.step(steps)
    with Simulation(desc, init=False) as sim:
        sim.init(N.INIT_REST, ())
        sim.set_sampling(1, 0)
        sim.step(steps)
        sim.sync()
        err = field_errors(sim.moments(), o.moments(), 0.05)[:, 0]
    o.close()
    assert err.max() < 1e-5, err


@pytest.mark.parametrize("storage,eps", [(1, 2.0 ** -11), (2, 2.0 ** -8), (3, 2.0 ** -11)])
@pytest.mark.parametrize("name", NAMES)
def test_narrow_storage_rounds_the_same_closures(cuda_device, name, storage, eps):
    from mrlbm_3d_cuda_gb300 import Simulation
    from mrlbm_3d_cuda_gb300 import native as N
    with Simulation(case(name, storage), init=False) as sim:
        sim.init(N.INIT_REST, ())
        sim.step(6)
        sim.sync()
        before = sim.moments()
        sim.step(1)
        sim.sync()
        got = sim.moments()
    with Simulation(case(name), init=False) as sim:
        sim.init(N.INIT_REST, ())
        sim.set_moments(before)
        sim.step(1)
        sim.sync()
        want = sim.moments()
    size = np.abs(want.astype(np.float64))
    size[0] = np.abs(want[0].astype(np.float64) - 1.0)
    scale = np.array([1.0] + [0.05] * 3 + [1.0 / 3.0] * 6).reshape((10,) + (1,) * (want.ndim - 1))
    excess = np.abs(got.astype(np.float64) - want) - eps * size - 1e-5 * np.maximum(scale, size)
    assert excess.max() <= 0.0, [float(e.max()) for e in excess]
