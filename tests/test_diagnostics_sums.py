"""Mass and energy sums over long segments: a lane adds the pairs of 16 planes, and these sums to its totals, in
FP32; FP64 from there on.

A uniform flow makes every term of a lane the same, so that rounding of a long FP32 sum would add up in one
direction in every lane (up to 94 x 2^-24 of the sum over 2 x 256 nodes added one by one).  n additions of equal
terms are off by at most (n + 1) / 2 half ulps of the result, 2^-24 each: 8.5 for the pairs of 16 planes, (m + 1) / 2 for
m = planes / 16 of their sums.  The term itself has four roundings more (the square's three, the storage
scale's one).  The field after the step holds the same density and velocity (collision keeps them), so the
reference is its FP64 sum."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [0, 3])  # velocities stored in FP32
@pytest.mark.parametrize("shape,lz", [((64, 16, 256), 256), ((32, 32, 256), 256), ((64, 16, 256), 9), ((128, 48, 40), 0)])
def test_long_segments(cuda_device, shape, lz, storage, monkeypatch):
    from mrlbm_3d_cuda_gb300 import Simulation, cases
    if lz:
        monkeypatch.setenv("MRLBM_LZ", str(lz))
    sums = 8.5 + ((lz or 40) / 16 + 1) / 2
    desc = cases.periodic_box(*shape, u0=0.05, re=100.0, length=8.0, storage=storage)
    for u, dev in (((0.0463, 0.0, 0.0), 0.0107), ((0.0391, -0.0278, 0.0171), 1.37e-3), ((0.011, 0.023, -0.031), 0.0031)):
        m = np.zeros((10,) + shape[::-1], np.float32)
        m[0] = dev
        for a in range(3):
            m[1 + a] = u[a]
        for f, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            m[4 + f] = u[a] * u[b]
        with Simulation(desc, init=False) as sim:
            sim.set_moments(m)
            sim.set_sampling(0, 1)
            sim.step(1)
            sim.sync()
            mass, energy = sim.diagnostics()[1][-1]
            got = sim.moments().astype(np.float64)
        want = 0.5 * (got[1:4] ** 2).sum()
        assert abs(energy / want - 1.0) <= (sums + 4.0) * 2.0 ** -24, (u, (energy / want - 1.0) * 2.0 ** 24)
        if storage == 0:  # the hybrid storage rounds rho when it stores it, after the sums
            n = float(np.prod(shape))
            assert abs((mass - n) / got[0].sum() - 1.0) <= sums * 2.0 ** -24 + n * 2.0 ** -52 / got[0].sum()
