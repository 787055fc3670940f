"""Step kernel at the edges of its tiles: 64-node tile columns (two 32-node blocks, the last one partial
or missing), tile heights with a remainder row block, z segments down to one plane, more work
items than CTAs.

FP32 against the FP32 oracle, and every (tile height, z segment) bit for bit against the default
tiling in every storage mode.  The oracle bound is the strict one of the parity tests: 1e-5 in the
scaled metric for short runs (FP32 rounding of u = j / rho is about 1e-7 absolute a step, 2e-6 of
u = 0.05, and grows with the square root of the steps: 6e-6 after 8)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import field_errors

pytestmark = pytest.mark.gpu
INIT = (0.03, 0.01, -0.02, 0.3, 13)


def run(shape, storage, steps, monkeypatch, tile=None, sr=0):
    from mrlbm_3d_cuda_gb300 import Simulation, cases
    from mrlbm_3d_cuda_gb300 import native as N
    for name, v in zip(("MRLBM_TILE_Y", "MRLBM_LZ"), tile or (None, None)):
        if v is None:
            monkeypatch.delenv(name, raising=False)
        else:
            monkeypatch.setenv(name, str(v))
    desc = cases.periodic_box(*shape, u0=0.05, re=100.0, length=8.0, storage=storage)
    desc.stochastic_rounding = sr
    with Simulation(desc, init=False) as sim:
        sim.init(N.INIT_NOISY_UNIFORM, INIT)
        sim.step(steps)
        sim.sync()
        return desc, sim.moments()


# one block; two; a block and a remainder; a tile and an 8-, 16- or 40-node remainder; heights of one row
# block, exactly one tile, a tile and a remainder; more items than SMs (64 tiles x 4 segments)
SHAPES = [(32, 8, 4), (64, 16, 8), (56, 24, 8), (72, 16, 12), (80, 40, 4), (104, 8, 20), (136, 136, 4), (512, 128, 32)]


@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_matches_oracle(cuda_device, shape, monkeypatch):
    import oracle
    from mrlbm_3d_cuda_gb300 import native as N
    steps = 8
    desc, m = run(shape, N.STORAGE_F32, steps, monkeypatch)
    o = oracle.Oracle(desc, 32)
    o.init(N.INIT_NOISY_UNIFORM, INIT)
    o.step(steps)
    err = field_errors(m, o.moments(), 0.05)[:, 0]
    o.close()
    assert err.max() < 1e-5, err


@pytest.mark.parametrize("storage,sr", [(0, 0), (1, 0), (2, 1), (3, 1)])
@pytest.mark.parametrize("shape", [(72, 24, 12), (136, 40, 8)])
def test_every_tiling_gives_the_same_bits(cuda_device, shape, storage, sr, monkeypatch):
    _, want = run(shape, storage, 5, monkeypatch, sr=sr)
    for tile in ((4, 1), (8, 3), (16, shape[2]), (16, 1)):
        _, got = run(shape, storage, 5, monkeypatch, tile=tile, sr=sr)
        assert np.array_equal(got, want), tile
