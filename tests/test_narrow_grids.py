"""Grids of at most 32 nodes along x: the step kernel's tiles of 32 rows of one x-block, where an owner warp holds two
rows that wrap within themselves.  Widths of 8 to 32 nodes, one tile and several, a remainder of rows, one
plane per segment, boundary tiles, batches of narrow and wide cases.

FP32 against the FP32 oracle with the strict bound of the parity tests (1e-5 in the scaled metric), and bit for
bit against 8-row tiles (two x-blocks wide) in every storage mode: the same operations on the same values."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import field_errors

pytestmark = pytest.mark.gpu
INIT = (0.03, 0.01, -0.02, 0.3, 13)


def narrow(kind, storage=0):
    from mrlbm_3d_cuda_gb300 import cases
    if kind == "annulus":
        return cases.annulus(32, 32, 8, 5.0, 12.0, 0.05, 40.0, storage=storage)
    if kind == "channel":
        return cases.cylinder_channel(32, 72, 12, 6, 14.3, 35.7, 0.05, 40.0, storage=storage)
    if kind == "plates":
        return cases.cylinder_channel(24, 40, 8, 4, 11.3, 19.7, 0.05, 40.0, periodic_z=False, storage=storage)
    return cases.periodic_box(*kind, u0=0.05, re=100.0, length=8.0, storage=storage)


def run(desc, steps):
    from mrlbm_3d_cuda_gb300 import Simulation
    from mrlbm_3d_cuda_gb300 import native as N
    with Simulation(desc, init=False) as sim:
        sim.init(N.INIT_NOISY_UNIFORM, INIT)
        sim.set_sampling(1, 1)
        sim.step(steps)
        sim.sync()
        return sim.moments(), sim.force_history()[1], sim.diagnostics()[1], int(sim.get_info().tile[1])


KINDS = [(8, 8, 4), (8, 40, 12), (16, 72, 8), (24, 32, 20), (32, 24, 8), (32, 136, 64), "annulus", "channel", "plates"]


@pytest.mark.parametrize("kind", KINDS)
def test_fp32_matches_oracle(cuda_device, kind):
    import oracle
    from mrlbm_3d_cuda_gb300 import native as N
    desc, steps = narrow(kind), 6
    m, _, _, rows = run(desc, steps)
    assert rows == 32
    o = oracle.Oracle(desc, 32)
    o.init(N.INIT_NOISY_UNIFORM, INIT)
    o.step(steps)
    err = field_errors(m, o.moments(), 0.05)[:, 0]
    o.close()
    assert err.max() < 1e-5, err


@pytest.mark.parametrize("storage,sr", [(0, 0), (1, 0), (2, 1), (3, 1)])
@pytest.mark.parametrize("kind", KINDS)
def test_every_tiling_gives_the_same_bits(cuda_device, kind, storage, sr, monkeypatch):
    desc = narrow(kind, storage)
    desc.stochastic_rounding = sr
    monkeypatch.setenv("MRLBM_TILE_Y", "8")
    want, forces, sums, rows = run(desc, 5)
    assert rows == 8
    for env in ({}, {"MRLBM_TILE_Y": "16", "MRLBM_LZ": "1"}):
        monkeypatch.delenv("MRLBM_TILE_Y", raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        got, f, s, rows = run(desc, 5)
        assert rows == 32
        assert np.array_equal(got, want)
        # FP64 sums whose block partials are added in another order, of FP32 per-lane sums (the energy's:
        # up to 2 x 64 terms, 128 half ulps of 2^-24)
        assert f.shape == forces.shape and np.all(np.abs(f - forces) <= 1e-9 * np.maximum(np.abs(forces).max(initial=0.0), 1e-12))
        assert np.all(np.abs(s - sums) <= np.array([1e-9, 128 * 2.0 ** -24]) * np.abs(sums))


def test_narrow_and_wide_cases_in_a_batch(cuda_device):
    from mrlbm_3d_cuda_gb300 import Batch, cases
    from mrlbm_3d_cuda_gb300 import native as N
    descs = [narrow(k) for k in KINDS] + [cases.cylinder_channel(64, 40, 12, 10, 24.3, 19.7, 0.05, 60.0),
                                          cases.periodic_box(72, 24, 12, u0=0.05, re=100.0, length=8.0)]
    for chosen in (descs, descs[:3]):  # both kernels; one alone
        want = [run(d, 6) for d in chosen]
        b = Batch(chosen)
        for c in b.cases:
            c.init(N.INIT_NOISY_UNIFORM, INIT)
        b.set_sampling(1)
        b.step(3)
        b.step_sequential(1)
        b.step(2)
        b.sync()
        for c, (m, f, _, _) in zip(b.cases, want):
            assert np.array_equal(c.moments(), m)
            got = c.force_history()[1]
            assert got.shape == f.shape
            if f.size:
                assert np.all(np.abs(got - f) <= 1e-9 * np.maximum(np.abs(f).max(), 1e-12))
        b.close()


@pytest.mark.parametrize("storage,sr", [(0, 0), (1, 1), (2, 0), (3, 1)])
def test_batch_of_plain_cases(cuda_device, storage, sr):
    """A batch without boundary nodes runs a kernel that reads no node marks: each case as if stepped alone."""
    from mrlbm_3d_cuda_gb300 import Batch
    from mrlbm_3d_cuda_gb300 import native as N
    descs = [narrow(k, storage) for k in ((72, 24, 12), (32, 40, 8), (136, 136, 20), (8, 8, 4), (64, 16, 32))]
    for d in descs:
        d.stochastic_rounding = sr
    want = [run(d, 5)[0] for d in descs]
    b = Batch(descs)
    for c in b.cases:
        c.init(N.INIT_NOISY_UNIFORM, INIT)
    b.step(5)
    b.sync()
    for c, m in zip(b.cases, want):
        assert np.array_equal(c.moments(), m)
    b.close()
