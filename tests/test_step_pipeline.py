"""The step kernel's pipeline where its warps do unequal work: tiles whose last rows do not exist (their
warps only hand the stages on, and run as far ahead as the ring allows), over many planes and items."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fields(monkeypatch, desc, init, steps, ty):
    from mrlbm_3d_cuda_gb300 import Simulation
    monkeypatch.setenv("MRLBM_TILE_Y", str(ty))
    with Simulation(desc, init=False) as sim:
        sim.init(*init)
        sim.step(steps)
        sim.sync()
        return sim.moments()


@pytest.mark.parametrize("storage", [0, 1, 3])
@pytest.mark.parametrize("kind", ["periodic", "channel"])
def test_rows_past_the_tile(cuda_device, kind, storage, monkeypatch):
    """8 of 16 rows missing in every other tile of a 24-row box, and in a third of a 40-row channel's
    (whose CTAs take over each other's items), against tiles of 8 rows, which are all whole: every
    store is of the same values, so the fields have the same bits."""
    from mrlbm_3d_cuda_gb300 import cases
    from mrlbm_3d_cuda_gb300 import native as N
    if kind == "periodic":
        desc = cases.periodic_box(512, 24, 256, u0=0.05, re=100.0, length=8.0, storage=storage)
        init = N.INIT_NOISY_UNIFORM, (0.03, 0.01, -0.02, 0.3, 13)
    else:
        desc = cases.cylinder_channel(320, 40, 128, 10, 63.6, 19.7, 0.05, 60.0, storage=storage)
        init = N.INIT_NOISY_UNIFORM, (0.05, 0.0, 0.0, 0.01, 5)
    want = fields(monkeypatch, desc, init, 12, 8)
    assert np.isfinite(want).all()
    got = fields(monkeypatch, desc, init, 12, 16)
    assert np.array_equal(got, want)


def test_tall_narrow_case_in_a_batch(cuda_device):
    """The segment length chosen for a batch keeps the tallest case's segments within a work item's 11 bits: one
    column of 220,000 planes would otherwise be cut into 2200 segments and refused."""
    from mrlbm_3d_cuda_gb300 import Batch, Simulation, cases
    from mrlbm_3d_cuda_gb300 import native as N
    desc = cases.periodic_box(8, 8, 220000, u0=0.05, re=100.0, length=8.0, storage=1)
    init = N.INIT_NOISY_UNIFORM, (0.03, 0.01, -0.02, 0.3, 13)
    with Simulation(desc, init=False) as sim:
        sim.init(*init)
        sim.step(2)
        sim.sync()
        want = sim.moments()
    b = Batch([desc])
    b.cases[0].init(*init)
    b.step(2)
    b.sync()
    assert np.array_equal(b.cases[0].moments(), want)
    b.close()


def test_side_buffer_holds_the_tiles_that_use_it(cuda_device):
    """Snapshots take 64 bytes for each node of a tile with stencil, wall or BCFLUID nodes, narrow tiles sharing slots of
    64 columns, and none for a tile that only touches a domain face.  A channel with a small cylinder needs little more on the
    device than its moments (131 MB; 126 MB more if each of its tiles, which all have face nodes, held 64 x 16
    columns), and a 136 x 136 x 112 annulus 20 slots, 140 MB, beside its 186 MB of moments (189 MB if all 27 tiles had one)."""
    import torch
    from mrlbm_3d_cuda_gb300 import Simulation, cases
    Simulation(cases.cylinder_channel(64, 40, 8, 10, 24.3, 19.7, 0.05, 60.0), init=False).close()  # context and module
    for desc, most in ((cases.cylinder_channel(320, 40, 128, 10, 63.6, 19.7, 0.05, 60.0), 48),
                       (cases.annulus(136, 136, 112, 32.0, 64.0, 0.03, 70.0), 140 + 24)):
        free = torch.cuda.mem_get_info()[0]
        with Simulation(desc, init=False):
            used = free - torch.cuda.mem_get_info()[0]
        moments = 2 * 4 * 10 * -(-desc.nx // 32) * 32 * desc.ny * desc.nz
        assert moments <= used <= moments + most * 2 ** 20, (used - moments) / 2 ** 20
