"""The step kernel's bounded waits: one that runs out ends in a status, with the kernel's copies landed and the
context usable.  The limit comes from the host (MRLBM_FAULT_WAIT_POLLS polls, read by each call that
steps): with 0 the warps that own the tile's rows give up at their first wait, while the copies of the
first planes are on their way; with a few, some waits run out and some do not.  A wait on copies that nobody
has issued would take the full limit, 16 s: each run ends long before that."""
from __future__ import annotations

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def descs(kind):
    from mrlbm_3d_cuda_gb300 import cases
    if kind == "periodic":  # more items than SMs, ragged in x and y, even and odd uses of every stage
        return cases.periodic_box(200, 136, 92, u0=0.05, re=100.0, length=8.0)
    return cases.cylinder_channel(128, 40, 64, 10, 32.6, 19.7, 0.05, 60.0)


def run(kind, steps, storage=0):
    from mrlbm_3d_cuda_gb300 import Simulation
    from mrlbm_3d_cuda_gb300 import native as N
    desc = descs(kind)
    desc.storage = storage
    with Simulation(desc, init=False) as sim:
        sim.init(N.INIT_NOISY_UNIFORM, (0.05, 0.0, 0.0, 0.01, 5))
        t = time.perf_counter()
        sim.step(steps)
        try:
            sim.sync()
            code = N.OK
        except N.MrlbmError as e:
            code = e.code
        assert time.perf_counter() - t < 8.0
        return code, sim.moments() if code == N.OK else None


@pytest.mark.parametrize("storage", [0, 1])
@pytest.mark.parametrize("tile_y", [4, 8, 16])
@pytest.mark.parametrize("kind", ["periodic", "channel"])
def test_wait_that_runs_out_is_a_status(cuda_device, kind, tile_y, storage, monkeypatch):
    from mrlbm_3d_cuda_gb300 import native as N
    monkeypatch.setenv("MRLBM_TILE_Y", str(tile_y))
    code, want = run(kind, 4, storage)
    assert code == N.OK
    for polls in (0, 1, 2, 3):
        monkeypatch.setenv("MRLBM_FAULT_WAIT_POLLS", str(polls))
        code, got = run(kind, 4, storage)
        assert code == (N.ERR_TIMEOUT if polls == 0 else code) and code in (N.OK, N.ERR_TIMEOUT)
        if code == N.OK:
            assert np.array_equal(got, want)
        monkeypatch.delenv("MRLBM_FAULT_WAIT_POLLS")
        code, got = run(kind, 4, storage)  # right behind it, on the same SMs
        assert code == N.OK and np.array_equal(got, want)


def test_allocation_free_step_reports_a_wait_that_ran_out(cuda_device, monkeypatch):
    """mrlbm_step_periodic_noalloc: with diagnostics the call itself returns the status; without, it has returned
    before its kernel ran, and the next call does (and launches nothing).  Either is reported once."""
    import ctypes as C

    import torch
    from mrlbm_3d_cuda_gb300 import native as N
    lib, shape = N.lib(), (72, 40, 16)
    g = torch.Generator().manual_seed(7)
    src = (1e-3 * torch.randn(96 * 40 * 16 * 10, generator=g)).cuda()
    stream = torch.cuda.current_stream().cuda_stream

    def call(dst, diag=None):
        return lib.mrlbm_step_periodic_noalloc(C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()), *shape,
                                               C.c_float(1.2), C.c_float(1.0), diag, C.c_void_p(stream))

    want, want_sums = torch.zeros_like(src), (C.c_double * 2)()
    assert call(want, want_sums) == N.OK
    for diag in ((C.c_double * 2)(), None):
        monkeypatch.setenv("MRLBM_FAULT_WAIT_POLLS", "0")
        assert call(torch.zeros_like(src), diag) == (N.ERR_TIMEOUT if diag is not None else N.OK)
        monkeypatch.delenv("MRLBM_FAULT_WAIT_POLLS")
        torch.cuda.synchronize()
        got, sums = torch.zeros_like(src), (C.c_double * 2)()
        if diag is None:
            assert call(got) == N.ERR_TIMEOUT and b"earlier call" in lib.mrlbm_last_error(None)
            torch.cuda.synchronize()
            assert not got.any()
        assert call(got, sums) == N.OK
        assert torch.equal(got, want) and list(sums) == list(want_sums)


def test_timed_out_handle_hands_out_nothing(cuda_device, monkeypatch, tmp_path):
    """After a wait ran out every read-back returns the status instead of the field's remains, and so does
    the next step once a read-back has seen it; a part of a new field does not clear it, a whole one does."""
    from mrlbm_3d_cuda_gb300 import Simulation
    from mrlbm_3d_cuda_gb300 import native as N
    init = N.INIT_NOISY_UNIFORM, (0.05, 0.0, 0.0, 0.01, 5)

    def refused(call):
        with pytest.raises(N.MrlbmError) as e:
            call()
        return e.value.code == N.ERR_TIMEOUT

    with Simulation(descs("channel"), init=False) as sim:
        sim.init(*init)
        sim.set_sampling(1, 1)
        sim.set_pressure_window(0, 100)
        field = sim.moments()
        sim.step(3)
        want = sim.moments()
        sim.init(*init)
        monkeypatch.setenv("MRLBM_FAULT_WAIT_POLLS", "0")
        sim.step(3)
        monkeypatch.delenv("MRLBM_FAULT_WAIT_POLLS")
        assert refused(sim.moments)
        assert refused(sim.force_history) and refused(sim.diagnostics) and refused(lambda: sim.forces(1))
        assert refused(lambda: sim.checkpoint_save(str(tmp_path / "restart.bin")))
        assert refused(lambda: sim.write_vti(str(tmp_path / "data.vti")))
        assert refused(lambda: sim.write_forces(str(tmp_path / "forces.dat")))
        assert refused(lambda: sim.write_pressure(str(tmp_path / "pressure.dat")))
        assert refused(lambda: sim.write_inlet_density(str(tmp_path / "inlet.dat")))
        assert refused(lambda: sim.step(1)) and refused(sim.sync)
        sim.set_moments(field[1:2], fields=["ux"])
        assert refused(sim.moments)
        sim.set_moments(field)
        assert np.array_equal(sim.moments(), field)
        sim.init(*init)
        sim.step(3)
        sim.sync()
        assert np.array_equal(sim.moments(), want)


def test_timed_out_batch_reports_every_case(cuda_device, monkeypatch):
    """Which items a batched launch left undone is not known: each case's handle has the status, and a new
    field for all of them steps again (the limit of a batch is the one it was created with)."""
    from mrlbm_3d_cuda_gb300 import Batch, cases
    from mrlbm_3d_cuda_gb300 import native as N
    monkeypatch.setenv("MRLBM_FAULT_WAIT_POLLS", "0")
    b = Batch([cases.periodic_box(64, 24, 8, u0=0.05, re=100.0, length=8.0), descs("channel"), descs("periodic")])
    monkeypatch.delenv("MRLBM_FAULT_WAIT_POLLS")
    for c in b.cases:
        c.init(N.INIT_NOISY_UNIFORM, (0.03, 0.0, 0.0, 0.01, 5))
    before = [c.moments() for c in b.cases]
    b.step(2)
    for c in b.cases:
        for call in (c.sync, c.moments):
            with pytest.raises(N.MrlbmError) as e:
                call()
            assert e.value.code == N.ERR_TIMEOUT
    with pytest.raises(N.MrlbmError) as e:
        b.sync()
    assert e.value.code == N.ERR_TIMEOUT
    for c, m in zip(b.cases, before):
        c.set_moments(m)
        assert np.array_equal(c.moments(), m)
    b.sync()
    b.close()
