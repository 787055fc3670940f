"""Steps that a caller captures into its own CUDA graph (mrlbm_set_stream), and the order of the kernels of
a step among themselves and against the steps before it."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def case(kind):
    from mrlbm_3d_cuda_gb300 import cases
    if kind == "periodic":
        return cases.periodic_box(72, 40, 16, u0=0.05, re=100.0, length=8.0)
    if kind == "channel":
        return cases.cylinder_channel(96, 40, 16, 10, 32.6, 19.7, 0.05, 60.0)
    return cases.annulus(48, 48, 8, 8.0, 20.0, 0.05, 50.0)


@pytest.mark.parametrize("kind", ["periodic", "channel", "annulus"])
def test_captured_pair_of_steps(cuda_device, kind):
    """Two steps (both buffer parities) captured on the caller's stream and replayed, against the
    same steps called one by one: the same kernels on the same state, so the same bits."""
    import torch
    from mrlbm_3d_cuda_gb300 import Simulation
    from mrlbm_3d_cuda_gb300 import native as N
    init = N.INIT_NOISY_UNIFORM, (0.03, 0.0, 0.0, 0.02, 3)
    with Simulation(case(kind), init=False) as sim:
        sim.init(*init)
        sim.step(14)
        sim.sync()
        want = sim.moments()
    with Simulation(case(kind), init=False) as sim:
        sim.init(*init)
        sim.step(2)
        sim.sync()
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        sim.set_stream(stream.cuda_stream)
        with torch.cuda.graph(graph, stream=stream):
            sim.step(2)
        with torch.cuda.stream(stream):
            for _ in range(6):
                graph.replay()
        stream.synchronize()
        got = sim.moments()
        sim.set_stream(None)
    assert np.array_equal(got, want)
