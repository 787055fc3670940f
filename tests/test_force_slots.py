"""Force samples start from zero: the node-list kernel clears the slot that the wall kernel adds to, at list lengths
that fill neither a warp's ten nodes nor a block.  A second run of the same steps finds the first run's sums in its
slots and must give the same forces: FP64 sums whose block partials are added atomically, equal up to the
order of those additions (1e-9 of the force's scale, as for batches)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [0, 1])
@pytest.mark.parametrize("kind", ["channel", "z walls", "annulus", "narrow"])
def test_slots_start_from_zero(cuda_device, kind, storage):
    from mrlbm_3d_cuda_gb300 import Simulation, cases
    from mrlbm_3d_cuda_gb300 import native as N
    if kind == "channel":
        desc = cases.cylinder_channel(96, 40, 8, 10, 63.6, 15.8, 0.05, 60.0, storage=storage)
    elif kind == "z walls":
        desc = cases.cylinder_channel(64, 40, 8, 10, 24.3, 19.7, 0.05, 60.0, periodic_z=False, storage=storage)
    elif kind == "annulus":
        desc = cases.annulus(80, 80, 8, 9.5, 33.0, 0.05, 50.0, u_outer=-0.02, periodic_z=False, storage=storage)
    else:
        desc = cases.cylinder_channel(24, 40, 8, 4, 11.3, 19.7, 0.05, 40.0, storage=storage)
    runs = []
    with Simulation(desc, init=False) as sim:
        for _ in range(2):
            sim.init(N.INIT_NOISY_UNIFORM, (0.03, 0.01, 0.0, 0.05, 13))
            sim.set_sampling(1, 0)
            sim.step(5)
            sim.sync()
            steps, f = sim.force_history()
            assert list(steps) == list(range(5))
            runs.append(f)
    assert np.abs(runs[0]).max() > 0.0
    assert np.all(np.abs(runs[1] - runs[0]) <= 1e-9 * np.abs(runs[0]).max(axis=(0, 2), keepdims=True))
