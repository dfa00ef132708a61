"""A batch whose second copy of the state does not fit is tuned without temporal
blocking."""
import gc

import numpy as np
import pytest

from fdtd_b200 import problem as P

pytestmark = pytest.mark.gpu


def _grids(fdtd):
    grids = []
    for q in range(8):
        n = 2000 - 10 * q
        p = P.Problem(P.TE, (n, 2000, 1), 1e-6, P.courant_dt(1e-6, 0.98 / np.sqrt(2.0)))
        p.materials.append(P.Material.constant(3.0))
        p.ids = np.zeros((1, 2000, n), np.uint8)
        p.ids[0, 500:900, 300:800] = 1
        p.sources.append(P.Source(2, (n // 2, 1000, 0), P.gaussian_pulse(90, 10, 5), "H"))
        grids.append(fdtd.Grid.from_problem(p, "f32"))
    return grids


def test_tuned_without_room_for_temporal_blocking(fdtd):
    """0.4 GB of state: the tuner's snapshot fits into the 0.85 GB left, the second
    copy with 1/eps per cell (0.52 GB) beside it does not."""
    import torch
    grids = _grids(fdtd)
    batch = fdtd.Batch(grids)
    gc.collect()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (850 << 20), dtype=torch.uint8, device="cuda")
    try:
        batch.tune(4)
        assert batch.temporal()["depth"] == 0
        batch.step(20)
        got = [g.get("Hz") for g in grids]
    finally:
        del hold
        torch.cuda.empty_cache()
    batch.close()
    alone = _grids(fdtd)
    want = fdtd.Batch(alone)
    want.step(20)
    for g, a in zip(got, alone):
        assert np.array_equal(g, a.get("Hz")) and np.any(g)
    want.close()
