"""The stored adjoint's memory: bounded by what the checkpoints of the caller's
ckpt_every take, laid out as a whole before the forward, and given back where
it does not fit, so that the checkpointed adjoint runs as it would have. Every
gradient equals that of the checkpointed adjoint (checkpoints every 64 or 128
steps, so that both fold their DFT samples 64 at a time)."""
import gc

import numpy as np
import pytest

from fdtd_b200 import problem as P

pytestmark = pytest.mark.gpu


def _adjoint(fdtd, kind, steps, ckpt, probe, design=((30, 25), (229, 224))):
    nx, ny = 260, 250
    dt = P.courant_dt(1e-6, 0.98 / np.sqrt(2.0))
    p = P.Problem(P.TM, (nx, ny, 1), 1e-6, dt)
    for a in (0, 1):
        for s in (0, 1):
            p.pml[(a, s)] = 8
    p.sources.append(P.Source(2, (20, 120, 0), np.sin(0.3 * np.arange(steps)), "E"))
    g = fdtd.Grid.from_problem(p, "f32")
    g.set_sweep_kernel(kind)
    g.prepare()
    return g, fdtd.Adjoint(g, *probe, 0.05, *design, ckpt)


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_checkpoint_spacing_bounds_the_memory(fdtd):
    """16384 steps of 200 x 200 design cells are 2.6 GB of kept values; 129
    checkpoints of the state, about 0.25 GB."""
    probe = ((235, 100), (235, 110))
    used, out = {}, {}
    for kind in ("regs", "auto"):
        g, adj = _adjoint(fdtd, kind, 16384, 128, probe)
        before = _free()
        J = adj.forward(16384)
        out[kind] = (J, adj.backward())
        used[kind] = before - _free()
        adj.close()
        g.close()
    assert used["auto"] <= 8.5 * used["regs"], used
    assert out["auto"][0] == out["regs"][0] != 0.0
    assert np.array_equal(out["auto"][1], out["regs"][1]) and np.any(out["auto"][1])


@pytest.mark.parametrize("room_mb", [400, 700], ids=["terms", "probe-values"])
def test_no_memory_for_the_stored_terms(fdtd, room_mb):
    """10000 steps: 600 MB for the terms of 150 x 100 design cells and as much
    for the values of a probe box as large; the first does not fit, or the
    second does not. The 158 checkpoints (about 0.2 GB) do."""
    import torch
    steps, design, probe = 10000, ((40, 40), (189, 139)), ((60, 120), (209, 219))
    g, adj = _adjoint(fdtd, "regs", steps, 64, probe, design)
    want = (adj.forward(steps), adj.backward())
    adj.close()
    g.close()
    g, adj = _adjoint(fdtd, "auto", steps, 64, probe, design)
    gc.collect()
    torch.cuda.empty_cache()
    hold = torch.empty(_free() - (room_mb << 20), dtype=torch.uint8, device="cuda")
    try:
        got = (adj.forward(steps), adj.backward())
    finally:
        del hold
        torch.cuda.empty_cache()
    assert got[0] == want[0] != 0.0 and np.array_equal(got[1], want[1]) and np.any(want[1])
    adj.close()
    g.close()
