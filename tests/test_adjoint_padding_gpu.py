"""Gradients of grids of odd extent in device memory that held values that are not
finite: what lies beyond a row's last cell is no part of them."""
import numpy as np
import pytest

from fdtd_b200 import problem as P

pytestmark = pytest.mark.gpu

NX, NY, STEPS = 65, 61, 90


def _gradient(fdtd, kind):
    p = P.Problem(P.TM, (NX, NY, 1), 1e-6, P.courant_dt(1e-6, 0.98 / np.sqrt(2.0)))
    for a in (0, 1):
        for s in (0, 1):
            p.pml[(a, s)] = 5
    p.eps_map = np.zeros((1, NY, NX))
    p.eps_map[0, 20:31, 20:31] = np.random.default_rng(0).uniform(1.0, 6.0, size=(11, 11))
    p.sources.append(P.Source(2, (14, 14, 0), np.sin(0.3 * np.arange(STEPS)), "E"))
    g = fdtd.Grid.from_problem(p, "f32")
    g.set_sweep_kernel(kind)
    adj = fdtd.Adjoint(g, (50, 30), (50, 33), 0.05, (20, 20), (30, 30), 64)
    out = adj.forward(STEPS), adj.backward()
    adj.close()
    g.close()
    return out


def test_memory_that_held_nan(fdtd):
    want = _gradient(fdtd, "regs")
    nan = np.full((1, NY, NX - 1 + 64), np.nan)
    # (arrays of the sizes that the gradient will lay out, and one that keeps
    # their memory from going back to the device)
    keep = fdtd.Grid.from_problem(P.Problem(P.TM, (NX, NY, 1), 1e-6, 1e-15), "f32")
    for _ in range(3):
        held = [fdtd.Grid.from_problem(P.Problem(P.TM, (nan.shape[2], NY, 1), 1e-6, 1e-15), "f32") for _ in range(12)]
        for h in held:
            for n in ("Ez", "Hx", "Hy"):
                h.set(n, nan)
        for h in held:
            h.close()
        got = _gradient(fdtd, "auto")
        assert got[0] == want[0] != 0.0
        assert np.array_equal(got[1], want[1]) and np.all(got[1])
    keep.close()
