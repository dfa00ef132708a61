"""A value that is not finite (or overflows) next to the outer ring and in the
grid's middle: 2D grids stepped in windows have the fields and spectra of the
launches per half step, cell by cell, the ring's among them (which keeps its
value)."""
import numpy as np
import pytest

from fdtd_b200 import problem as P
from helpers import mode_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("npml,value", [(0, np.inf), (8, np.nan), (0, 3e38)])
@pytest.mark.parametrize("cell", [(3, 2), (66, 87), (30, 50)])
def test_non_finite_cells(fdtd, prec, mode, npml, value, cell):
    nx, ny = 90, 70
    p = P.Problem(mode, (nx, ny, 1), 1e-6, P.courant_dt(1e-6, 0.98 / np.sqrt(2.0)))
    if npml:
        for a in (0, 1):
            for s in (0, 1):
                p.pml[(a, s)] = npml
    E, H, _, _ = mode_fields(mode)
    e = E[-1]
    for c in ([0, 1, 5] if mode == P.TE else [2, 3, 4]):
        p.dfts.append(P.DFTRegion(c, (0, 0, 0), (nx - 1, ny - 1, 0), [0.02]))
    v = np.random.default_rng(0).normal(size=(1, ny, nx))
    v[0, cell[0], cell[1]] = value
    v[0, 0, :] = v[0, -1, :] = v[0, :, 0] = 0.25
    out = []
    for kind in ("auto", "regs"):
        g = fdtd.Grid.from_problem(p, prec)
        g.set_sweep_kernel(kind)
        g.set(e, v)
        if prec == "f64":
            g.set("D" + e[1], v * 8.854e-12)
        g.step(8)
        out.append([g.get(n) for n in E + H] + [g.dft(h) for h in g.dft_handles])
    for q, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(np.isfinite(a), np.isfinite(b)), q
        ok = np.isfinite(a)
        assert np.array_equal(a[ok], b[ok]) and np.any(a[ok]), q
