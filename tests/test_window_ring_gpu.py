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


def test_adjoint_forward_of_a_non_finite_grid(fdtd):
    """The same for the forward of the stored adjoint, a spectrum over the whole
    grid beside the probe's."""
    nx, ny = 90, 70
    out = []
    for kind in ("auto", "regs"):
        p = P.Problem(P.TM, (nx, ny, 1), 1e-6, P.courant_dt(1e-6, 0.98 / np.sqrt(2.0)))
        p.dfts.append(P.DFTRegion(2, (0, 0, 0), (nx - 1, ny - 1, 0), [0.02]))
        p.dfts.append(P.DFTRegion(4, (0, 5, 0), (nx - 1, 5, 0), [0.02]))
        g = fdtd.Grid.from_problem(p, "f32")
        g.set_sweep_kernel(kind)
        v = np.random.default_rng(0).normal(size=(1, ny, nx))
        v[0, 3, 2] = np.inf
        v[0, 0, :] = v[0, -1, :] = v[0, :, 0] = 0.25
        g.set("Ez", v)
        adj = fdtd.Adjoint(g, (70, 30), (70, 33), 0.05, (40, 30), (50, 40), 64)
        J = adj.forward(12)
        out.append([np.array(J), g.get("Ez"), g.get("Hy"), g.dft(0), g.dft(1)])
        adj.close()
    for q, (a, b) in enumerate(zip(*out)):
        ok = np.isfinite(a)
        assert np.array_equal(ok, np.isfinite(b)), q
        assert np.array_equal(a[ok], b[ok]) and np.any(a[ok]), q


@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
def test_non_finite_cells_beside_poles(fdtd, mode):
    """FP32 windows of a grid with Drude cells in its corner, where the value is."""
    nx, ny = 90, 70
    p = P.Problem(mode, (nx, ny, 1), 1e-6, P.courant_dt(1e-6, 0.98 / np.sqrt(2.0)))
    p.materials.append(P.Material.drude(1.0, 0.25 / p.dt, 0.02 / p.dt))
    p.ids = np.zeros((1, ny, nx), np.uint8)
    p.ids[0, :12, :15] = 1
    E, H, _, _ = mode_fields(mode)
    for c in ([0, 1, 5] if mode == P.TE else [2, 3, 4]):
        p.dfts.append(P.DFTRegion(c, (0, 0, 0), (nx - 1, ny - 1, 0), [0.02]))
    v = np.random.default_rng(0).normal(size=(1, ny, nx))
    v[0, 3, 2] = np.inf
    v[0, 0, :] = v[0, -1, :] = v[0, :, 0] = 0.25
    out = []
    for kind in ("windows", "regs"):
        g = fdtd.Grid.from_problem(p, "f32")
        g.always_window() if kind == "windows" else g.set_sweep_kernel(kind)
        g.set(E[-1], v)
        g.step(8)
        out.append([g.get(n) for n in E + H] + [g.dft(h) for h in g.dft_handles])
    for q, (a, b) in enumerate(zip(*out)):
        ok = np.isfinite(a)
        assert np.array_equal(ok, np.isfinite(b)), q
        assert np.array_equal(a[ok], b[ok]) and np.any(a[ok]), q
