"""2D grids stepped in windows (several steps per launch) against the
same grid stepped with one launch per half step (the sweep kernel set by
hand): the arithmetic per cell is the same, so every stored value is equal.
Extents at and around the windows' edges (64 columns, 32 and 64 rows, and the
inner cells they own), calls of one, few and many steps."""
import numpy as np
import pytest

from fdtd_b200 import problem as P
from helpers import mode_fields

pytestmark = pytest.mark.gpu


def _problem(mode, nx, ny, seed):
    rng = np.random.default_rng(seed)
    dt = P.courant_dt(1e-6, 0.98 / np.sqrt(2.0))
    p = P.Problem(mode, (nx, ny, 1), 1e-6, dt)
    for a, n in ((0, nx), (1, ny)):
        for s in (0, 1):
            if n >= 20 and (seed + a + 2 * s) % 5:
                p.pml[(a, s)] = 3 + (seed + s) % 4
    p.materials = [P.Material.vacuum(), P.Material.constant(3.0), P.Material.constant(1.7)]
    p.ids = rng.integers(0, 3, size=(1, ny, nx)).astype(np.uint8)
    if seed % 3 == 0:
        p.eps_map = np.where(rng.random((1, ny, nx)) < 0.3, rng.uniform(1.0, 5.0, (1, ny, nx)), 0.0)
    e, h = (2, 0) if mode == P.TM else (0, 2)
    at = lambda: (int(rng.integers(1, nx - 1)), int(rng.integers(1, ny - 1)), 0)
    c = at()
    g = lambda t0: P.gaussian_pulse(90, t0, 7)
    p.sources += [P.Source(e, c, g(12), "E"), P.Source(e, c, 0.4 * g(30), "E"),
                  P.Source(h, at(), 1e-3 * g(14), "H"), P.Source(e, at(), 1e-12 * g(10), "D"),
                  P.Source(h, at(), 1e-9 * g(16), "B"),
                  P.Source(e, (1, min(4, ny - 2), 0), g(18), "E", hi=(nx - 2, min(4, ny - 2), 0)),
                  P.Source(h, (nx // 2, 1, 0), 1e-3 * g(22), "H", hi=(nx // 2, ny - 2, 0))]
    for q in (e, 3 + h):
        p.dfts.append(P.DFTRegion(q, (0, ny // 2, 0), (nx - 1, ny // 2, 0), [0.02, 0.05]))
    p.dfts.append(P.DFTRegion(e, (nx // 3, 0, 0), (nx // 2, ny - 1, 0), [0.03]))
    return p


@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("nx,ny", [(3, 3), (5, 70), (64, 64), (65, 33), (63, 32), (107, 65), (108, 44), (129, 97),
                                   (300, 20), (701, 590)])
def test_windows_equal_the_half_step_launches(fdtd, mode, nx, ny):
    p = _problem(mode, nx, ny, nx + ny)
    E, H, _, _ = mode_fields(mode)
    psi = [n for n in fdtd.PSI_NAMES]
    out = []
    for kind in ("auto", "regs"):
        g = fdtd.Grid.from_problem(p, "f32")
        g.set_sweep_kernel(kind)
        for n in (1, 2, 3, 13, 64, 71):
            g.step(n)
        assert g.step_count == 154 and g.error_flags() == 0
        vals = [g.get(n) for n in E + H] + [g.dft(h) for h in g.dft_handles]
        for n in psi:
            try:
                vals.append(g.get(n))
            except fdtd.FdtdError:
                pass
        out.append(vals)
    assert any(np.any(v) for v in out[0])
    for q, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), (q, float(np.abs(a - b).max()))


def test_windows_on_a_caller_stream_without_graphs(fdtd):
    """Eager windows on a stream of the caller, and a grid changed between
    calls (another material map, then a boundary condition the windows do not
    cover), follow the launches per half step."""
    import torch
    p = _problem(P.TE, 150, 101, 4)
    s = torch.cuda.Stream()
    out = []
    for kind in ("auto", "regs"):
        g = fdtd.Grid.from_problem(p, "f32")
        g.set_sweep_kernel(kind)
        g.use_graphs(False)
        g.step(40, stream=s.cuda_stream)
        s.synchronize()
        g.set_material_ids(np.roll(p.ids, 7, axis=2))
        g.step(41)
        g.set_boundary(0, 0, "pec")
        g.step(9)
        out.append([g.get(n) for n in ("Ex", "Ey", "Hz")] + [g.dft(0)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def _problem64(mode, nx, ny, seed, poles):
    """The same with TFSF planes where they fit, and materials with poles."""
    p = _problem(mode, nx, ny, seed)
    dt = p.dt
    if poles:
        p.materials[1] = P.Material.drude(1.0, 0.25 / dt, 0.02 / dt)
        lor = [(1.2, 0.1 / dt, 0.01 / dt), (0.6, 0.2 / dt, 0.02 / dt)][:poles]
        p.materials[2] = P.Material.lorentz(1.5, lor)
        rng = np.random.default_rng(seed)
        p.ids = (rng.integers(0, 3, size=(1, ny, nx)) * (rng.random((1, ny, nx)) < 0.2)).astype(np.uint8)
    if min(nx, ny) >= 30:
        k = (np.cos(0.3), np.sin(0.3), 0.0)
        pe, ph = P.ref_te_polarisation(k) if mode == P.TE else P.ref_tm_polarisation(k)
        p.tfsf = P.TFSF(2 * max(nx, ny), P.gaussian_pulse(120, 30, 8, offset=1.0), (nx / 2, ny / 2, 0.0), k, pe, ph,
                        P.tfsf_box_planes(mode, (11, 10), (nx - 12, ny - 11)))
    return p


@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("nx,ny,poles", [(3, 3, 0), (64, 32, 0), (65, 33, 1), (31, 64, 2), (113, 47, 0), (112, 48, 1),
                                         (200, 131, 2), (410, 300, 0)])
def test_fp64_windows_equal_the_half_step_launches(fdtd, mode, nx, ny, poles):
    p = _problem64(mode, nx, ny, nx + ny, poles)
    E, H, D, B = mode_fields(mode)
    names = E + H + D + B + ["Px", "Py", "Pz", "Jx", "Jy", "Jz"] + list(fdtd.PSI_NAMES)
    out = []
    for kind in ("auto", "regs"):
        g = fdtd.Grid.from_problem(p, "f64")
        g.set_sweep_kernel(kind)
        for n in (1, 2, 3, 13, 64, 71):
            g.step(n)
        vals = []
        for n in names:
            try:
                vals.append(g.get(n))
            except fdtd.FdtdError:
                pass
        out.append(vals + [g.dft(h) for h in g.dft_handles])
    assert any(np.any(v) for v in out[0])
    for q, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), (q, float(np.abs(a - b).max()))


@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("eps,mu_r", [(np.inf, 1.0), (1e60, 1.0), (1e-25, 1e-25), (2.0, np.inf), (2.0, 1e60)])
def test_fp64_windows_with_divisors_at_the_ends_of_the_range(fdtd, mode, eps, mu_r):
    """Divisors whose reciprocals do not give the quotient, and zeros of either
    sign: every stored value, the zeros' signs too, as the half-step launches'."""
    nx, ny = 70, 41
    p = _problem64(mode, nx, ny, 5, 0)
    p.tfsf = None
    p.materials = [P.Material.constant(1.5, mu_r), P.Material.constant(eps, mu_r)]
    p.ids = (np.indices((1, ny, nx))[2] % 7 == 3).astype(np.uint8)
    E, H, D, B = mode_fields(mode)
    rng = np.random.default_rng(1)
    start = {n: np.where(rng.random((1, ny, nx)) < 0.5, -0.0, rng.normal(size=(1, ny, nx)) * 1e-12) for n in D + B}
    out = []
    for kind in ("auto", "regs"):
        g = fdtd.Grid.from_problem(p, "f64")
        g.set_sweep_kernel(kind)
        for n, v in start.items():
            g.set(n, v)
        g.step(4)
        out.append([g.get(n) for n in E + H + D + B])
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)
        ok = ~np.isnan(a)
        assert np.array_equal(np.signbit(a[ok]), np.signbit(b[ok]))


@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("nx,ny,poles", [(3, 3, 1), (31, 64, 0), (64, 32, -1), (65, 33, 1), (113, 47, 2), (112, 48, 0),
                                         (130, 66, -1), (200, 131, 2), (410, 300, 1), (701, 590, -1)])
def test_windows_with_poles_and_planes(fdtd, mode, nx, ny, poles):
    """FP32 windows of grids with poles (-1: Drude alone, which keeps no P) and
    TFSF planes: each window's edges, cells of every material in one row, pole
    cells on planes, on box edges and under sources; a grid of one material with
    poles; J and P left in cells whose material has none are not touched."""
    p = _problem64(mode, nx, ny, nx + ny, abs(poles))
    dt = p.dt
    if poles == -1:
        p.materials[2] = P.Material.drude(2.0, 0.15 / dt, 0.03 / dt)
    if (nx, ny) == (65, 33):
        p.materials, p.ids, p.eps_map = p.materials[2:], None, None
    E, H, _, _ = mode_fields(mode)
    names = E + H + ["Px", "Py", "Pz", "Jx", "Jy", "Jz"] + list(fdtd.PSI_NAMES)
    rng = np.random.default_rng(3)
    stray = rng.normal(size=(1, ny, nx)) * 1e-3
    out = []
    for kind in ("auto", "regs"):
        g = fdtd.Grid.from_problem(p, "f32")
        g.set_sweep_kernel(kind)
        if poles:
            g.set("J" + E[0][1], stray)
        for n in (1, 2, 3, 13, 64, 71):
            g.step(n)
        vals = []
        for n in names:
            try:
                vals.append(g.get(n))
            except fdtd.FdtdError:
                pass
        out.append(vals + [g.dft(h) for h in g.dft_handles])
    assert any(np.any(v) for v in out[0])
    for q, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), (q, float(np.abs(a - b).max()))
