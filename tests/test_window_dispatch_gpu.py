"""Which grids step in windows, seen by the launches of a call, and windows forced
where the launches per half step would be the faster: every stored value equal
to the launches per half step."""
import gc

import numpy as np
import pytest

from fdtd_b200 import problem as P
from helpers import mode_fields
from test_window_gpu import _problem, _problem64

pytestmark = pytest.mark.gpu


def _values(fdtd, g, p, prec):
    E, H, D, B = mode_fields(p.mode)
    names = E + H + (D + B if prec == "f64" else []) + ["Px", "Py", "Pz", "Jx", "Jy", "Jz"] + list(fdtd.PSI_NAMES)
    vals = []
    for n in names:
        try:
            vals.append(g.get(n))
        except fdtd.FdtdError:
            pass
    return vals + [g.dft(h) for h in g.dft_handles]


def _launches(g, n):
    before = g.launch_count
    g.step(n)
    return g.launch_count - before


def _compare(fdtd, p, prec, calls, windows=True, change=None):
    out = []
    for kind in ("windows", "regs"):
        g = fdtd.Grid.from_problem(p, prec)
        if kind == "regs":
            g.set_sweep_kernel("regs")
        else:
            g.always_window()
        for q, n in enumerate(calls):
            if change is not None:
                change(g, q)
            launches = _launches(g, n)
            # per half step: two sweeps a step at least; in windows: two launches
            # for a short call, an eighth of that for a stretch of 64 steps, and
            # the tables, the counter and the DFT flush
            if kind == "windows" and n >= 13:
                assert (launches < 2 * n) == windows, (n, launches)
        assert g.error_flags() == 0
        out.append(_values(fdtd, g, p, prec))
        g.close()
    assert any(np.any(v) for v in out[0])
    for q, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), (q, float(np.abs(a - b).max()))


@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("nx,ny,poles", [(3, 3, 0), (64, 32, 0), (65, 33, 1), (31, 64, 2), (113, 47, 0), (112, 48, 1),
                                         (200, 131, 2), (410, 300, 0)])
def test_fp64_windows_forced(fdtd, mode, nx, ny, poles):
    # (two poles are more than a TE window holds)
    _compare(fdtd, _problem64(mode, nx, ny, nx + ny, poles), "f64", (1, 2, 3, 13, 64, 71), windows=not (mode == P.TE and poles == 2))


@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("nx,ny,poles", [(3, 3, 1), (31, 64, 0), (64, 32, -1), (65, 33, 1), (113, 47, 2), (112, 48, 0), (200, 131, 2)])
def test_fp32_windows_forced(fdtd, mode, nx, ny, poles):
    p = _problem64(mode, nx, ny, nx + ny, abs(poles))
    if poles == -1:
        p.materials[2] = P.Material.drude(2.0, 0.15 / p.dt, 0.03 / p.dt)
    _compare(fdtd, p, "f32", (1, 2, 3, 13, 64, 71))


def _vacuum(mode, nx, ny, dft=True):
    p = P.Problem(mode, (nx, ny, 1), 1e-6, P.courant_dt(1e-6, 0.98 / np.sqrt(2.0)))
    for a in (0, 1):
        for s in (0, 1):
            p.pml[(a, s)] = 8
    p.sources.append(P.Source(2, (nx // 2, ny // 2, 0), P.gaussian_pulse(90, 20, 7), "H" if mode == P.TE else "E"))
    if dft:
        p.dfts.append(P.DFTRegion(2 if mode == P.TM else 5, (0, 5, 0), (nx - 1, 5, 0), [0.02]))
    return p


@pytest.mark.parametrize("mode,prec,n,poles,windows", [
    (P.TE, "f32", 16, 0, True), (P.TM, "f32", 64, 0, True), (P.TE, "f64", 2, 0, False), (P.TM, "f64", 2, 0, False), (P.TE, "f64", 16, 0, True),
    (P.TM, "f64", 64, 0, True), (P.TE, "f64", 16, 1, False), (P.TE, "f64", 64, 1, False)])
def test_the_faster_form_is_taken(fdtd, mode, prec, n, poles, windows):
    """256 x 256 cells, where the two forms are far apart (a Lorentz pole in every
    cell, or none)."""
    p = _vacuum(mode, 256, 256, dft=False)
    if poles:
        p.materials = [P.Material.lorentz(1.5, [(1.2, 0.1 / p.dt, 0.01 / p.dt)])]
    g = fdtd.Grid.from_problem(p, prec)
    g.prepare()
    assert (_launches(g, n) < 2 * n) == windows
    g.set_sweep_kernel("regs")
    assert _launches(g, n) >= 2 * n


# at each limit of what a window lists, and one past it
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("boxes,windows", [(8, True), (9, False)])
def test_box_sources(fdtd, prec, boxes, windows):
    p = _vacuum(P.TE, 150, 90)
    for q in range(boxes):
        lo = (10 + 9 * q, 8 + 3 * q, 0)
        comp, target = ((0, "E"), (1, "E"), (2, "H"))[q % 3]
        p.sources.append(P.Source(comp, lo, 1e-3 * P.gaussian_pulse(90, 15 + q, 7), target, hi=(lo[0] + 20, lo[1] + 12, 0)))
    _compare(fdtd, p, prec, (3, 64, 40), windows)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("regions,windows", [(32, True), (33, False)])
def test_dft_regions(fdtd, prec, regions, windows):
    p = _vacuum(P.TM, 150, 90, dft=False)
    for q in range(regions):
        p.dfts.append(P.DFTRegion(2, (q, 2 * q, 0), (q + 60, 2 * q + 10, 0), [0.02, 0.03]))
    p.dfts.append(P.DFTRegion(3, (0, 0, 0), (149, 89, 0), [0.05]))
    _compare(fdtd, p, prec, (3, 64, 40), windows)


@pytest.mark.parametrize("more,windows", [(0, True), (1, False)])
def test_fp64_acts(fdtd, more, windows):
    """32 of sources, boxes and twice the planes: 8 boxes, 4 planes and 16 sources;
    and one plane more."""
    p = _vacuum(P.TM, 150, 90)
    planes = P.tfsf_box_planes(P.TM, (15, 15), (134, 74))
    planes += P.tfsf_box_planes(P.TM, (20, 20), (120, 70))[:more]
    p.tfsf = P.TFSF(300, P.gaussian_pulse(120, 30, 8, offset=1.0), (75.0, 45.0, 0.0), (1.0, 0.0, 0.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0), planes)
    for q in range(8):
        p.sources.append(P.Source(2, (10 + 9 * q, 8 + 3 * q, 0), 1e-3 * P.gaussian_pulse(90, 15 + q, 7), "E", hi=(30 + 9 * q, 20 + 3 * q, 0)))
    for q in range(15):
        p.sources.append(P.Source(2, (20 + 7 * q, 40, 0), P.gaussian_pulse(90, 18 + q, 7), "E"))
    _compare(fdtd, p, "f64", (3, 64, 40), windows)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("poles", [0, 1])
def test_block_maps(fdtd, prec, mode, poles):
    """Materials by blocks of cells, a plane wave across them, and an eps map."""
    nx, ny = 141, 75
    p = _problem64(mode, nx, ny, 9, poles)  # (an eps map: the seed is a multiple of 3)
    rng = np.random.default_rng(3)
    p.ids, p.block_shift = None, 3
    p.block_ids = rng.integers(0, 3, size=(1, (ny + 7) // 8, (nx + 7) // 8)).astype(np.uint16)
    assert p.eps_map is not None
    _compare(fdtd, p, prec, (1, 2, 13, 64, 30))


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
def test_half_steps_between_windows(fdtd, prec, mode):
    """step_half before, between and after calls in windows: the soft sources'
    last values cross the two copies of the state."""
    p = _problem(mode, 107, 65, 6)

    def halves(g, q):
        for _ in range(1 + q % 2):
            g.step_half(0)
            g.step_half(1)

    _compare(fdtd, p, prec, (13, 64, 15, 1, 70), change=halves)


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_no_memory_for_the_second_copy(fdtd, prec):
    """A grid whose second copy finds no device memory keeps the launches per half
    step; it takes windows once it is changed and there is room."""
    import torch
    n = 9000 if prec == "f32" else 5500  # 1 GB and 1.5 GB of state
    p = _vacuum(P.TM, n, n)
    g = fdtd.Grid.from_problem(p, prec)
    g.step_half(0)
    g.step_half(1)  # the CPML and the DFT buffers
    g.synchronize()
    r = fdtd.Grid.from_problem(p, prec)
    r.set_sweep_kernel("regs")
    r.step_half(0)
    r.step_half(1)
    r.step(20)
    r.synchronize()
    gc.collect()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (500 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert _launches(g, 20) >= 40
        g.synchronize()
    finally:
        del hold
        torch.cuda.empty_cache()
    for q in ("Ez", "Hx", "Hy"):
        assert np.array_equal(g.get(q), r.get(q)) and np.any(r.get(q))
    g.always_window()
    assert _launches(g, 20) < 40
    r.step(20)
    assert np.array_equal(g.get("Ez"), r.get("Ez"))
    g.close()
    r.close()
