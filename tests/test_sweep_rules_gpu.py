"""3D sweeps at the sizes where the rule of their tiles or of their chained launches
changes (rounds of CTAs on the chip): the FP32 ones counted along the rows against
the flat sweeps, and both precisions replayed from a graph against the same steps
launched one by one, which are chained by other rules."""
import numpy as np
import pytest

from fdtd_b200 import problem as P

pytestmark = pytest.mark.gpu

NAMES = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _problem(nx, ny, nz, box=False, poles=0, dft=False):
    rng = np.random.default_rng(nx)
    dt = P.courant_dt(1e-6, 0.97 / np.sqrt(3.0))
    p = P.Problem(P.THREED, (nx, ny, nz), 1e-6, dt)
    for a, n in enumerate((nx, ny, nz)):
        for s in (0, 1):
            if n >= 16:
                p.pml[(a, s)] = 3 + s
    if poles:
        p.materials = [P.Material.lorentz(1.5, [(1.2, 0.1 / dt, 0.01 / dt), (0.6, 0.2 / dt, 0.02 / dt)])]
    else:
        p.materials = [P.Material.vacuum(), P.Material.drude(1.0, 0.2 / dt, 0.01 / dt), P.Material.constant(2.2)]
        p.ids = rng.integers(0, 3, size=(nz, ny, nx)).astype(np.uint8)
    p.sources += [P.Source(2, (nx // 2, ny // 2, nz // 2), P.gaussian_pulse(40, 10, 4), "E"), P.Source(0, (1, 1, 1), P.gaussian_pulse(40, 8, 4), "E"),
                  P.Source(1, (nx - 2, ny - 2, nz - 2), P.gaussian_pulse(40, 9, 4), "E")]
    if box:
        k = (1.0, 0.0, 0.0)
        p.tfsf = P.TFSF(2 * max(nx, ny, nz), P.gaussian_pulse(120, 30, 8, offset=1.0), (nx / 2, ny / 2, nz / 2), k, (0.0, 0.0, 1.0), (0.0, -1.0, 0.0),
                        P.tfsf_box_planes(P.THREED, (9, 9, 9), (nx - 10, ny - 10, nz - 10)))
    if dft:
        for c in (0, 2, 4):
            p.dfts.append(P.DFTRegion(c, (2, 2, 2), (nx - 3, 2, nz - 3), [0.03]))
            p.dfts.append(P.DFTRegion(c, (2, 2, 2), (2, ny - 3, nz - 3), [0.03]))
    return p


# two tiles to a plane or more, one CTA less along the rows; rows that end inside
# a warp, many planes (a round of CTAs is 1036 of the E sweep, 1184 of the H)
@pytest.mark.parametrize("nx,ny,nz", [(5, 9, 700), (64, 7, 600), (66, 20, 250), (70, 79, 55), (132, 21, 125), (257, 18, 110)])
def test_groups_along_rows_of_more_than_a_round(fdtd, nx, ny, nz):
    """As the smaller grids' test: 40 steps of FP32 rounding, 6e-8 each at most, stay
    within 3e-6 of the field's norm."""
    p = _problem(nx, ny, nz)
    out = []
    for kind in ("auto", "flat"):
        g = fdtd.Grid.from_problem(p, "f32")
        g.set_sweep_kernel(kind)
        g.step(40)
        out.append([g.get(n) for n in NAMES])
        g.close()
    norms = [max(np.linalg.norm(v) for v in out[1][h:h + 3]) for h in (0, 3)]
    for q, (a, b) in enumerate(zip(*out)):
        assert np.linalg.norm(a - b) <= 3e-6 * norms[q // 3] and np.any(a), q


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("kind", ["plain", "box", "dft", "box-dft", "poles", "periodic-dft"])
@pytest.mark.parametrize("nx,ny,nz", [(36, 36, 36), (60, 60, 40), (70, 79, 55), (98, 150, 45), (130, 120, 90)])
def test_replayed_steps_equal_launched_ones(fdtd, prec, kind, nx, ny, nz):
    p = _problem(nx, ny, nz, "box" in kind, kind == "poles", "dft" in kind)
    out = []
    for graphs in (True, False):
        g = fdtd.Grid.from_problem(p, prec)
        g.use_graphs(graphs)
        if "periodic" in kind:
            for a in range(3):
                for s in (0, 1):
                    g.set_boundary(a, s, "periodic")
        g.step(64)
        g.step(64)
        out.append([g.get(n) for n in NAMES] + [g.dft(h) for h in g.dft_handles])
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b) and np.any(a)
