"""The staged 3D FP32 sweeps with a plane's groups counted along its rows (rows
that would leave a tenth of the 128-cell tiles empty) against the flat sweeps'
tiles, and the TFSF aux grid at the lengths where its kernel changes."""
import copy

import numpy as np
import pytest

import scenarios
from fdtd_b200 import problem as P
from helpers import mode_fields, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (5, 9, 6), (64, 7, 5), (66, 20, 19), (113, 5, 9), (116, 6, 8),
                                      (132, 21, 17), (256, 6, 7), (257, 18, 5)])
def test_groups_along_rows_match_the_flat_sweeps(fdtd, nx, ny, nz):
    """Per cell both run the same update (their own instantiations, so that a
    product may be contracted differently): 40 steps of FP32 rounding, 6e-8
    each at most, stay within 3e-6 of the field's norm."""
    rng = np.random.default_rng(nx)
    dt = P.courant_dt(1e-6, 0.97 / np.sqrt(3.0))
    p = P.Problem(P.THREED, (nx, ny, nz), 1e-6, dt)
    for a, n in enumerate((nx, ny, nz)):
        for s in (0, 1):
            if n >= 16:
                p.pml[(a, s)] = 3 + s
    p.materials = [P.Material.vacuum(), P.Material.drude(1.0, 0.2 / dt, 0.01 / dt), P.Material.constant(2.2)]
    p.ids = rng.integers(0, 3, size=(nz, ny, nx)).astype(np.uint8)
    c = (nx // 2, ny // 2, nz // 2)
    p.sources += [P.Source(2, c, P.gaussian_pulse(40, 10, 4), "E"), P.Source(0, (1, 1, 1), P.gaussian_pulse(40, 8, 4), "E"),
                  P.Source(1, (nx - 2, ny - 2, nz - 2), P.gaussian_pulse(40, 9, 4), "E")]
    out = []
    for kind in ("auto", "flat"):
        g = fdtd.Grid.from_problem(p, "f32")
        g.set_sweep_kernel(kind)
        g.step(40)
        out.append([g.get(n) for n in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")])
    norm = max(np.linalg.norm(v) for v in out[1][:3])
    hnorm = max(np.linalg.norm(v) for v in out[1][3:])
    for q, (a, b) in enumerate(zip(*out)):
        assert np.linalg.norm(a - b) <= 3e-6 * (norm if q < 3 else hnorm), q


@pytest.mark.parametrize("ncells", [950, 974, 975, 1500, 1998, 1999, 2300])
def test_aux_grid_lengths_match_oracle(fdtd, oracle, ncells):
    """Aux grids of ncells + 50 cells: a cell per thread up to 1024, then windows; FP64, so the fields equal the oracle's within 1e-12."""
    p = copy.deepcopy(scenarios.tm_tfsf_reference_polarisation())
    p.tfsf.aux_ncells = ncells
    # the incident wave starts at the aux grid's low end: bring the box there
    p.tfsf.origin = (p.tfsf.origin[0] + (ncells + 50) / 2 - 40.0, *p.tfsf.origin[1:]) if p.tfsf.k[0] else p.tfsf.origin
    o = oracle.run_oracle(p)
    g = fdtd.Grid.from_problem(p, "f64")
    g.step(p.steps // 2)
    g.step(p.steps - p.steps // 2)
    E, H, _, _ = mode_fields(p.mode)
    for n in E + H:
        assert rel_l2(g.get(n), o.get(n)) <= 1e-12, n


@pytest.mark.parametrize("ncells", [975, 976, 1037, 1038, 1039, 1198, 1200, 2030, 6000])
@pytest.mark.parametrize("calls", [(64, 1, 2, 3), (5, 63, 2, 65)])
def test_aux_windows_match_oracle(fdtd, oracle, ncells, calls):
    """Rows of more than 1024 cells are stepped in windows of 128 cells: lengths
    where the last window ends on the row's last cell and one to each side, calls
    that split into one to 32 steps per launch, single steps between them; FP64,
    so the fields equal the oracle's within 1e-12."""
    p = copy.deepcopy(scenarios.tm_tfsf_reference_polarisation())
    p.tfsf.aux_ncells = ncells
    p.tfsf.origin = (p.tfsf.origin[0] + (ncells + 50) / 2 - 40.0, *p.tfsf.origin[1:]) if p.tfsf.k[0] else p.tfsf.origin
    p.steps = sum(calls)
    o = oracle.run_oracle(p)
    g = fdtd.Grid.from_problem(p, "f64")
    for n in calls:
        g.step(n)
    E, H, _, _ = mode_fields(p.mode)
    for n in E + H:
        assert rel_l2(g.get(n), o.get(n)) <= 1e-12, n
