"""2D grids changed between calls in windows: the cells' factors follow the
materials, the block goes when the grid stops taking windows, and work in flight
on a stream of the caller's keeps the materials it was launched with. Every value
equals that of the launches per half step."""
import numpy as np
import pytest

from fdtd_b200 import problem as P
from helpers import mode_fields
from test_window_gpu import _problem, _problem64

pytestmark = pytest.mark.gpu


def _fields(g, p):
    E, H, _, _ = mode_fields(p.mode)
    return [g.get(n) for n in E + H] + [g.dft(h) for h in range(len(g.dft_meta))]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("poles", [0, 1])
def test_changes_between_short_calls(fdtd, prec, mode, poles):
    nx, ny = 150, 101
    p = _problem64(mode, nx, ny, 4, poles)
    rng = np.random.default_rng(5)
    eps = np.where(rng.random((1, ny, nx)) < 0.3, rng.uniform(1.0, 5.0, (1, ny, nx)), 0.0)
    e = 2 if mode == P.TM else 0
    changes = [
        lambda g: g.set_eps_map(eps),
        lambda g: g.add_source(e, (40, 30, 0), P.gaussian_pulse(300, 40, 7), "E"),
        lambda g: g.set_material_ids(np.roll(p.ids, 7, axis=2)),
        lambda g: g.add_dft(e, (3, 3, 0), (60, 3, 0), [0.03]),
        lambda g: g.set_eps_map(None),
        lambda g: g.set_boundary(0, 0, "pec"),
        lambda g: g.set_boundary(0, 0, "none"),
        lambda g: g.set_pml(1, 0, 5),
        lambda g: g.set_materials(p.materials[::-1]),
        lambda g: g.set_material_blocks(3, rng.integers(0, 3, size=(1, (ny + 7) // 8, (nx + 7) // 8)).astype(np.uint16)),
        lambda g: g.set_materials([P.Material.constant(1.5)] * 3),
    ]
    out = []
    for kind in ("windows", "regs"):
        rng = np.random.default_rng(6)
        g = fdtd.Grid.from_problem(p, prec)
        g.always_window() if kind == "windows" else g.set_sweep_kernel(kind)
        for c in changes:
            g.step(13)
            c(g)
        g.step(64)
        out.append(_fields(g, p))
        g.close()
    for q, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b) and np.any(a), (q, float(np.abs(a - b).max()))


def test_the_block_goes_with_the_windows(fdtd):
    p = _problem(P.TE, 300, 200, 4)
    g = fdtd.Grid.from_problem(p, "f32")
    g.step(1)
    without = g.memory_bytes
    g.step(64)
    with_block = g.memory_bytes
    assert with_block - without > 3 * 4 * 300 * 200
    g.set_boundary(0, 0, "pec")
    g.step(2)
    assert g.memory_bytes == without
    g.set_boundary(0, 0, "none")
    g.step(64)
    assert g.memory_bytes == with_block


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_materials_changed_behind_work_in_flight(fdtd, prec):
    """6400 steps are on their way on the caller's stream when an eps map comes."""
    import torch
    p = _problem(P.TM, 256, 256, 4)
    eps = np.where(np.random.default_rng(5).random((1, 256, 256)) < 0.5, 3.0, 0.0)
    s = torch.cuda.Stream()
    out = []
    for wait in (True, False):
        g = fdtd.Grid.from_problem(p, prec)
        g.always_window()
        g.prepare()
        g.step(6400, stream=s.cuda_stream)
        if wait:
            s.synchronize()
        g.set_eps_map(eps)
        g.step(64, stream=s.cuda_stream)
        s.synchronize()
        out.append(_fields(g, p))
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b) and np.any(a)
