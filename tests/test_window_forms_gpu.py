"""That the tests' windows are windows: cases in which a grid chooses its launches
by itself, here with windows forced (seen by the launches of a call) and, for the
adjoint, with the kept terms seen by the launches of the forward. Every value
equals that of the launches per half step."""
import numpy as np
import pytest

from fdtd_b200 import problem as P
from helpers import mode_fields
from test_window_dispatch_gpu import _launches
from test_window_gpu import _problem64

pytestmark = pytest.mark.gpu


def _same(a, b):
    assert np.array_equal(a, b, equal_nan=True)
    ok = ~np.isnan(a)
    assert np.array_equal(np.signbit(a[ok]), np.signbit(b[ok]))


@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("eps,mu_r", [(np.inf, 1.0), (1e60, 1.0), (1e-25, 1e-25), (2.0, np.inf), (2.0, 1e60)])
def test_fp64_divisors_at_the_ends_of_the_range(fdtd, mode, eps, mu_r):
    """Divisors whose reciprocals do not give the quotient, zeros of either sign and
    dividends down to the subnormals."""
    nx, ny = 70, 41
    p = _problem64(mode, nx, ny, 5, 0)
    p.tfsf = None
    p.materials = [P.Material.constant(1.5, mu_r), P.Material.constant(eps, mu_r)]
    p.ids = (np.indices((1, ny, nx))[2] % 7 == 3).astype(np.uint8)
    E, H, D, B = mode_fields(mode)
    rng = np.random.default_rng(1)
    v = {n: np.where(rng.random((1, ny, nx)) < 0.5, -0.0, rng.normal(size=(1, ny, nx)) * 10.0 ** rng.integers(-320, 0, size=(1, ny, nx)))
         for n in D + B}
    out = []
    for kind in ("windows", "regs"):
        g = fdtd.Grid.from_problem(p, "f64")
        g.always_window() if kind == "windows" else g.set_sweep_kernel(kind)
        for n, x in v.items():
            g.set(n, x)
        launches = _launches(g, 13)
        assert (launches < 26) == (kind == "windows"), launches
        out.append([g.get(n) for n in E + H + D + B])
        g.close()
    for a, b in zip(*out):
        _same(a, b)


@pytest.mark.parametrize("prec,poles", [("f32", 0), ("f32", 1), ("f64", 0), ("f64", 1)])
@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
def test_caller_streams_without_graphs(fdtd, mode, prec, poles):
    """Eager windows on streams of the caller, another material map between the calls."""
    import torch
    p = _problem64(mode, 150, 101, 4, poles)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    E, H, _, _ = mode_fields(mode)
    out = []
    for kind in ("windows", "regs"):
        g = fdtd.Grid.from_problem(p, prec)
        g.always_window() if kind == "windows" else g.set_sweep_kernel(kind)
        g.use_graphs(False)
        for s, n in zip(streams, (40, 71)):
            before = g.launch_count
            g.step(n, stream=s.cuda_stream)
            s.synchronize()
            assert (g.launch_count - before < 2 * n) == (kind == "windows")
            g.set_material_ids(np.roll(p.ids, 7, axis=2))
        g.step(41)
        out.append([g.get(n) for n in E + H] + [g.dft(h) for h in g.dft_handles])
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b) and np.any(a)


# extents around the windows', steps that end inside a launch and one past whole
# stretches of 64, enough for the wave to reach the probe; design boxes one cell
# wide and across windows; no more values to keep than 8 times the checkpoints
@pytest.mark.parametrize("nx,ny,npml,steps,design", [
    (40, 36, 4, 65, (12, 12, 12, 12)), (64, 32, 3, 129, (20, 10, 40, 20)), (65, 33, 3, 130, (9, 8, 50, 24)),
    (112, 97, 6, 257, (20, 20, 90, 70)), (130, 64, 0, 300, (5, 5, 120, 55)), (620, 470, 8, 200, (270, 200, 350, 280))])
def test_the_adjoint_keeps_its_terms(fdtd, nx, ny, npml, steps, design):
    p = P.Problem(P.TM, (nx, ny, 1), 1e-6, P.courant_dt(1e-6, 0.98 / np.sqrt(2.0)))
    if npml:
        for a in (0, 1):
            for s in (0, 1):
                p.pml[(a, s)] = npml
    x0, y0, x1, y1 = design
    p.eps_map = np.zeros((1, ny, nx))
    p.eps_map[0, y0:y1 + 1, x0:x1 + 1] = np.random.default_rng(nx).uniform(1.0, 8.0, size=(y1 - y0 + 1, x1 - x0 + 1))
    p.sources.append(P.Source(2, (x0, y0, 0), np.sin(2 * np.pi * 0.05 * np.arange(steps)), "E"))
    out = []
    for kind in ("auto", "regs"):
        g = fdtd.Grid.from_problem(p, "f32")
        g.set_sweep_kernel(kind)
        adj = fdtd.Adjoint(g, (x1 + 1, y0, 0), (x1 + 1, min(y0 + 3, ny - 2), 0), 0.05, (x0, y0, 0), (x1, y1, 0), 64)
        before = g.launch_count
        J = adj.forward(steps)
        forward = g.launch_count - before
        grad = adj.backward()
        both = g.launch_count - before
        if kind == "auto":  # several steps per launch each way
            assert forward < steps and both < 2 * steps, (forward, both)
        else:  # E and H of each step; the segments' steps again, and their reverse
            assert forward >= 2 * steps and both >= 6 * steps, (forward, both)
        out.append((J, grad, g.get("Ez"), g.get("Hx")))
        adj.close()
        g.close()
    assert out[0][0] == out[1][0] != 0.0
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b) and np.any(a)
