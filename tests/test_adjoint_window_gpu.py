"""The adjoint in windows (the forward keeps the design cells' curl terms, the
backward reverses several steps per launch) against the checkpointed adjoint
with launches per half step, which a sweep kernel set by hand brings: the same
arithmetic per cell, so J and every gradient value are equal. (Checkpoints every
64 steps, so that both fold their DFT samples 64 at a time.)"""
import numpy as np
import pytest

from fdtd_b200 import problem as P

pytestmark = pytest.mark.gpu


def _gradients(fdtd, p, probe, design, ckpt):
    out = []
    for kind in ("auto", "regs"):
        g = fdtd.Grid.from_problem(p, "f32")
        g.set_sweep_kernel(kind)
        adj = fdtd.Adjoint(g, *probe, 0.05, *design, ckpt)
        J = adj.forward(p.steps)
        out.append((J, adj.backward(), g.get("Ez"), g.get("Hx")))
        adj.close()
    return out


# extents around the windows' (64 columns, 32 rows) and a grid of many; steps
# that end inside a launch and one past whole stretches of 64; design boxes
# one cell wide, and across windows; in the two of few steps on wide boxes the
# wave does not reach the probe and every value is zero
@pytest.mark.parametrize("nx,ny,npml,steps,design", [
    (40, 36, 4, 65, (12, 12, 12, 12)), (64, 32, 3, 40, (20, 10, 40, 20)), (65, 33, 3, 130, (9, 8, 50, 24)),
    (112, 97, 6, 129, (20, 20, 90, 70)), (130, 64, 0, 33, (5, 5, 120, 55)), (620, 470, 8, 70, (270, 200, 350, 280)),
    (130, 64, 0, 300, (5, 5, 120, 55)), (620, 470, 8, 200, (270, 200, 350, 280))])
def test_stored_adjoint_equals_the_checkpointed_one(fdtd, nx, ny, npml, steps, design):
    rng = np.random.default_rng(nx)
    dt = P.courant_dt(1e-6, 0.98 / np.sqrt(2.0))
    p = P.Problem(P.TM, (nx, ny, 1), 1e-6, dt)
    if npml:
        for a in (0, 1):
            for s in (0, 1):
                p.pml[(a, s)] = npml
    x0, y0, x1, y1 = design
    eps = np.zeros((1, ny, nx))
    eps[0, y0:y1 + 1, x0:x1 + 1] = rng.uniform(1.0, 8.0, size=(y1 - y0 + 1, x1 - x0 + 1))
    p.eps_map = eps
    v = np.sin(2 * np.pi * 0.05 * np.arange(steps))
    p.sources += [P.Source(2, (x0, y0, 0), v, "E"), P.Source(2, (npml + 2, 1, 0), 0.3 * v, "E", hi=(npml + 2, ny - 2, 0))]
    p.steps = steps
    probe = ((x1 + 1, y0, 0), (x1 + 1, min(y0 + 3, ny - 2), 0))
    a, b = _gradients(fdtd, p, probe, ((x0, y0, 0), (x1, y1, 0)), 64)
    assert a[0] == b[0]
    for x, y in zip(a[1:], b[1:]):
        assert np.array_equal(x, y)
