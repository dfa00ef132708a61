"""Half steps on a stream of the caller's from the first one on, the CPML not yet
laid out: the values of the same half steps on the grid's own stream."""
import numpy as np
import pytest

from fdtd_b200 import problem as P
from helpers import mode_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("mode", [P.TE, P.TM, P.THREED], ids=["te", "tm", "3d"])
def test_first_half_steps_on_a_caller_stream(fdtd, prec, mode):
    import torch
    shape = (60, 50, 40) if mode == P.THREED else (900, 700, 1)
    p = P.Problem(mode, shape, 1e-6, P.courant_dt(1e-6, 0.98 / np.sqrt(3.0 if mode == P.THREED else 2.0)))
    axes = 3 if mode == P.THREED else 2
    for a in range(axes):
        for s in (0, 1):
            p.pml[(a, s)] = 10
    E, H, _, _ = mode_fields(mode)
    p.sources.append(P.Source("xyz".index(E[-1][1]), (12, 12, 12 if axes == 3 else 0), P.gaussian_pulse(40, 6, 3), "E"))
    stream = torch.cuda.Stream()
    out = []
    for s in (None, stream.cuda_stream):
        g = fdtd.Grid.from_problem(p, prec)
        for _ in range(12):
            g.step_half(0, stream=s)
            g.step_half(1, stream=s)
        stream.synchronize()
        out.append([g.get(n) for n in E + H])
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b) and np.any(a)
