"""The second copy of a 2D grid's state goes when the grid stops taking windows."""
import pytest

from fdtd_b200 import problem as P
from test_window_gpu import _problem

pytestmark = pytest.mark.gpu


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
