"""Batches whose first call of a length is issued while another batch's steps are
in flight: the work lists that such a call lays out are in place before its
launches read them, and every grid ends as when each call is waited for."""
import numpy as np
import pytest

from fdtd_b200 import problem as P

pytestmark = pytest.mark.gpu


def _batch(fdtd, mode, n, seed, depth):
    rng = np.random.default_rng(seed)
    grids = []
    for nx, ny in rng.integers(150, 460, size=(n, 2)):
        nx, ny = int(nx), int(ny)
        p = P.Problem(mode, (nx, ny, 1), 1e-6, P.courant_dt(1e-6, 0.98 / np.sqrt(2.0)))
        for a in (0, 1):
            for s in (0, 1):
                p.pml[(a, s)] = 8
        p.materials = [P.Material.vacuum(), P.Material.constant(3.0)]
        p.ids = (rng.random((1, ny, nx)) < 0.3).astype(np.uint8)
        e = 2 if mode == P.TM else 0
        p.sources.append(P.Source(e, (nx // 2, ny // 3, 0), P.gaussian_pulse(400, 20, 7), "E"))
        grids.append(fdtd.Grid.from_problem(p, "f32"))
    b = fdtd.Batch(grids)
    if depth is None:
        b.configure(False, 4)
    else:
        b.set_temporal(depth)
    return b


def _fields(b, mode):
    return [g.get(n) for g in b.grids for n in (("Ez", "Hx") if mode == P.TM else ("Ex", "Hz"))]


@pytest.mark.parametrize("mode", [P.TE, P.TM], ids=["te", "tm"])
@pytest.mark.parametrize("depth", [4, 2, None])
def test_first_calls_behind_another_batch(fdtd, mode, depth):
    import torch
    plane = torch.empty(460 * 460, dtype=torch.float32, device="cuda")
    calls = (43, 61, 30, 22)  # in windows each has launches of a length of its own
    out = []
    for wait in (True, False):
        busy, b = _batch(fdtd, mode, 30, 1, 4), _batch(fdtd, mode, 12, 2, depth)
        busy.step(200)
        for g in busy.grids:
            g.synchronize()
        for n in calls:
            busy.step(200)
            for g in busy.grids:  # the members' streams wait for the batch
                g.copy_plane("Ez" if mode == P.TM else "Hz", 0, plane.data_ptr(), False)
            if wait:
                for g in busy.grids:
                    g.synchronize()
            b.step(n)
            if wait:
                for g in b.grids:
                    g.synchronize()
        for g in b.grids + busy.grids:
            g.synchronize()
        out.append(_fields(b, mode))
        for x in (busy, b):
            grids = x.grids
            assert x.error_flags() == 0
            x.close()
            for g in grids:
                g.close()
    for a, c in zip(*out):
        assert np.array_equal(a, c) and np.any(a)


@pytest.mark.parametrize("change", [lambda b: b.set_item_rows([4 * (1 + q % 2) for q in range(len(b.grids))]), lambda b: b.configure(False, 8),
                                    lambda b: b.set_temporal(3)], ids=["item_rows", "configure", "temporal"])
def test_set_up_behind_steps_on_a_caller_stream(fdtd, change):
    """The launch mode of a batch set while its steps are in flight on a stream of
    the caller's: the lists and arguments that those read stay until they are done."""
    import torch
    s = torch.cuda.Stream()
    out = []
    for wait in (True, False):
        b = _batch(fdtd, P.TE, 12, 3, None)
        b.step(150, stream=s.cuda_stream)
        if wait:
            s.synchronize()
        change(b)
        b.step(50, stream=s.cuda_stream)
        s.synchronize()
        out.append(_fields(b, P.TE))
        grids = b.grids
        b.close()
        for g in grids:
            g.close()
    for a, c in zip(*out):
        assert np.array_equal(a, c) and np.any(a)
