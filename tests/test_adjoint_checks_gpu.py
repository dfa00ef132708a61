"""What fdtd_adjoint_forward requires of the grid is asked when it runs, not
only when the adjoint is created: a pending E half step, and what create
refuses, added to the grid in between, are refused on the host before any
launch, whichever way the forward would take its steps."""
import numpy as np
import pytest

from fdtd_b200 import problem as P

pytestmark = pytest.mark.gpu

INVALID, UNSUPPORTED = -1, -3


def _created(fdtd, kind):
    nx, ny = 72, 60
    dt = P.courant_dt(1e-6, 0.98 / np.sqrt(2.0))
    p = P.Problem(P.TM, (nx, ny, 1), 1e-6, dt)
    for a in (0, 1):
        for s in (0, 1):
            p.pml[(a, s)] = 6
    p.sources.append(P.Source(2, (12, 20, 0), np.sin(0.3 * np.arange(70)), "E"))
    g = fdtd.Grid.from_problem(p, "f32")
    g.set_sweep_kernel(kind)
    return p, g, fdtd.Adjoint(g, (50, 20), (50, 23), 0.05, (25, 20), (40, 35), 16)


@pytest.mark.parametrize("kind", ["auto", "regs"])
def test_forward_refuses_a_pending_half_step(fdtd, kind):
    _, g, adj = _created(fdtd, kind)
    g.step_half(0)
    ez = g.get("Ez")
    with pytest.raises(fdtd.FdtdError) as e:
        adj.forward(70)
    assert e.value.code == INVALID
    assert g.step_count == 0 and np.array_equal(g.get("Ez"), ez)


def _add_plane(p, g):
    v = P.gaussian_pulse(80, 20, 8, offset=1.0)
    g.add_tfsf_plane(0, 0, (20, 15, 0), (20, 44, 0), (36.0, 30.0, 0.0), (1.0, 0.0, 0.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0), 72, v)


def _add_poles(p, g):
    g.set_materials([P.Material.drude(1.0, 0.2 / p.dt, 0.01 / p.dt)])


def _add_mu(p, g):
    g.set_materials([P.Material.constant(1.0, 2.0)])


def _add_boundary(p, g):
    g.set_boundary(0, 0, "pec")


def _add_flux_source(p, g):
    g.add_source(2, (30, 25, 0), np.ones(20), "D")


def _widen_cpml(p, g):
    g.set_pml(0, 0, 26)


@pytest.mark.parametrize("kind", ["auto", "regs"])
@pytest.mark.parametrize("change", [_add_plane, _add_poles, _add_mu, _add_boundary, _add_flux_source, _widen_cpml])
def test_forward_refuses_what_create_refuses(fdtd, kind, change):
    p, g, adj = _created(fdtd, kind)
    change(p, g)
    with pytest.raises(fdtd.FdtdError) as e:
        adj.forward(70)
    assert e.value.code == UNSUPPORTED and g.step_count == 0


@pytest.mark.parametrize("kind", ["auto", "regs"])
def test_backward_refuses_a_cpml_laid_out_anew(fdtd, kind):
    """A CPML set after the forward, and its integrators laid out (reading one
    does): the checkpoints and the adjoint state belong to the old ones."""
    _, g, adj = _created(fdtd, kind)
    adj.forward(70)
    g.set_pml(0, 0, 3)
    g.get(fdtd.PSI_NAMES[2 * 3 + 0])
    with pytest.raises(fdtd.FdtdError) as e:
        adj.backward()
    assert e.value.code == INVALID
