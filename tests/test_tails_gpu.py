"""The far tails of a distribution, entry by entry.  Every |x| of a sweep is a sum
of non-negative terms, so each entry, however small, is computed to a few
roundings by the oracle and has to be by the step kernels: what flows into a
block from the blocks upstream may only be left out where it is small against
that entry itself, and no tolerance of the iteration may decide it.

Tolerance 1e-11: a Maxwellian exp(-a), a up to 500 at 1e-217, carries a times the
relative error of its argument, and T of a row carries the roundings of a sum
over the velocities (2e-16 sqrt(nv)); that is 2e-12 at most.  Entries below
1e-200 are left out (2^-1000 of the bound 4e5 n is where a fold ends)."""
import numpy as np
import pytest
import torch

from kineticeq_b200.plan import HoloPlan, ImplicitPlan, InstanceSpec, holo_params_struct, implicit_params_struct
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _problem(nx, nv, cfl, Tl, Tr):
    """Two states side by side, the colder one with tails far below the other's."""
    g = O.Grid(nx, nv)
    f = O.initial_condition(g, ((0.0, 0.5, 1.0, 0.2, Tl), (0.5, 1.0, 0.125, -0.1, Tr)))
    return g, f, cfl * g.dx / 10.0


def _spec(g, f, dt, dt_tau):
    a = torch.from_numpy(f).cuda()
    return InstanceSpec(v=torch.from_numpy(g.v()).cuda(), dx=g.dx, dv=g.dv, dt=dt, tau_tilde=dt / dt_tau, a=a,
                        b=torch.empty_like(a))


def _compare(got, want):
    m = want >= 1e-200
    assert want[m].min() < 1e-40  # there are tails to compare
    assert np.abs(got.cpu().numpy()[m] / want[m] - 1.0).max() <= 1e-11


SIZES = [(256, 128, 0.85, 1.0, 0.1), (256, 128, 0.3, 0.5, 0.3), (1500, 64, 0.3, 0.1, 1.0), (200, 600, 0.85, 0.2, 1.0)]


@pytest.mark.parametrize("sp", [dict(picard_iter=1), dict(picard_iter=60), dict(picard_iter=60, abs_tol=1e-3),
                                dict(picard_iter=60, aa_enable=True, aa_m=4)], ids=str)
@pytest.mark.parametrize("dt_tau", [1e-3, 0.1])
@pytest.mark.parametrize("nx,nv,cfl,Tl,Tr", SIZES)
def test_implicit(nx, nv, cfl, Tl, Tr, dt_tau, sp):
    sp = {"picard_tol": 1e-10, "abs_tol": 1e-16, **sp}
    g, f, dt = _problem(nx, nv, cfl, Tl, Tr)
    p = implicit_params_struct(None, **sp)
    alone = ImplicitPlan([_spec(g, f, dt, dt_tau)], p)
    two = ImplicitPlan([_spec(g, f, dt, dt_tau), _spec(g, f, dt, dt_tau)], p)  # the kernel for several
    for plan in (alone, two):
        plan.step(1)
    O.implicit_step(f, g.v(), g.dx, g.dv, dt, dt / dt_tau, O.implicit_params(None, **sp))
    _compare(alone.state(0), f)
    assert torch.equal(two.state(1), alone.state(0))


@pytest.mark.parametrize("ho_iter", [1, 20])
@pytest.mark.parametrize("nx,nv,cfl,Tl,Tr", SIZES)
def test_holo(nx, nv, cfl, Tl, Tr, ho_iter):
    sp = dict(ho_iter=ho_iter, ho_tol=1e-10, lo_iter=40, lo_tol=1e-10)
    g, f, dt = _problem(nx, nv, cfl, Tl, Tr)
    plan = HoloPlan([_spec(g, f, dt, 0.1)], holo_params_struct(None, **sp))
    plan.step(1)
    O.holo_step(f, g.v(), g.dx, g.dv, dt, 10.0 * dt, O.holo_params(None, **sp))
    _compare(plan.state(0), f)
