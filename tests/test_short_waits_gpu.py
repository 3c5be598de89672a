"""Waits of every length: with a limit of a few polls some waits of a step give up
and others do not, and where that happens depends on timing.  Whatever gives up, a
step that reports what a step with full waits reports (success; or that the method
diverges, as it does for one of the HOLO cases) has the same state, and one that
does not says so in its status and in the plan's error bits.  (A wait that gives up returns; the launch
ends by itself and the next one is a fresh one.)"""
import pytest
import torch

from kineticeq_b200 import _native as N
from kineticeq_b200.plan import HoloPlan, ImplicitPlan, InstanceSpec, holo_params_struct, implicit_params_struct
from oracle import oracle as O

pytestmark = pytest.mark.gpu
LIMITS = [0, 1, 2, 3, 5, 8, 13, 21, 34, 55, 90, 150, 250, 400, 700, 1200, 2000, 4000, 8000, 1 << 25]


def _plan(cls, params, sizes, cfl, u):
    specs = []
    for nx, nv in sizes:
        g = O.Grid(nx, nv)
        f = O.initial_condition(g, ((0.0, 0.5, 1.0, u, 1.0), (0.5, 1.0, 0.125, u - 0.1, 0.8)))
        a = torch.from_numpy(f).cuda()
        dt = cfl * g.dx / 10.0
        specs.append(InstanceSpec(v=torch.from_numpy(g.v()).cuda(), dx=g.dx, dv=g.dv, dt=dt, tau_tilde=10.0 * dt, a=a,
                                  b=torch.empty_like(a)))
    return cls(specs, params)


def _check(make):
    ref = make()
    f0 = [ref.state(b).clone() for b in range(ref.n)]
    ref.step(1)
    want = [ref.state(b).clone() for b in range(ref.n)]
    full = [int(r["status"]) for r in ref.stats.fetch()]
    assert N.KEQ_ERR_TIMEOUT not in full and ref.device_error_bits() == 0
    plan = make()
    codes = set()
    for limit in LIMITS:
        for _ in range(3):
            plan.set_spin_limit(limit)
            plan.reset_errors()
            for b in range(plan.n):
                plan.state(b).copy_(f0[b])
                plan.other(b).fill_(-1.0)
            plan.step(1)
            bits = plan.device_error_bits()
            for b, rec in enumerate(plan.stats.fetch()):
                code = int(rec["status"])
                codes.add(code)
                assert code in (full[b], N.KEQ_ERR_TIMEOUT)
                if code == full[b]:  # (compared as bits: a NaN equals itself)
                    assert torch.equal(plan.state(b).view(torch.int64), want[b].view(torch.int64)), (limit, b)
                else:
                    assert bits & (1 << N.KEQ_ERR_TIMEOUT), (limit, b)
    assert codes == {*full, N.KEQ_ERR_TIMEOUT}


@pytest.mark.parametrize("sizes", [[(300, 64)], [(700, 300)], [(300, 64), (90, 200), (700, 100)]])
@pytest.mark.parametrize("sp", [dict(), dict(conv_type="w"), dict(aa_enable=True, aa_m=4), dict(fixed_iters=1)], ids=str)
def test_implicit(sizes, sp):
    p = implicit_params_struct(None, **{"picard_iter": 40, "picard_tol": 1e-10, "abs_tol": 1e-16, **sp})
    _check(lambda: _plan(ImplicitPlan, p, sizes, 0.5, 0.2))


@pytest.mark.parametrize("sizes", [[(300, 64)], [(2000, 100)], [(300, 64), (90, 200)]])
@pytest.mark.parametrize("cfl,u", [(0.5, 0.2), (0.9, 3.0), (4.0, 3.0)])  # LO windows, PCR chunks, coupled chunks
def test_holo(sizes, cfl, u):
    p = holo_params_struct(None, ho_iter=12, ho_tol=1e-10, lo_iter=40, lo_tol=1e-10)
    _check(lambda: _plan(HoloPlan, p, sizes, cfl, u))
