"""The row-block kernel of the HOLO step at the sizes where it can go wrong:
fewer rows than a low-order chunk, one row more than whole chunks, windows that
reach over several chunks, remainders of rows and velocities; flow speeds and
v_max dt/dx on both sides of the bound up to which the low-order windows are
used (2 c |u| / (1 - 2 c |u|) <= 0.074, c = dt / (4 dx)), up to strongly
coupled chunks and to the limit beyond which the look-back kernel runs; against
the CPU oracle with the parity tolerance of the other HOLO tests (1e-12
normwise in f, equal HO and LO iteration counts), and in one plan against
alone, bit for bit."""
import numpy as np
import pytest
import torch

from kineticeq_b200 import _native as N
from kineticeq_b200.plan import HoloPlan, InstanceSpec, holo_params_struct
from kineticeq_b200.schemes.common import maxwellian, region_moments
from kineticeq_b200.state import allocate_state_1d1v
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-12
SP = dict(ho_iter=12, ho_tol=1e-10, lo_iter=40, lo_tol=1e-10)


def _state(nx, nv, u=0.0):
    rng = np.random.default_rng(1000 * nx + nv)
    st = allocate_state_1d1v(nx, nv, 1.0, 10.0, "cuda", torch.float64)
    xd = float(rng.uniform(0.3, 0.7))
    st.n, st.u, st.T = region_moments(st.x, (
        {"x_range": (0.0, xd), "n": float(rng.uniform(0.5, 2)), "u": float(rng.uniform(-0.3, 0.3)) + u,
         "T": float(rng.uniform(0.5, 2))},
        {"x_range": (xd, 1.0), "n": float(rng.uniform(0.1, 0.5)), "u": float(rng.uniform(-0.3, 0.3)) + u,
         "T": float(rng.uniform(0.5, 2))}))
    maxwellian(st, out=st.f)
    return st


def _spec(st, cfl):
    dt = cfl * st.dx / 10.0
    return InstanceSpec(v=st.v, dx=st.dx, dv=st.dv, dt=dt, tau_tilde=10.0 * dt, a=st.f.clone(),
                        b=torch.empty_like(st.f))


def _check(nx, nv, cfl, u=0.0, steps=2, **sp):
    sp = {**SP, **sp}
    st = _state(nx, nv, u)
    dt = cfl * st.dx / 10.0
    plan = HoloPlan([_spec(st, cfl)], holo_params_struct(None, **sp))
    f_o, v, p_o = st.f.cpu().numpy().copy(), st.v.cpu().numpy(), O.holo_params(None, **sp)
    for _ in range(steps):
        plan.step(1)
        bl = O.holo_step(f_o, v, st.dx, st.dv, dt, 10.0 * dt, p_o)
        rec = plan.stats.fetch()[0]
        assert (int(rec["iters"]), int(rec["lo_iters"])) == (bl["ho_iter"], bl["lo_iter"])
        if not np.isfinite(f_o).all():
            return  # the method diverges (v_max dt/dx = 20): no values to compare with
        assert int(rec["status"]) == 0
        f = plan.state(0).cpu().numpy()
        assert np.abs(f - f_o).max() / np.abs(f_o).max() <= TOL


@pytest.mark.parametrize("nx,nv", [(3, 16), (4, 33), (18, 31), (34, 64), (35, 40), (51, 16), (67, 130),
                                   (100, 65), (260, 600), (4000, 34), (9600, 34)])
def test_sizes(nx, nv):
    _check(nx, nv, 0.5)


@pytest.mark.parametrize("cfl,u", [(0.9, 1.4), (0.9, 1.6), (0.9, -3.0), (2.0, 0.0), (4.0, 3.0), (7.0, 0.0), (20.0, 0.0)])
@pytest.mark.parametrize("nx", [5, 99, 500])
def test_speeds_and_steps(nx, cfl, u):
    _check(nx, 96, cfl, u)


@pytest.mark.parametrize("flags", [dict(Con_Terms_do=False), dict(flux_consistency_do=False)])
@pytest.mark.parametrize("u", [0.0, 3.0])
def test_options(flags, u):
    _check(131, 48, 0.9, u, **flags)


def test_one_plan_equals_alone():
    cases = [(35, 33, 0.5, 0.0), (300, 64, 0.9, 3.0), (200, 70, 20.0, 0.0), (130, 48, 0.9, 1.5), (90, 33, 7.0, 0.0)]
    p = holo_params_struct(None, **SP)
    together = HoloPlan([_spec(_state(nx, nv, u), c) for nx, nv, c, u in cases], p)
    together.step(2)
    for b, (nx, nv, c, u) in enumerate(cases):
        alone = HoloPlan([_spec(_state(nx, nv, u), c)], p)
        alone.step(2)
        assert torch.equal(together.state(b).view(torch.int64), alone.state(0).view(torch.int64)), b


@pytest.mark.parametrize("nx,nv", [(200, 64), (700, 300)])
def test_timeout_reported_and_plan_recovers(nx, nv):
    """Spin limit 0: every wait that is not already satisfied gives up at once,
    the launch says so, and the plan steps as a fresh one behind it."""
    p = holo_params_struct(None, **SP)
    ref = HoloPlan([_spec(_state(nx, nv), 0.5)], p)
    ref.step(2)
    plan = HoloPlan([_spec(_state(nx, nv), 0.5)], p)
    plan.set_spin_limit(0)
    for _ in range(3):
        plan.step(1)
        assert int(plan.stats.fetch()[0]["status"]) == N.KEQ_ERR_TIMEOUT
    assert plan.device_error_bits() & (1 << N.KEQ_ERR_TIMEOUT)
    plan.set_spin_limit(1 << 25)
    plan.reset_errors()
    plan.step(1)  # (back to the first buffer as input)
    plan.state(0).copy_(_state(nx, nv).f)
    plan.step(2)
    assert int(plan.stats.fetch()[0]["status"]) == 0
    assert plan.device_error_bits() == 0
    assert torch.equal(plan.state(0), ref.state(0))


@pytest.mark.parametrize("nx,nv", [(40, 33), (300, 64)])
def test_a_nan_is_reported(nx, nv):
    st = _state(nx, nv)
    st.f[nx // 2, nv // 3] = float("nan")
    plan = HoloPlan([_spec(st, 0.5)], holo_params_struct(None, **{**SP, "ho_iter": 4}))
    plan.step(1)
    rec = plan.stats.fetch()[0]
    assert (int(rec["status"]), int(rec["iters"])) == (N.KEQ_ERR_NONFINITE, 4)
    row = plan.state(0)[nx // 2]
    assert torch.isnan(row).all()


@pytest.mark.parametrize("nx,nv,cfl", [(300, 64, 0.5), (700, 300, 0.5), (300, 64, 20.0)])
def test_phase_trace(nx, nv, cfl):
    """A trace has the phases of every HO iteration in order, from both kernels (the
    look-back kernel at v_max dt/dx = 20), and the LO iterations."""
    plan = HoloPlan([_spec(_state(nx, nv), cfl)], holo_params_struct(None, **{**SP, "fixed_ho_iters": 3}))
    plan.step(1)
    plan.enable_trace(64)
    plan.step(1)
    rec = plan.stats.fetch()[0]
    t = plan._trace.cpu().numpy().reshape(16, 16)
    end = 0
    for z in range(3):
        a0, a1, l0, l1, c0, c1, lo = (int(x) for x in t[z, :7])
        assert end < a0 < a1 and a0 < l0 < l1 < c1 and a0 < c0 < c1
        assert 1 <= lo <= SP["lo_iter"]
        assert all(0 < t[z, q] < t[z, q + 1] for q in (8, 10, 12))
        end = c0
    assert lo == int(rec["lo_iters"])
    assert (t[3, [1, 3, 5]] == 0).all()  # as attached: no fourth HO iteration
    assert len(plan.trace_phases()) == 12


@pytest.mark.parametrize("cfl", [6.0, 7.0, 8.0])  # the row-block kernel takes v_max dt/dx up to 6.3
@pytest.mark.parametrize("nx", [99, 500])
def test_both_sides_of_the_largest_step(nx, cfl):
    """The oracle is finite here, so the values are compared."""
    st = _state(nx, 96)
    dt = cfl * st.dx / 10.0
    f_o = st.f.cpu().numpy().copy()
    O.holo_step(f_o, st.v.cpu().numpy(), st.dx, st.dv, dt, 10.0 * dt, O.holo_params(None, **SP))
    assert np.isfinite(f_o).all()
    _check(nx, 96, cfl)


@pytest.mark.parametrize("nx", [99, 500])
def test_divergence_is_reported(nx):
    """At v_max dt/dx = 20 the method diverges: the oracle is not finite, and the step
    says so."""
    st = _state(nx, 96)
    dt = 20.0 * st.dx / 10.0
    f_o = st.f.cpu().numpy().copy()
    bl = O.holo_step(f_o, st.v.cpu().numpy(), st.dx, st.dv, dt, 10.0 * dt, O.holo_params(None, **SP))
    assert not np.isfinite(f_o).all()
    plan = HoloPlan([_spec(st, 20.0)], holo_params_struct(None, **SP))
    plan.step(1)
    rec = plan.stats.fetch()[0]
    assert int(rec["status"]) == N.KEQ_ERR_NONFINITE
    assert (int(rec["iters"]), int(rec["lo_iters"])) == (bl["ho_iter"], bl["lo_iter"])


@pytest.mark.parametrize("tag", [0, 1, 2, 3, 7, 0xFFFFFFFF])
@pytest.mark.parametrize("u", [0.0, 3.0])
def test_whatever_the_workspace_holds(tag, u):
    """The workspace is not initialised, or another plan's: words that look like
    published ones of any iteration change nothing."""
    p = holo_params_struct(None, **SP)
    ref, plan = (HoloPlan([_spec(_state(300, 64, u), 0.9)], p) for _ in range(2))
    word = tag << 32 | 0x3FF00000
    plan._ws[0].view(torch.int64).fill_(word - (1 << 64) if word >= 1 << 63 else word)
    ref.step(3)
    plan.step(3)
    assert torch.equal(plan.state(0), ref.state(0))
