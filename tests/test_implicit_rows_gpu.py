"""The row-block kernel of the implicit step at the sizes where it can go
wrong: one row, one block, remainders of rows and velocities, odd velocity
counts, several rounds of blocks per CTA, large v_max dt/dx (down to the
dispatch's limit and beyond it, where the look-back kernel runs), negative
values, a zero absolute tolerance; against the CPU oracle with the parity
tolerance of the other tests (1e-12 normwise in f, equal iteration counts)."""
import ctypes as C

import numpy as np
import pytest
import torch

from kineticeq_b200 import _native as N
from kineticeq_b200.plan import ImplicitPlan, InstanceSpec, implicit_params_struct
from kineticeq_b200.schemes.common import maxwellian, region_moments
from kineticeq_b200.state import allocate_state_1d1v
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-12
SP = dict(picard_iter=60, picard_tol=1e-10, abs_tol=1e-16)


def _state(nx, nv, seed=0):
    rng = np.random.default_rng(1000 * nx + nv + seed)
    st = allocate_state_1d1v(nx, nv, 1.0, 10.0, "cuda", torch.float64)
    xd = float(rng.uniform(0.3, 0.7))
    st.n, st.u, st.T = region_moments(st.x, (
        {"x_range": (0.0, xd), "n": float(rng.uniform(0.5, 2)), "u": float(rng.uniform(-0.5, 0.5)),
         "T": float(rng.uniform(0.5, 2))},
        {"x_range": (xd, 1.0), "n": float(rng.uniform(0.05, 0.5)), "u": float(rng.uniform(-0.5, 0.5)),
         "T": float(rng.uniform(0.5, 2))}))
    maxwellian(st, out=st.f)
    return st


def _spec(st, cfl, tau):
    return InstanceSpec(v=st.v, dx=st.dx, dv=st.dv, dt=cfl * st.dx / 10.0, tau_tilde=tau, a=st.f,
                        b=torch.empty_like(st.f))


def _check(st, cfl, dt_tau, steps=2, **sp):
    sp = {**SP, **sp}
    dt = cfl * st.dx / 10.0
    tau = dt / dt_tau
    f_o, v = st.f.cpu().numpy().copy(), st.v.cpu().numpy()
    plan = ImplicitPlan([_spec(st, cfl, tau)], implicit_params_struct(None, **sp))
    p_o = O.implicit_params(None, **{k: x for k, x in sp.items() if k != "tile_rows"})
    for _ in range(steps):
        plan.step(1)
        bl = O.implicit_step(f_o, v, st.dx, st.dv, dt, tau, p_o)
        rec = plan.stats.fetch()[0]
        assert int(rec["status"]) == 0
        assert int(rec["iters"]) == bl["picard_iter"]
        f = plan.state(0).cpu().numpy()
        assert np.abs(f - f_o).max() / np.abs(f_o).max() <= TOL


@pytest.mark.parametrize("aa", [False, True])
@pytest.mark.parametrize("nx,nv", [(3, 2), (4, 33), (9, 31), (10, 64), (11, 97), (35, 65), (131, 130),
                                   (260, 600), (600, 40), (5000, 34)])
def test_sizes(nx, nv, aa):
    _check(_state(nx, nv), 0.3, 0.1, aa_enable=aa, aa_m=4)


@pytest.mark.parametrize("rows", [0, 8, 32])
@pytest.mark.parametrize("cfl", [1e-3, 0.9, 2.9, 6.0, 40.0])
def test_cfl(cfl, rows):
    _check(_state(333, 70), cfl, 0.1, tile_rows=rows)


@pytest.mark.parametrize("conv", ["f", "w"])
@pytest.mark.parametrize("dt_tau", [1e-4, 2.0])
def test_convergence_types(conv, dt_tau):
    _check(_state(200, 48), 0.5, dt_tau, conv_type=conv, aa_enable=conv == "w", aa_m=7)


def test_negative_values():
    st = _state(150, 66)
    st.f[40:60, 5:30] -= 1e-3
    _check(st, 0.8, 0.05)


def test_zero_abs_tol():
    _check(_state(64, 40), 0.2, 0.05, abs_tol=0.0)


def test_instances_of_both_kernels_in_one_plan_equal_alone():
    sizes = [(200, 64, 0.4), (90, 33, 60.0), (400, 128, 1.5), (64, 32, 30.0)]
    specs, alone = [], []
    for nx, nv, cfl in sizes:
        st = _state(nx, nv)
        f0 = st.f.clone()
        p = ImplicitPlan([_spec(st, cfl, 1e-3)], implicit_params_struct(None, **SP))
        p.step(2)
        alone.append(p.state(0).clone())
        st.f = f0
        specs.append(_spec(st, cfl, 1e-3))
    plan = ImplicitPlan(specs, implicit_params_struct(None, **SP))
    mask = torch.ones(len(sizes), dtype=torch.int32, device="cuda")
    plan.set_enable_mask(mask)
    plan.step(2)
    for i in range(len(sizes)):
        assert torch.equal(plan.state(i), alone[i]), i
    before = plan.state(1).clone()
    mask[1] = 0
    mask[2] = 0
    plan.step(1)
    assert torch.equal(plan.other(1), before)


@pytest.mark.parametrize("aa_m", [1, 3, 7])
@pytest.mark.parametrize("stride,start", [(1, 1), (1, 5), (2, 2), (3, 1), (7, 4)])
def test_anderson_calls_with_gaps(aa_m, stride, start):
    """Calls that follow on one another keep older Gram entries; calls behind a
    gap, or behind a late start, form them all."""
    _check(_state(200, 70), 0.5, 0.5, aa_enable=True, aa_m=aa_m, aa_stride=stride, aa_start_iter=start)


@pytest.mark.parametrize("nx,nv", [(150, 66), (700, 300)])
def test_single_plan_masked_launches_and_graph_replays(nx, nv):
    """A plan of one instance counts its launches on the device: masked launches,
    which do nothing, and graph replays leave the same state as plain steps."""
    p = implicit_params_struct(None, **SP)
    make = lambda: ImplicitPlan([_spec(_state(nx, nv), 0.4, 1e-3)], p)  # noqa: E731
    ref, masked, graph = make(), make(), make()
    ref.step(7)
    mask = torch.ones(1, dtype=torch.int32, device="cuda")
    masked.set_enable_mask(mask)
    for n, off in ((1, 2), (2, 4), (3, 0)):
        masked.step(n)
        mask.zero_()
        masked.step(off)  # (an even number, so that the buffers keep their roles)
        mask.fill_(1)
    masked.step(1)
    assert torch.equal(masked.state(0), ref.state(0))
    graph.step(1)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        graph.step(2)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(graph.state(0), ref.state(0))


@pytest.mark.parametrize("conv", ["f", "w"])
@pytest.mark.parametrize("nx,nv", [(30, 40), (200, 70), (90, 600)])
def test_a_nan_stays_and_spreads_as_in_the_oracle(nx, nv, conv):
    """One NaN makes its row's moments NaN, hence the whole row and what lies
    downstream; the iteration neither converges nor loses it."""
    st = _state(nx, nv)
    st.f[nx // 2, nv // 3] = float("nan")
    sp = {**SP, "picard_iter": 6, "conv_type": conv}
    plan = ImplicitPlan([_spec(st, 0.3, 1e-3)], implicit_params_struct(None, **sp))
    f_o = st.f.cpu().numpy().copy()
    O.implicit_step(f_o, st.v.cpu().numpy(), st.dx, st.dv, 0.3 * st.dx / 10.0, 1e-3, O.implicit_params(None, **sp))
    plan.step(1)
    rec = plan.stats.fetch()[0]
    assert (int(rec["status"]), int(rec["iters"])) == (5, 6)
    assert np.array_equal(np.isnan(plan.state(0).cpu().numpy()), np.isnan(f_o))


def test_overflow_is_reported():
    """An under-resolved grid on which the Picard iteration diverges: the oracle
    overflows to NaN, and so does the step."""
    st = _state(11, 9)
    dt_tau = 0.5
    sp = {**SP, "picard_iter": 200, "conv_type": "w"}
    f_o, dt = st.f.cpu().numpy().copy(), 0.05 * st.dx / 10.0
    f_o[:], v = np.exp(-8.0 * (st.v.cpu().numpy() - 0.1) ** 2)[None, :] + 1e-30, st.v.cpu().numpy()
    st.f.copy_(torch.from_numpy(f_o))
    plan = ImplicitPlan([_spec(st, 0.05, dt / dt_tau)], implicit_params_struct(None, **sp))
    O.implicit_step(f_o, v, st.dx, st.dv, dt, dt / dt_tau, O.implicit_params(None, **sp))
    plan.step(1)
    assert (int(plan.stats.fetch()[0]["status"]) == 5) == (not np.isfinite(f_o).all())


def test_divergence_is_reported():
    """The same problem: the oracle is not finite, and the step says so."""
    st = _state(11, 9)
    sp = {**SP, "picard_iter": 200, "conv_type": "w"}
    v, dt = st.v.cpu().numpy(), 0.05 * st.dx / 10.0
    f_o = np.tile(np.exp(-8.0 * (v - 0.1) ** 2) + 1e-30, (11, 1))
    st.f.copy_(torch.from_numpy(f_o))
    plan = ImplicitPlan([_spec(st, 0.05, dt / 0.5)], implicit_params_struct(None, **sp))
    O.implicit_step(f_o, v, st.dx, st.dv, dt, dt / 0.5, O.implicit_params(None, **sp))
    plan.step(1)
    assert not np.isfinite(f_o).all()
    assert int(plan.stats.fetch()[0]["status"]) == 5


@pytest.mark.parametrize("nx,nv,cfl", [(333, 70, 0.3), (26, 33, 0.9), (27, 40, 2.9), (4000, 300, 0.5), (333, 70, 40.0)])
@pytest.mark.parametrize("aa", [False, True])
def test_blocks_of_24_rows(nx, nv, cfl, aa):
    _check(_state(nx, nv), cfl, 0.1, tile_rows=24, aa_enable=aa, aa_m=4)


@pytest.mark.parametrize("tag", [0, 1, 2, 3, 7, 0xFFFFFFFF])
@pytest.mark.parametrize("nx,nv,aa", [(200, 64, False), (700, 300, False), (300, 70, True), (700, 300, True)])
def test_whatever_the_workspaces_hold(nx, nv, aa, tag):
    """One buffer for one call after another, plan and instance workspace in it, as
    keq_implicit_step has it: filled with words that look like published ones of any
    iteration, or left by a call of another size."""
    p = implicit_params_struct(None, aa_enable=aa, aa_m=4, **SP)
    lib = N.load()
    st, other = _state(nx, nv), _state(150, 200)
    grids = [N.Grid(s.f.shape[0], s.f.shape[1], s.dx, s.dv, s.v.data_ptr(), -1, 0.0) for s in (st, other)]
    nb = C.c_size_t(0)
    need = 0
    for g in grids:
        N.check(lib.keq_implicit_workspace_size(C.byref(g), C.byref(p), C.byref(nb)), "size")
        need = max(need, nb.value)
    ws = torch.empty((need + 7) // 8, dtype=torch.int64, device="cuda")
    word = tag << 32 | 0x3FF00000
    ws.fill_(word - (1 << 64) if word >= 1 << 63 else word)
    stats = torch.zeros(N.STATS_BYTES, dtype=torch.uint8, device="cuda")
    outs = []
    for s, g in ((st, grids[0]), (other, grids[1]), (st, grids[0])):
        out = torch.empty_like(s.f)
        N.check(lib.keq_implicit_step(C.byref(g), 0.4 * s.dx / 10.0, 1e-3, C.byref(p), s.f.data_ptr(), out.data_ptr(),
                                      stats.data_ptr(), ws.data_ptr(), ws.numel() * 8, N.stream_handle()), "step")
        outs.append(out)
    plan = ImplicitPlan([_spec(st, 0.4, 1e-3)], p)
    plan.step(1)
    assert torch.equal(outs[0], plan.state(0)) and torch.equal(outs[2], plan.state(0))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("its", [1, 2])
@pytest.mark.parametrize("conv", ["f", "w"])
@pytest.mark.parametrize("nx,nv,cfl", [(5000, 34, 0.05), (3000, 100, 0.05), (2000, 300, 0.3), (1200, 64, 0.02)])
def test_non_finite_values_reach_everything_downstream(nx, nv, cfl, conv, its, bad):
    """One such value makes its row's moments NaN, hence the whole row and, in the
    same sweep and however far away, all that lies downstream of it; then no row has
    finite moments."""
    st = _state(nx, nv)
    row = nx // 2
    st.f[row, nv // 3] = bad
    p = implicit_params_struct(None, **{**SP, "picard_iter": its, "conv_type": conv})
    alone = ImplicitPlan([_spec(st, cfl, 1e-3)], p)
    two = ImplicitPlan([InstanceSpec(**{**vars(_spec(st, cfl, 1e-3)), "a": st.f.clone()}) for _ in range(2)], p)
    finite = np.zeros((nx, nv), bool)
    finite[[0, -1]] = True  # boundary rows stay as they are
    if its == 1:
        pos = st.v.cpu().numpy() > 0.0
        finite[:row, pos] = True
        finite[row + 1:, ~pos] = True
    for plan in (alone, two):
        plan.step(1)
        assert int(plan.stats.fetch()[0]["status"]) == 5
        assert np.array_equal(np.isfinite(plan.state(0).cpu().numpy()), finite)


@pytest.mark.parametrize("aa", [False, True])
@pytest.mark.parametrize("rows", [0, 8, 24, 32])
@pytest.mark.parametrize("mixed", [False, True])
def test_instances_of_one_and_two_velocity_tiles_equal_alone(mixed, rows, aa):
    """They run in CTAs of two warps: whole plans of them, and those of a plan that is
    long enough for two launches (blocks of 8 rows; with taller ones the same plan
    makes one launch)."""
    sp = dict(SP, picard_iter=8, aa_enable=aa, aa_m=3, tile_rows=rows)
    shapes = [(3, 2), (34, 31), (35, 32), (200, 33), (331, 64), (90, 63)]
    n_of_each = 1
    if mixed:
        shapes, n_of_each = [(1500, 33), (1700, 64), (700, 20), (1100, 66), (900, 130)], 8
    p = implicit_params_struct(None, **sp)
    states, alone = [], []
    for nx, nv in shapes:
        st = _state(nx, nv)
        f0 = st.f.clone()
        one = ImplicitPlan([_spec(st, 0.5, 1e-3)], p)
        one.step(2)
        alone.append(one.state(0).clone())
        st.f = f0
        states.append(st)
    specs = []
    for _ in range(n_of_each):
        for st in states:
            specs.append(InstanceSpec(v=st.v, dx=st.dx, dv=st.dv, dt=0.5 * st.dx / 10.0, tau_tilde=1e-3,
                                      a=st.f.clone(), b=torch.empty_like(st.f)))
    plan = ImplicitPlan(specs, p)
    mask = torch.ones(len(specs), dtype=torch.int32, device="cuda")
    plan.set_enable_mask(mask)
    plan.step(2)
    for i in range(len(specs)):
        assert torch.equal(plan.state(i), alone[i % len(shapes)]), i
    off = [0, len(specs) - 1]
    before = [plan.state(i).clone() for i in off]
    mask[off] = 0
    plan.step(1)
    for i, b in zip(off, before):
        assert torch.equal(plan.other(i), b), i
