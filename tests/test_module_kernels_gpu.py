"""The module-level solvers at the sizes where their split changes: one row,
one chunk, remainders, one warp to several, the largest system in shared memory
and the first beyond it, several systems; systems that are not diagonally
dominant take the sequential path.  Tolerances: 1e-13 normwise against the
oracle's Thomas and block-Thomas sweeps for dominant systems (both sides err by
a few roundings a row, and errors decay along a dominant system); 1e-10 for the
second-difference matrix (condition number about n^2 / 2 = 2e5 at n = 600)."""
import numpy as np
import pytest
import torch

from kineticeq_b200.cuda_kernel import INV_SQRT_2PI, load_gtsv, load_implicit_fused, load_lo_blocktridiag
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("n,batch", [(1, 1), (2, 3), (3, 5), (31, 2), (96, 7), (97, 2), (288, 3), (289, 2),
                                     (1000, 4), (4608, 2), (4609, 2), (5900, 2), (6100, 2), (9001, 3)])
def test_gtsv_dominant(n, batch):
    rng = np.random.default_rng(n)
    dl, du = rng.uniform(-0.5, 0.5, (2, batch, n))
    d = rng.choice([-1.0, 1.0], (batch, n)) * (1.0 + np.abs(dl) + np.abs(du) * rng.uniform(0.2, 1.0, (batch, n)))
    d = np.sign(d) * np.maximum(np.abs(d), np.abs(dl) + np.abs(du) + 1e-3)
    B = rng.uniform(-1, 1, (batch, n))
    X = load_gtsv().gtsv_strided(_cu(dl), _cu(d), _cu(du), _cu(B)).cpu().numpy()
    assert _rel(X, O.gtsv(dl, d, du, B)) <= 1e-13


def test_gtsv_not_dominant():
    n, batch = 600, 3
    dl, du = -np.ones((2, batch, n))
    d = 2.0 * np.ones((batch, n))
    B = np.random.default_rng(1).uniform(-1, 1, (batch, n))
    d[1] += 1.0  # one dominant system among them
    X = load_gtsv().gtsv_strided(_cu(dl), _cu(d), _cu(du), _cu(B)).cpu().numpy()
    ref = O.gtsv(dl, d, du, B)
    for b in range(batch):
        assert _rel(X[b], ref[b]) <= 1e-10


@pytest.mark.parametrize("n", [1, 2, 9, 10, 19, 288, 289, 4094, 4609, 15500])
def test_block_tridiag(n):
    rng = np.random.default_rng(n)
    A, C = rng.normal(size=(2, 2, n, 3, 3)) * 0.1
    B = np.eye(3) * 2.0 + rng.normal(size=(2, n, 3, 3)) * 0.1
    D = rng.normal(size=(2, n, 3))
    X = load_lo_blocktridiag().block_tridiag_solve(_cu(A), _cu(B), _cu(C), _cu(D)).cpu().numpy()
    for b in range(2):
        assert _rel(X[b], O.block_tridiag_solve(A[b], B[b], C[b], D[b])) <= 1e-13


@pytest.mark.parametrize("nx,nv", [(3, 1), (130, 7), (131, 9), (300, 64)])
def test_build_system(nx, nv):
    rng = np.random.default_rng(nx)
    n, T = rng.uniform(0.1, 2.0, (2, nx))
    nu = rng.uniform(-0.5, 0.5, nx)
    v = np.linspace(-10.0, 10.0, nv) if nv > 1 else np.array([0.5])
    B0 = rng.uniform(0, 1, (nv, nx - 2))
    fl, fr = rng.uniform(0, 1, (2, nv))
    out = [torch.zeros((nv, nx - 2), dtype=torch.float64, device="cuda") for _ in range(4)]
    load_implicit_fused().build_system_from_moments(_cu(B0), _cu(v), 1e-3, 1e-2, 0.1, INV_SQRT_2PI, _cu(n), _cu(nu),
                                                    _cu(T), _cu(fl), _cu(fr), *out)
    u = nu[1:-1] / n[1:-1]
    M = n[1:-1] / np.sqrt(2 * np.pi * T[1:-1]) * np.exp(-(v[:, None] - u) ** 2 / (2 * T[1:-1]))
    it = 1e-3 * n[1:-1] * np.sqrt(T[1:-1]) / 0.1
    al, be = 0.1 * np.maximum(v, 0)[:, None], 0.1 * np.maximum(-v, 0)[:, None]
    B = B0 + it * M
    B[:, :1] += al * fl[:, None]
    B[:, -1:] += be * fr[:, None]
    dl, du = np.broadcast_to(-al, B.shape).copy(), np.broadcast_to(-be, B.shape).copy()
    dl[:, 0], du[:, -1] = 0.0, 0.0
    for got, want in zip(out, (dl, 1.0 + al + be + it, du, B)):
        # exp's argument reaches 400, of which a relative rounding is 1e-13 of M
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-13 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("T", [1.0, 1e-150, 1e-250])
def test_build_system_nearly_empty_cells(T):
    """A cell without density (n clamped to 1e-300) whose momentum is of ordinary
    size has |u| near 1e300 and a Maxwellian of 0; a quotient that overflows (cold
    cells) ends the same way.  Finite, and equal to the oracle's."""
    nx, nv = 40, 16
    rng = np.random.default_rng(3)
    n, Tc = rng.uniform(0.1, 2.0, (2, nx))
    nu = rng.uniform(-0.5, 0.5, nx)
    n[[5, 6, 20]], nu[[5, 6, 20]], Tc[[5, 6, 20]] = (0.0, -1.0, 1e-200), (0.1, -0.2, 0.3), T
    Tc[30], n[30], nu[30] = 1e-190, 1.0, 0.1
    v, B0 = np.linspace(-10.0, 10.0, nv), rng.uniform(0, 1, (nv, nx - 2))
    fl, fr = rng.uniform(0, 1, (2, nv))
    out = [torch.zeros((nv, nx - 2), dtype=torch.float64, device="cuda") for _ in range(4)]
    load_implicit_fused().build_system_from_moments(_cu(B0), _cu(v), 1e-3, 1e-2, 0.1, INV_SQRT_2PI, _cu(n), _cu(nu),
                                                    _cu(Tc), _cu(fl), _cu(fr), *out)
    for got, want in zip(out, O.build_system(B0, v, 1e-3, 1e-2, 0.1, n, nu, Tc, fl, fr)):
        got = got.cpu().numpy()
        assert np.isfinite(want).all() and np.isfinite(got).all()
        assert np.abs(got - want).max() <= 1e-13 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("n", [20, 300, 600, 5000, 9001])
@pytest.mark.parametrize("c", [0.01, 0.2, 0.45])
def test_gtsv_decaying_solutions(n, c):
    """A few sources, from which the solution decays through the whole range of a
    double: each entry is a sum of non-negative terms, so all of them are good to a
    few roundings a row (2e-12 for the 2000 rows at most that an entry comes from)."""
    rng = np.random.default_rng(n)
    dl, du = -c * rng.uniform(0.5, 1.0, (2, 2, n))
    d, B = 1.0 + 0.1 * rng.uniform(0.0, 1.0, (2, n)), np.zeros((2, n))
    B[0, 0], B[0, n // 2], B[1, n - 1] = 1.0, 1e-5, 2.0
    X = load_gtsv().gtsv_strided(_cu(dl), _cu(d), _cu(du), _cu(B)).cpu().numpy()
    ref = O.gtsv(dl, d, du, B)
    m = ref >= 1e-250
    assert np.abs(X[m] / ref[m] - 1.0).max() <= 2e-12


@pytest.mark.parametrize("n", [7, 100, 700, 5000])
@pytest.mark.parametrize("c", [0.01, 0.1])
def test_block_tridiag_decaying_solutions(n, c):
    """The same for blocks with non-negative inverses; an inverse by cofactors
    errs by a few roundings more (1e-11)."""
    rng = np.random.default_rng(n)
    A, C = -c * rng.uniform(0.5, 1.0, (2, n, 3, 3))
    B, D = np.eye(3) - 0.05 * rng.uniform(0.0, 1.0, (n, 3, 3)), np.zeros((n, 3))
    D[0], D[n // 2, 1] = 1.0, 1e-5
    X = load_lo_blocktridiag().block_tridiag_solve(_cu(A), _cu(B), _cu(C), _cu(D)).cpu().numpy()
    ref = O.block_tridiag_solve(A, B, C, D)
    m = ref >= 1e-250
    assert np.abs(X[m] / ref[m] - 1.0).max() <= 1e-11


@pytest.mark.parametrize("n", [5, 40, 400, 5000, 9001])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_right_hand_sides_reach_every_row(n, bad):
    """As in the sequential solves: one NaN or infinity leaves no finite row in its
    system, and the other systems alone."""
    dl, du, d, B = -0.1 * np.ones((3, n)), -0.2 * np.ones((3, n)), np.ones((3, n)), np.ones((3, n))
    B[1, n // 2] = bad
    X = load_gtsv().gtsv_strided(_cu(dl), _cu(d), _cu(du), _cu(B)).cpu().numpy()
    assert np.array_equal(np.isfinite(X), np.array([[True], [False], [True]]) & np.ones((1, n), bool))
    A, C = np.full((2, n, 3, 3), -0.02), np.full((2, n, 3, 3), -0.01)
    Bm, D = np.broadcast_to(np.eye(3), (2, n, 3, 3)).copy(), np.ones((2, n, 3))
    D[0, n // 2, 1] = bad
    X = load_lo_blocktridiag().block_tridiag_solve(_cu(A), _cu(Bm), _cu(C), _cu(D)).cpu().numpy()
    assert not np.isfinite(X[0]).any() and np.isfinite(X[1]).all()


@pytest.mark.parametrize("n", [1, 2, 14, 15, 16, 17])
def test_gtsv_many_small_systems(n):
    """On both sides of the size up to which a thread takes a system: more systems
    than the chip has threads resident, dominant and not."""
    batch = 300001
    rng = np.random.default_rng(n)
    dl, du = rng.uniform(-0.5, 0.5, (2, batch, n))
    d, B = rng.uniform(1.2, 2.0, (batch, n)), rng.uniform(-1, 1, (batch, n))
    d[::7] = rng.uniform(0.9, 1.0, d[::7].shape)
    X = load_gtsv().gtsv_strided(_cu(dl), _cu(d), _cu(du), _cu(B)).cpu().numpy()
    ref = O.gtsv(dl, d, du, B)
    # a pivot is at least 0.9 - 0.25 / 0.62 > 0.49, and half of its neighbours'
    # error is passed on at each row: some ten units of rounding
    assert np.abs(X - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("n,batch", [(16, 9472), (16, 9473), (16, 32767), (23, 32768), (24, 32768), (64, 20000),
                                     (600, 4000), (5000, 300)])
def test_gtsv_many_systems_some_not_dominant(n, batch):
    """Where a call has more systems than a few waves of CTAs, those that are not
    dominant are left to a second kernel."""
    rng = np.random.default_rng(n)
    dl, du = rng.uniform(-0.5, 0.5, (2, batch, n))
    d, B = rng.uniform(1.2, 2.0, (batch, n)), rng.uniform(-1, 1, (batch, n))
    d[::7] = rng.uniform(0.9, 1.0, d[::7].shape)
    d[batch - 1] = 0.95
    X = load_gtsv().gtsv_strided(_cu(dl), _cu(d), _cu(du), _cu(B)).cpu().numpy()
    ref = O.gtsv(dl, d, du, B)
    assert np.abs(X - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("n,batch", [(1, 70001), (12, 1), (12, 5000), (13, 3327), (13, 3328), (32, 8191), (32, 8192),
                                     (33, 8448), (64, 3000)])
def test_block_tridiag_many_small_systems(n, batch):
    """On both sides of the sizes up to which a thread takes a system."""
    rng = np.random.default_rng(n)
    A, C = rng.normal(size=(2, batch, n, 3, 3)) * 0.1
    B = np.eye(3) * 2.0 + rng.normal(size=(batch, n, 3, 3)) * 0.1
    D = rng.normal(size=(batch, n, 3))
    A[:, 0], C[:, n - 1] = np.nan, np.nan  # not read
    X = load_lo_blocktridiag().block_tridiag_solve(_cu(A), _cu(B), _cu(C), _cu(D)).cpu().numpy()
    assert np.isfinite(X).all()
    A[:, 0], C[:, n - 1] = 0.0, 0.0
    for b in np.unique(np.concatenate([[0, batch - 1], rng.integers(0, batch, 100)])):
        assert _rel(X[b], O.block_tridiag_solve(A[b], B[b], C[b], D[b])) <= 1e-13
