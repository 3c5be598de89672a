"""Device math helpers against CUDA's own exp and IEEE division."""
import numpy as np
import pytest
import torch

from kineticeq_b200 import _native as N

pytestmark = pytest.mark.gpu


def _run(kind, x):
    lib = N.load()
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    N.check(lib.keq_math_selftest(kind, xd.data_ptr(), yd.data_ptr(), xd.numel(), N.stream_handle()),
            "selftest")
    return yd


def ulp_err(a, b):
    a = a.cpu().numpy() if hasattr(a, "cpu") else a
    b = b.cpu().numpy() if hasattr(b, "cpu") else b
    return np.abs(a - b) / np.spacing(np.maximum(np.abs(b), np.finfo(np.float64).tiny))


def test_exp_nonpos_matches_cuda_exp():
    rng = np.random.default_rng(11)
    x = np.concatenate([-rng.uniform(0, 1, 200000), -rng.uniform(0, 40, 200000),
                        -rng.uniform(0, 745, 200000), -np.logspace(-300, 2.8, 20000),
                        np.array([0.0, -0.0, -1e-320, -708.39, -708.4, -744.0, -745.1, -746.0, -1e300])])
    y = _run(0, x)
    ref = torch.exp(torch.from_numpy(x).cuda())
    normal = ref.cpu().numpy() >= np.finfo(np.float64).tiny
    assert ulp_err(y, ref)[normal].max() <= 2.0
    # subnormal results: absolute agreement within one subnormal step
    assert np.abs((y - ref).cpu().numpy()[~normal]).max() <= 2 * 4.9407e-324
    assert torch.isnan(_run(0, np.array([np.nan])))[0]
    assert _run(0, np.array([-np.inf]))[0].item() == 0.0


def test_recip_ge1_matches_division():
    rng = np.random.default_rng(12)
    x = np.concatenate([1.0 + rng.uniform(0, 1, 200000), 10 ** rng.uniform(0, 30, 200000),
                        np.array([1.0, 2.0, 3.0, 1e38, 3e38])])
    y = _run(1, x)
    assert ulp_err(y, 1.0 / x).max() <= 1.0


# ---- helpers of the row-block kernels, against 80-bit arithmetic -----------------
def _ulp80(y, ref):
    """Error in units of the last place of the 80-bit reference's double."""
    return np.abs(y.cpu().numpy().astype(np.longdouble) - ref) / np.spacing(np.abs(ref).astype(np.float64))


def _values(seed, lo, hi, n=200000):
    return 10.0 ** np.random.default_rng(seed).uniform(lo, hi, n)


def test_exp_neg():
    """Below one unit: half of it is the last rounding, a sixth the one before it
    (|r| <= ln 2 / 2), the rest the argument's and the polynomial's."""
    rng = np.random.default_rng(21)
    x = np.concatenate([-rng.uniform(0, 1, 200000), -rng.uniform(0, 40, 200000), -rng.uniform(0, 707, 200000),
                        -np.logspace(-300, 2.84, 20000), [0.0, -0.0, -1e-320]])
    assert _ulp80(_run(2, x), np.exp(x.astype(np.longdouble))).max() <= 1.0
    far = np.array([-708.4, -744.0, -746.0, -1e6, -1e300, -np.inf])
    assert (_run(2, far).cpu().numpy() <= 2.0 ** -1021).all()
    assert (_run(2, far[1:]) == 0.0).all()


def test_recip3():
    """One rounding, and 2^-60 in front of it (2^-6 units at most)."""
    x = np.concatenate([1.0 + np.random.default_rng(22).uniform(0, 1, 200000), _values(23, -270, 270),
                        -_values(24, -30, 30), [1.0, 2.0, 3.0, 1e270, 1e-270]])
    assert _ulp80(_run(3, x), 1 / x.astype(np.longdouble)).max() <= 0.52


def _div(a, d):
    a, d = np.broadcast_arrays(np.asarray(a, float), np.asarray(d, float))
    ad, y = torch.from_numpy(a.copy()).cuda(), torch.from_numpy(d.copy()).cuda()
    N.check(N.load().keq_math_selftest(4, ad.data_ptr(), y.data_ptr(), ad.numel(), N.stream_handle()), "selftest")
    return y


def test_div_nr():
    """Rounds like the division up to ties; where the quotient is not finite, or an
    operand is special, it is the division's result."""
    a, d = _values(25, -30, 30) * np.random.default_rng(26).choice([-1.0, 1.0], 200000), _values(27, -30, 30)
    assert _ulp80(_div(a, d), a.astype(np.longdouble) / d).max() <= 0.52
    s = np.array([0.0, -0.0, 1.0, -2.5, 1e-300, 1e300, -1.7e308, np.inf, -np.inf, np.nan, 1e-320, 3e-200, 4e200])
    a, d = (t.ravel() for t in np.meshgrid(s, s))
    got = _div(a, d).cpu().numpy()
    with np.errstate(all="ignore"):
        want = a / d
    near = np.isfinite(want) & (np.abs(want) > 1e-290)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
    assert np.isfinite(got[np.isfinite(want)]).all()
    assert np.abs(got[near] / want[near] - 1.0).max() <= 2.3e-16
    assert np.abs(got[np.isfinite(want) & ~near]).max() <= 1.1e-290


def test_sqrt_nr():
    """The root is corrected once (one rounding); 1/sqrt carries the rounding of
    x y in its residual, half a unit, besides its own."""
    x = np.concatenate([_values(28, -270, 270), _values(29, -3, 3), [1.0, 4.0, 1e-270, 1e270, 1e-300, 1e300]])
    ref = np.sqrt(x.astype(np.longdouble))
    assert _ulp80(_run(5, x), ref).max() <= 0.52
    assert _ulp80(_run(6, x), 1 / ref).max() <= 1.05
    s = np.array([0.0, np.inf, -1.0, np.nan])
    with np.errstate(all="ignore"):
        for kind, want in ((5, np.sqrt(s)), (6, 1 / np.sqrt(s))):
            assert np.array_equal(_run(kind, s).cpu().numpy(), want, equal_nan=True)
