"""Error of the device code's reciprocal, quotient and power (wds_math) against
80-bit arithmetic, in units in the last place of the exact value."""
import ctypes

import numpy as np
import pytest
import torch

from wdsgpu_b200 import _lib

pytestmark = pytest.mark.gpu


def _eval(cuda, function, x, y=None):
    x = torch.tensor(x, device=cuda)
    y = None if y is None else torch.tensor(y, device=cuda)
    out = torch.empty_like(x)
    _lib.check(_lib.load().wds_math(
        function, x.numel(), x.data_ptr(), 0 if y is None else y.data_ptr(), out.data_ptr(),
        ctypes.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)), "wds_math")
    return out.cpu().numpy()


def _ulps(got, exact):
    with np.errstate(over="ignore", invalid="ignore"):
        near = exact.astype(np.float64)
        unit = np.spacing(np.abs(near)).astype(np.longdouble)
        err = np.abs(got.astype(np.longdouble) - exact) / unit
    return np.where(np.isinf(near) & (got == near), 0, err)   # an overflow is infinite


def test_reciprocal_and_quotient(cuda):
    # two Newton steps from 20 bits or more, then one rounding: 0.5 plus 2^-26;
    # the quotient's residual is exact, its last rounding likewise
    rng = np.random.default_rng(1)
    b = np.concatenate([2.0 ** rng.uniform(-300, 300, 100000), rng.uniform(1, 2, 100000),
                        [1.0, np.nextafter(1.0, 2), np.nextafter(2.0, 1), 2.0, 1e-7, 1e8, 1e300]])
    a = np.concatenate([2.0 ** rng.uniform(-300, 300, b.size - 50000), -rng.uniform(1, 2, 50000)])
    A, B = a.astype(np.longdouble), b.astype(np.longdouble)
    assert _ulps(_eval(cuda, _lib.MATH_RECIP, b), 1 / B).max() <= 0.51
    assert _ulps(_eval(cuda, _lib.MATH_QUOTIENT, a, b), A / B).max() <= 0.51


# half a unit of the last rounding and at most 0.19 of the sum 1 + t + w before
# it, the logarithm's error below 0.02 at exponents of 2; beyond, the bound
# that CUDA states for its own power
@pytest.mark.parametrize("lo,hi,bound", [(-1.0, 2.0, 0.75), (-30.0, 30.0, 2.0)])
def test_power(cuda, lo, hi, bound):
    rng = np.random.default_rng(2)
    x = 10.0 ** rng.uniform(-30, 6, 200000)
    x[:50000] = rng.uniform(0.5, 2.0, 50000)
    s = np.sqrt(0.5)
    x[:9] = [1.0, np.nextafter(1, 0), np.nextafter(1, 2), s, np.nextafter(s, 0), np.nextafter(s, 1),
             2 * s, np.nextafter(2 * s, 2), 1e-30]
    y = rng.uniform(lo, hi, x.size)
    y[::4] = rng.choice([0.852, 1.0, 2.0, 0.5, -0.148, 0.0], y[::4].size)
    exact = np.power(x.astype(np.longdouble), y.astype(np.longdouble))
    assert _ulps(_eval(cuda, _lib.MATH_POWER, x, y), exact).max() <= bound


def test_power_at_the_ends(cuda):
    # arguments that are not positive, normal and finite, and results that
    # overflow or leave the normal range
    x = np.array([0.0, -0.0, 5e-324, 1e-310, 2.2250738585072014e-308, np.inf, np.nan, -1.0, -2.5,
                  1.7976931348623157e308])
    y = np.array([0.852, -0.148, 2.0, 1.0, -1.0, 0.0, np.inf, -np.inf, np.nan, 3.0])
    x, y = (v.ravel() for v in np.meshgrid(x, y))
    rng = np.random.default_rng(3)
    e = rng.uniform(980.0, 1090.0, 4000) * rng.choice([-1.0, 1.0], 4000)   # y log2 x
    z = rng.uniform(0.3, 40.0, 4000)
    big = 2.0 ** (np.abs(e) / z).clip(max=1000.0)
    x = np.concatenate([x, big])
    y = np.concatenate([y, np.sign(e) * z])
    with np.errstate(all="ignore"):
        exact = np.power(x.astype(np.longdouble), y.astype(np.longdouble))
        want = exact.astype(np.float64)
    got = _eval(cuda, _lib.MATH_POWER, x, y)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    plain = np.isfinite(want) & (np.abs(want) < 1.797e308)
    edge = ~np.isnan(want) & ~plain
    assert np.array_equal(got[edge & (np.abs(exact) > 1.8e308)], want[edge & (np.abs(exact) > 1.8e308)])
    assert _ulps(got[plain], exact[plain]).max() <= 2.0
