"""The reciprocal of the LU kernels (recip in dense64.cu) against correctly rounded division."""
import ctypes

import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu


def recip(x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.zeros_like(x)
    dp = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    assert sqbem.lib().sqbem_test_recip(len(x), dp(x), dp(y)) == 0
    return y


def numbers(exponent, mantissas):
    return (np.asarray(exponent, np.uint64) << np.uint64(52) | mantissas.astype(np.uint64)).view(np.float64)


# a seed good to 2^-19 leaves 2^-57 of the series: 2^-4 of a unit in the last place beside the rounding
def check(x):
    y, ref = recip(x), 1.0 / x
    exact = 1 / np.asarray(x, np.longdouble)
    assert np.all(np.abs(y - exact) <= (0.5 + 2.0 ** -4) * np.spacing(np.abs(ref)))
    assert np.all(np.abs(y - ref) <= np.spacing(np.abs(ref)))
    np.testing.assert_array_equal(recip(-x), -y)


def test_dense_mantissas():
    rng = np.random.default_rng(1)
    top = np.arange(2 ** 20, dtype=np.uint64) << np.uint64(32)  # every upper half of a mantissa
    check(numbers(1023, top | rng.integers(0, 2 ** 32, 2 ** 20, dtype=np.uint64)))
    ends = np.concatenate([np.arange(4096), 2 ** 52 - 1 - np.arange(4096), 2 ** 51 + np.arange(-2048, 2048)])
    check(numbers(1023, ends))


def test_every_exponent_and_both_cutovers():
    rng = np.random.default_rng(2)
    e = np.repeat(np.arange(1, 2045), 64)  # beyond 2044 the reciprocal is subnormal
    check(numbers(e, rng.integers(0, 2 ** 52, e.size)))
    out = np.concatenate([np.arange(1, 64), np.arange(1981, 2047)]).repeat(64)  # division itself
    x = numbers(out, rng.integers(0, 2 ** 52, out.size))
    np.testing.assert_array_equal(recip(x), 1.0 / x)
    for c in (63, 64, 1980, 1981):
        check(numbers(c, np.concatenate([np.arange(64), 2 ** 52 - 1 - np.arange(64)])))


def test_zero_subnormal_and_not_finite():
    x = np.array([0.0, -0.0, 5e-324, 1e-310, -2.2250738585072009e-308, np.inf, -np.inf, np.nan, 1.7976931348623157e308])
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(recip(x), 1.0 / x)
