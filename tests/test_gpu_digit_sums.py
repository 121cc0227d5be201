"""Digit products (oz_gemm.cu) at the ends of what their sums and their read-out hold: digits of one
sign, and rows and columns with infinities or NaN beside good ones."""
import numpy as np
import pytest

from test_gpu_gemm64 import exact

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu


def digits(rng, shape, lo, hi):
    """Numbers whose six leading base-256 digits lie in [lo, hi], hence 48 bits."""
    return sum(rng.integers(lo, hi + 1, shape).astype(float) * 2.0 ** (-8 * i) for i in range(6))


def err(C, A, B):
    hi, lo = exact(A, B)
    return float(np.max(np.abs((C - hi) - lo)) / (A.shape[1] * np.abs(A).max() * np.abs(B).max()))


# one chunk of the short kernel and its remainders, chunks of the long one
@pytest.mark.parametrize("K", [96, 160, 161, 176, 240, 256, 257, 512, 1024, 1300, 4100])
@pytest.mark.parametrize("lo,hi,sign", [(100, 127, 1.0), (100, 127, -1.0), (120, 127, 1.0), (127, 127, 1.0), (64, 127, 1.0)])
def test_digits_of_one_sign(K, lo, hi, sign):
    rng = np.random.default_rng([K, lo])
    A, B = digits(rng, (130, K), lo, hi), sign * digits(rng, (K, 140), lo, hi)
    # the result is rounded once, to 2^-53 of at most K times the largest product; below that the
    # digits left out and the sums of weight 6
    assert err(sqbem.gemm64(A, B, route=1), A, B) <= 2.0 ** -53 + 2.0 ** -59


@pytest.mark.parametrize("K", [160, 256, 1024])
def test_digits_of_both_signs(K):
    rng = np.random.default_rng(K)
    A, B = digits(rng, (130, K), -127, 127), digits(rng, (K, 140), -127, 127)
    assert err(sqbem.gemm64(A, B, route=1), A, B) <= 2.0 ** -53 + 2.0 ** -59


@pytest.mark.parametrize("n", [129, 300, 640])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("row", [0, 100, -1])
def test_a_bad_right_hand_side_is_alone(n, bad, row):
    rng = np.random.default_rng([n, 3])
    A = rng.uniform(-1, 1, (n, n)) / n + np.eye(n)
    B = rng.normal(size=(n, 150))
    cols = [0, 33, 149]
    other = np.setdiff1d(np.arange(150), cols)
    B[:, cols] = 0.0
    ref, _ = sqbem.solve_dense(A, B)
    B[row, cols] = bad
    X, _ = sqbem.solve_dense(A, B)
    np.testing.assert_array_equal(X[:, other], ref[:, other])
    assert not np.isfinite(X[:, cols]).all(axis=0).any()


@pytest.mark.parametrize("K", [40, 300])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 1.0), (-1.5, 0.5)])
def test_infinities_beside_good_entries(K, alpha, beta):
    rng = np.random.default_rng(K)
    A, B, C0 = rng.normal(size=(200, K)), rng.normal(size=(K, 200)), rng.normal(size=(200, 200))
    rows, cols = [3, 40, 199], [0, 64, 131]
    A[rows, [0, K // 2, K - 1]] = [np.inf, np.nan, -np.inf]
    B[[1, K // 2, K - 1], cols] = [np.nan, np.inf, -np.inf]
    A[:, K - 1] = np.where(np.isfinite(A[:, K - 1]), 0.25, A[:, K - 1])
    good = np.ix_(np.setdiff1d(np.arange(200), rows), np.setdiff1d(np.arange(200), cols))
    with np.errstate(all="ignore"):
        plain = alpha * (A @ B) + (beta * C0 if beta else 0.0)
    got = sqbem.gemm64(A, B, C0, alpha, beta, route=1)
    assert np.isfinite(got[good]).all()
    np.testing.assert_allclose(got[good], plain[good], rtol=0, atol=2.0 ** -53 * 8 * K * np.abs(plain[good]).max())
    bad = np.ones((200, 200), bool)
    bad[good] = False
    np.testing.assert_array_equal(np.isnan(got[bad]), np.isnan(plain[bad]))
    np.testing.assert_array_equal(got[bad][~np.isnan(got[bad])], plain[bad][~np.isnan(plain[bad])])
