"""Digit products (oz_gemm.cu) at the ends of what their sums and their read-out hold: rows and columns
with infinities or NaN beside good ones."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu


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
