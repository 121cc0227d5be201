"""FP64 products and LU solves whose rows, columns or summation index have different scales:
elimination in FP64 does not see a scaling of rows or columns, and the digit products
(oz_gemm.cu) that stand in for it must not either."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu

LD = np.longdouble


def backward_error(A, X, B):
    """The largest |B - A X| of a row over what its terms add up to: row by row, so that no scaling hides it."""
    c = np.unique(np.linspace(0, B.shape[1] - 1, 4).astype(int))  # four of the columns
    X, B = X[:, c], B[:, c]
    R = np.asarray(B, LD) - np.asarray(A, LD) @ np.asarray(X, LD)
    return float(np.max(np.abs(R) / (np.abs(A) @ np.abs(X) + np.abs(B))))


def bound(n):
    # entries off the diagonal up to 1 / n of it: the n products of a row add up to half its diagonal
    # term at most, and a partial sum of at most n / 8 of them is rounded n / 8 times
    return 2.0 ** -53 * (4 + n / 8)


def system(n, nrhs):
    rng = np.random.default_rng([n, nrhs])
    return rng.uniform(-1, 1, (n, n)) / n + np.eye(n), rng.normal(size=(n, nrhs))


@pytest.mark.parametrize("n", [300, 640, 1001])
@pytest.mark.parametrize("nrhs", [1, 70])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -20, 1e-12, 2.0 ** -200])
@pytest.mark.parametrize("what", ["rows", "columns", "both"])
def test_lu_of_scaled_systems(n, nrhs, scale, what):
    A, B = system(n, nrhs)
    d, e = np.ones(n), np.ones(n)
    if what != "columns":
        d[64:] = scale  # smaller rows below: the multipliers stay below 1, no exchanges
    if what != "rows":
        e[np.arange(n) % 3 == 1] = scale
    A, B = A * d[:, None] * e, B * d[:, None]
    X, pivoted = sqbem.solve_dense(A, B)
    assert not pivoted
    assert backward_error(A, X, B) <= bound(n)


@pytest.mark.parametrize("n", [300, 640])
def test_lu_of_rows_whose_scale_falls_steadily(n):
    A, B = system(n, 70)
    d = np.exp2(-np.arange(n) // 2)
    X, pivoted = sqbem.solve_dense(A * d[:, None], B * d[:, None])
    assert not pivoted
    assert backward_error(A * d[:, None], X, B * d[:, None]) <= bound(n)


@pytest.mark.parametrize("n", [300, 640])
@pytest.mark.parametrize("scale", [2.0 ** -30, 1e-13])
def test_decoupled_right_hand_sides_keep_their_digits(n, scale):
    # two systems that do not see each other: the small right-hand sides of the second are solved
    # as exactly as on their own
    A, B = system(n, 70)
    h = n // 2
    A[:h, h:] = 0.0
    A[h:, :h] = 0.0
    B[h:] *= scale
    X, _ = sqbem.solve_dense(A, B)
    assert backward_error(A[:h, :h], X[:h], B[:h]) <= bound(n)
    assert backward_error(A[h:, h:], X[h:], B[h:]) <= bound(n)


# both ways the scales are found: K up to 512 and beyond; K = 80: a partial chunk
@pytest.mark.parametrize("M,N,K", [(130, 96, 80), (200, 70, 256), (64, 140, 500), (130, 70, 700), (64, 66, 1300)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_scales_along_the_summation_index(M, N, K, ta, tb):
    rng = np.random.default_rng([M, N, K])
    A, B = rng.uniform(0.5, 1, (M, K)), rng.uniform(0.5, 1, (K, N))
    s = np.exp2(rng.integers(-200, 200, K))
    s[::9] = 1.0
    As, Bs = A * s, B / s[:, None]
    Bs = Bs * np.exp2(rng.integers(-60, 60, N))
    C = sqbem.gemm64(As.T if ta else As, Bs.T if tb else Bs, route=1, ta=ta, tb=tb)
    ref = np.asarray(As, LD) @ np.asarray(Bs, LD)
    # positive terms: the digits leave 2^-60 of the largest per term, and the result is rounded once
    assert np.max(np.abs((C - ref) / ref)) <= 2.0 ** -52
    C0 = rng.normal(size=(M, N)) * np.asarray(ref, float)
    C = sqbem.gemm64(As.T if ta else As, Bs.T if tb else Bs, C0, -1.0, 1.0, ta, tb, route=1)
    assert np.max(np.abs((C - (C0 - ref)) / (np.abs(C0) + ref))) <= 2.0 ** -51


def test_scales_at_the_ends_of_the_range():
    # rows of B of zeros, of subnormal numbers and of the largest; columns of A to match
    rng = np.random.default_rng(4)
    for K in (96, 600):
        A, B = rng.uniform(0.5, 1, (70, K)), rng.uniform(0.5, 1, (K, 70))
        A[:, :16] *= 2.0 ** 1000
        B[:16] *= 2.0 ** -1060
        A[:, 16:32] *= 2.0 ** -1000
        B[16:32] *= 2.0 ** 1000
        B[32:40] = 0.0
        A[:, 40:48] = 0.0
        A[7] = 0.0
        B[:, 9] = 0.0
        C = sqbem.gemm64(A, B, route=1)
        ref = np.asarray(A, LD) @ np.asarray(B, LD)
        assert np.all(np.abs(C - ref) <= 2.0 ** -52 * ref)
