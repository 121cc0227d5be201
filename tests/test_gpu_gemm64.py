"""FP64 products: digit products on the tensor cores (oz_gemm.cu), the few-column kernels
and the LU built on them, against products in extended precision."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu

LD = np.longdouble


def exact(A, B):
    """A B summed in at least 2 x 53 bits (two-term splitting of every product)."""
    A, B = np.asarray(A), np.asarray(B)
    c = 134217729.0  # Dekker's splitter, 2^27 + 1
    split = lambda x: (x * c - (x * c - x), x - (x * c - (x * c - x)))  # noqa: E731
    (ah, al), (bh, bl) = split(A), split(B)
    out = np.zeros((A.shape[0], B.shape[1]))
    err = np.zeros_like(out)
    for k in range(A.shape[1]):
        p = np.multiply.outer(A[:, k], B[k])
        e = ((np.multiply.outer(ah[:, k], bh[k]) - p) + np.multiply.outer(ah[:, k], bl[k])
             + np.multiply.outer(al[:, k], bh[k])) + np.multiply.outer(al[:, k], bl[k])
        s = out + p
        t = s - out
        err += ((out - (s - t)) + (p - t)) + e
        out = s
    return out, err


def err_vs_exact(C, A, B, alpha=1.0, beta=0.0, C0=None):
    hi, lo = exact(A, B)
    ref = alpha * hi + (beta * C0 if C0 is not None else 0.0)
    d = (C - ref) - alpha * lo
    scale = abs(alpha) * np.abs(A).max(1)[:, None] * np.abs(B).max(0)[None, :] * A.shape[1]
    return np.max(np.abs(d) / (scale + (abs(beta) * np.abs(C0) if C0 is not None else 0.0)))


# one tile and its edges, K remainders of a k16 step, of a stage and of the chunks of
# 256 and 1024 k, several tiles per CTA, all transposes
SHAPES = [(1, 1, 1), (17, 5, 3), (128, 128, 16), (129, 127, 17), (64, 200, 255), (130, 260, 257), (300, 96, 1025),
          (257, 129, 2061), (1700, 1601, 80)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_digit_product_against_extended_precision(M, N, K, ta, tb):
    if M * N > 1e6 and (ta or tb):
        pytest.skip("the many-tile shape once")
    rng = np.random.default_rng([M, N, K])
    A = rng.normal(size=(M, K)) * np.exp2(rng.integers(-20, 20, (M, 1)))
    B = rng.normal(size=(K, N)) * np.exp2(rng.integers(-300, 300, (1, N)))
    C0 = rng.normal(size=(M, N))
    C = sqbem.gemm64(A.T if ta else A, B.T if tb else B, route=1, ta=ta, tb=tb)
    # eight digits leave 2^-60 of the largest entries' product per term, FP64 rounds the
    # result once: 2^-53 of at most K times that product
    assert err_vs_exact(C, A, B) <= 2.0 ** -53
    C = sqbem.gemm64(A.T if ta else A, B.T if tb else B, C0, -1.5, 0.5, ta, tb, route=1)
    assert err_vs_exact(C, A, B, -1.5, 0.5, C0) <= 2.0 ** -51


def test_digit_product_of_integers_is_exact():
    # constant operands: every digit has the same sign, the largest sums the accumulators see
    for v in (255.0 / 256, 2.0 ** 31 - 1, 127.5 / 128, -(2.0 ** 26 - 1)):
        A, B = np.full((130, 1300), v), np.full((1300, 140), v)
        ref = float(1300 * int(v * 2 ** 40) * int(v * 2 ** 40) / 2 ** 80)
        np.testing.assert_array_equal(sqbem.gemm64(A, B, route=1), np.full((130, 140), ref))
    rng = np.random.default_rng(5)
    A, B = rng.integers(-9, 9, (200, 700)), rng.integers(-9, 9, (700, 140))
    np.testing.assert_array_equal(sqbem.gemm64(A, B, route=1), (A @ B).astype(float))


@pytest.mark.parametrize("N", [1, 63, 64, 65, 128, 129, 192, 321])
@pytest.mark.parametrize("K", [15, 33, 256])
def test_short_digit_product_at_its_column_tiles(N, K):
    # K <= 256: column tiles of 64, the whole 80-bit total rounded in integers.  Integers of 20
    # bits with empty rows and columns, exact in FP64; then equal entries whose digits are the
    # largest (sums of 2^62 before the last pass), sums that cancel to 2^-70 of the row's largest
    # entry, and results beyond the normal numbers on either side
    rng = np.random.default_rng([N, K])
    A, B = rng.integers(-2 ** 20, 2 ** 20, (131, K)), rng.integers(-2 ** 20, 2 ** 20, (K, N))
    A[::7] = 0
    B[:, ::5] = 0
    np.testing.assert_array_equal(sqbem.gemm64(A, B, route=1), (A @ B).astype(float))
    for v in (255.0 / 256, 127.5 / 128, 2.0 ** 31 - 1):
        A, B = np.full((131, K), v), np.full((K, N), -v)
        ref = -float(K * int(v * 2 ** 40) * int(v * 2 ** 40) / 2 ** 80)
        np.testing.assert_array_equal(sqbem.gemm64(A, B, route=1), np.full((131, N), ref))
    A = np.ones((131, K))
    A[:, 1] = -1.0
    A[:, 2:] = 0.0
    B = np.full((K, N), 0.75)
    B[0] += 2.0 ** -53 * 64
    np.testing.assert_array_equal(sqbem.gemm64(A, B, route=1), np.full((131, N), 2.0 ** -47))
    for a, b in ((2.0 ** -600, 2.0 ** -460), (2.0 ** 600, 2.0 ** 460), (2.0 ** -512, 2.0 ** -510)):
        A, B = np.zeros((131, K)), np.zeros((K, N))
        A[:, 0], B[0] = a, -b
        np.testing.assert_array_equal(sqbem.gemm64(A, B, route=1), np.full((131, N), -(a * b)))


def test_digit_product_no_less_exact_than_the_fp64_pipe():
    # rows and columns whose entries span four orders of magnitude, as the blocks' do
    rng = np.random.default_rng(7)
    A = rng.normal(size=(256, 1500)) * 10.0 ** rng.uniform(-4, 0, (256, 1500))
    B = rng.normal(size=(1500, 256)) * 10.0 ** rng.uniform(-4, 0, (1500, 256))
    hi, lo = exact(A, B)
    e = [np.linalg.norm((sqbem.gemm64(A, B, route=r) - hi) - lo) for r in (0, 1)]
    assert e[1] <= e[0]


def test_digit_product_extremes():
    tiny, huge = 5e-324, 1.7e308
    A = np.zeros((130, 40))
    B = np.zeros((40, 130))
    A[0, 0], B[0, 0] = huge, 0.5
    A[1, 1], B[1, 1] = tiny, 4.0
    A[2, 2], B[2, 2] = huge, huge           # overflow
    A[3, 3], B[3, 3] = 1e-200, 1e-200       # underflow
    A[4, 4], B[4, 4] = 1e-160, 1e-160       # subnormal
    A[5, 5] = np.inf
    B[6, 7] = np.nan
    B[5, 9] = 2.0
    with np.errstate(all="ignore"):
        ref = A @ B
    np.testing.assert_array_equal(sqbem.gemm64(A, B, route=1), ref)


@pytest.mark.parametrize("M,K", [(1, 1), (31, 7), (33, 129), (700, 1000)])
@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("ta", [False, True])
def test_few_columns(M, K, N, ta):
    rng = np.random.default_rng([M, K, N])
    A, B, C0 = rng.normal(size=(M, K)), rng.normal(size=(K, N)), rng.normal(size=(M, N))
    C = sqbem.gemm64(A.T if ta else A, B, C0, -1.0, 1.0, ta)
    assert err_vs_exact(C, A, B, -1.0, 1.0, C0) <= 2.0 ** -50
    np.testing.assert_array_equal(sqbem.gemm64(A.T if ta else A, B, ta=ta), sqbem.gemm64(A.T if ta else A, B, ta=ta))


# edges of the 32-wide steps, of the 128-wide panels, and several panels
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 127, 128, 129, 160, 161, 257, 640, 1001])
@pytest.mark.parametrize("nrhs", [1, 9, 70])
def test_lu_solve(n, nrhs):
    rng = np.random.default_rng([n, nrhs])
    A = rng.uniform(-1, 1, (n, n)) / n + np.eye(n)  # keeps its diagonal under pivoting
    B = rng.normal(size=(n, nrhs))
    X, pivoted = sqbem.solve_dense(A, B)
    assert not pivoted
    R = B - exact(A, X)[0]
    assert np.max(np.abs(R)) <= 2.0 ** -53 * 40 * n * np.max(np.abs(X))
    P = rng.permutation(n)
    Xp, pivoted = sqbem.solve_dense(A[P], B[P])
    assert pivoted == (not np.array_equal(P, np.arange(n)))
    np.testing.assert_allclose(Xp, X, rtol=0, atol=2.0 ** -53 * 200 * n * np.max(np.abs(X)))
