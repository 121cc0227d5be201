"""Small systems with many right-hand sides: the FP64 pipe takes all columns at once, eight per CTA
(solve_one_block in dense64.cu), where digit products would cost more than the arithmetic."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu


def launches(n, nrhs):
    A, B = np.eye(n), np.ones((n, nrhs))
    before = sqbem.launch_count()
    sqbem.solve_dense(A, B)
    return sqbem.launch_count() - before


@pytest.mark.parametrize("n", [1, 10, 31, 100, 256])
def test_many_columns_cost_no_more_launches_than_one(n):
    assert launches(n, 64) == launches(n, 1)


# remainders of eight columns, both ends of the sizes that come here, and more columns than a
# grid has rows of CTAs
@pytest.mark.parametrize("n,nrhs", [(1, 64), (1, 8 * 65535 + 13), (2, 71), (7, 1000), (10, 200), (33, 65), (200, 129),
                                    (256, 64), (256, 457), (256, 458)])
def test_columns_match_one_at_a_time(n, nrhs):
    rng = np.random.default_rng([n, nrhs])
    A = rng.uniform(-1, 1, (n, n)) / n + np.eye(n)
    B = rng.normal(size=(n, nrhs))
    X, pivoted = sqbem.solve_dense(A, B)
    assert not pivoted
    # two products with the block's inverses, n roundings each
    bound = 2.0 ** -53 * 8 * n * np.max(np.abs(B))
    assert np.max(np.abs(A @ X - B)) <= bound
    for c in (0, nrhs // 2, nrhs - 1):
        x, _ = sqbem.solve_dense(A, B[:, c:c + 1])
        assert np.max(np.abs(X[:, c:c + 1] - x)) <= bound


def test_a_permuted_system_and_a_bad_column():
    rng = np.random.default_rng(3)
    A = rng.uniform(-1, 1, (40, 40)) / 40 + np.eye(40)
    B = rng.normal(size=(40, 70))
    P = rng.permutation(40)
    X, pivoted = sqbem.solve_dense(A[P], B[P])
    assert pivoted
    assert np.max(np.abs(A @ X - B)) <= 2.0 ** -53 * 320 * np.max(np.abs(B))
    B[7, 5] = np.nan
    Y, _ = sqbem.solve_dense(A[P], B[P])
    other = np.arange(70) != 5
    np.testing.assert_array_equal(Y[:, other], X[:, other])
    assert np.isnan(Y[:, 5]).any()
