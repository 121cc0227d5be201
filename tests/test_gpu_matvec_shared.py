"""Products of one matrix with several members' columns (mv_plain_shared, matvec.cu) as an
ensemble runs them: the members have the results they have alone."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu


# one member (its own kernel), the kernels of four and of eight, remainders of both
@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 9, 17])
def test_members_of_an_ensemble_match_single_swimmers(n):
    rng = np.random.default_rng(n)
    e = rng.normal(size=(n, 3))
    y0 = np.concatenate([rng.uniform(0.0, 0.9, (n, 1)), np.zeros((n, 2)),
                         e / np.linalg.norm(e, axis=1)[:, None]], axis=1)
    alpha = rng.uniform(-5.0, 5.0, n)
    p = sqbem.TrajParams(a_over_R=0.4, n_theta=11, sphere_level=1, dt=0.05)
    _, U, Om, status, _ = sqbem.trajectory_ensemble(y0, alpha, p, 1, 1, sqbem.MIXED)
    assert not np.any(status)
    for k in range(n):
        _, u, om, st, _ = sqbem.trajectory_ensemble(y0[k:k + 1], alpha[k:k + 1], p, 1, 1, sqbem.MIXED)
        # the first evaluation's motion: the same blocks and the same preconditioner
        np.testing.assert_allclose(U[k, 0], u[0, 0], rtol=0, atol=1e-9 * np.abs(u).max())
        np.testing.assert_allclose(Om[k, 0], om[0, 0], rtol=0, atol=1e-9 * np.abs(u).max())
