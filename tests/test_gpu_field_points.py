"""velocity_at: a point that is no number, infinite or far away leaves the other points' results
as they are."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu


def setup(n, seed=0):
    rng = np.random.default_rng(seed)
    m = sqbem.tube_mesh(1.0, sqbem.uniform_z(0.0, 4.0, 7), 9, 2)
    r, t, z = 0.97 * np.sqrt(rng.uniform(size=n)), rng.uniform(0, 2 * np.pi, n), rng.uniform(0.01, 3.99, n)
    pts = np.stack([r * np.cos(t), r * np.sin(t), z], 1)
    return m, rng.normal(size=(m.P, 3)), rng.normal(size=(m.P, 3)), pts


# points sharing a cluster, a CTA, one and four per warp; index 0: the first of a CTA, 8 and 32: of
# the next one in either of the last two
@pytest.mark.parametrize("n", [5, 400, 1300, 4900])
@pytest.mark.parametrize("index", [0, 3, 8, 32])
@pytest.mark.parametrize("bad", [(np.nan, 0.1, 0.2), (0.1, np.inf, 0.2), (0.1, 0.2, -1e12), (1e30, -1e30, 0.0),
                                 (1e200, 0.0, 0.0)])
@pytest.mark.parametrize("precision", [sqbem.FP64, sqbem.MIXED])
def test_a_bad_point_is_alone(n, index, bad, precision):
    if index >= n:
        pytest.skip("past the points")
    m, u, f, pts = setup(n)
    ref = sqbem.velocity_at(m, u, f, 1.3, pts, precision)
    other = np.arange(n) != index
    pts[index] = bad
    got = sqbem.velocity_at(m, u, f, 1.3, pts, precision)
    np.testing.assert_array_equal(got[other], ref[other])
    if np.isnan(bad[0]):
        assert np.isnan(got[index]).all()
    elif abs(bad[2]) == 1e12:
        exact = sqbem.velocity_at(m, u, f, 1.3, pts[index:index + 1])
        # FP32 kernel sums over 126 panels
        np.testing.assert_allclose(got[index], exact[0], rtol=0, atol=126 * 2.0 ** -22 * np.abs(exact).max())


@pytest.mark.parametrize("n", [3, 1300, 4900])
@pytest.mark.parametrize("distance", [1e3, 1e6, 1e8, 1e12])
def test_bodies_far_apart(n, distance):
    # two tubes far apart in one panel set, points in both: the panels of a tile of 128 are not
    # neighbours, and the FP32 offsets must not lose digits to the distance between them
    m, u, f, pts = setup(n, 3)
    d = np.array([0.0, 0.25 * distance, distance])
    far = sqbem.Mesh(np.concatenate([m.V, m.V + np.tile(d, 3)]), np.concatenate([m.tags, m.tags]))
    u2, f2 = np.concatenate([u, f]), np.concatenate([f, u])
    p2 = pts.copy()
    p2[::2] += d
    exact = sqbem.velocity_at(far, u2, f2, 1.3, p2)
    got = sqbem.velocity_at(far, u2, f2, 1.3, p2, sqbem.MIXED)
    assert np.abs(got - exact).max() <= 126 * 2.0 ** -22 * np.abs(exact).max()
