"""velocity_at over the forms its kernel takes: points sharing a cluster, a CTA, one and four
per warp, ragged panel tiles, near panels of every rule, infinities in the data."""
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


# 1, 303 | 304, 1215 | 1216, 4863 | 4864 points: the limits of the four forms, and remainders
@pytest.mark.parametrize("n", [1, 5, 303, 304, 1215, 1216, 1221, 4863, 4864, 4891])
def test_every_form_against_the_oracle(oracle, n):
    m, u, f, pts = setup(n)
    om = oracle.tube_mesh(1.0, oracle.uniform_z(0.0, 4.0, 7), 9, 2)
    ref = oracle.velocity_at(om, u, f, 1.3, pts)
    scale = np.abs(ref).max()
    assert np.abs(sqbem.velocity_at(m, u, f, 1.3, pts) - ref).max() <= 1e-12 * scale
    a = sqbem.velocity_at(m, u, f, 1.3, pts, sqbem.MIXED)
    # FP32 kernel sums: 126 panels of terms up to the largest, 2^-24 each
    assert np.abs(a - ref).max() <= 126 * 2.0 ** -22 * scale
    np.testing.assert_array_equal(a, sqbem.velocity_at(m, u, f, 1.3, pts, sqbem.MIXED))


@pytest.mark.parametrize("n", [3, 400, 1300, 4900])
def test_scales_and_translations(n):
    m, u, f, pts = setup(n, 1)
    ref = sqbem.velocity_at(m, u, f, 1.0, pts, sqbem.MIXED)
    scale = np.abs(ref).max()
    for k in (1e-200, 1e90, 1e250):  # far outside FP32's range
        np.testing.assert_allclose(sqbem.velocity_at(m, k * u, k * f, 1.0, pts, sqbem.MIXED) / k, ref, rtol=0,
                                   atol=1e-12 * scale)
    d = np.array([3e6, -1e6, 2e6])  # FP64 coordinates lose 22 bits there, FP32 pairs must not lose more
    t = sqbem.Mesh(m.V + np.tile(d, 3), m.tags)
    exact = sqbem.velocity_at(t, u, f, 1.0, pts + d)
    got = sqbem.velocity_at(t, u, f, 1.0, pts + d, sqbem.MIXED)
    assert np.abs(got - exact).max() <= 126 * 2.0 ** -22 * scale


@pytest.mark.parametrize("n", [3, 400, 1300, 4900])
@pytest.mark.parametrize("precision", [sqbem.FP64, sqbem.MIXED])
def test_infinite_and_nan_data_reach_every_point(n, precision):
    m, u, f, pts = setup(n, 2)
    f[17, 1] = np.inf
    assert not np.isfinite(sqbem.velocity_at(m, u, f, 1.0, pts, precision)).any()
    f[17, 1] = np.nan
    assert np.isnan(sqbem.velocity_at(m, u, f, 1.0, pts, precision)).all()
