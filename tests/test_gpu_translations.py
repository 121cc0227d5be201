"""FP64 results far from the coordinates' origin.  The meshes' coordinates are multiples of 2^-16
and the translations whole numbers, so that a translated mesh is the same mesh exactly: what an
integral takes from differences of its coordinates does not change.  (A centroid is rounded to
its distance from the origin, and must not enter where a vertex will do.)"""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu

SHIFT = np.array([2.0 ** 33, -2.0 ** 32, 2.0 ** 33 + 5])


def grid(x):
    return np.round(np.asarray(x) * 65536.0) / 65536.0


def points(n):
    rng = np.random.default_rng(n)
    r, t, z = 0.97 * np.sqrt(rng.uniform(size=n)), rng.uniform(0, 2 * np.pi, n), rng.uniform(0.01, 3.99, n)
    return grid(np.stack([r * np.cos(t), r * np.sin(t), z], 1))


# the forms of the field kernel: points sharing a cluster, a CTA, one and four per warp
@pytest.mark.parametrize("n", [5, 400, 1300, 4900])
def test_field(n):
    m = sqbem.tube_mesh(1.0, sqbem.uniform_z(0.0, 4.0, 7), 9, 2)
    m = sqbem.Mesh(grid(m.V), m.tags)
    rng = np.random.default_rng(1)
    u, f, pts = rng.normal(size=(m.P, 3)), rng.normal(size=(m.P, 3)), points(n)
    ref = sqbem.velocity_at(m, u, f, 1.3, pts)
    got = sqbem.velocity_at(sqbem.Mesh(m.V + np.tile(SHIFT, 3), m.tags), u, f, 1.3, pts + SHIFT)
    # 126 panels, a few roundings each; the choice of a rule at a threshold is the centroid's
    np.testing.assert_allclose(got, ref, rtol=0, atol=126 * 2.0 ** -50 * np.abs(ref).max())

