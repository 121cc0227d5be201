"""velocity_at at the lines between the forms for fewer than 1216 points: clusters of eight, four and two
CTAs, a CTA, four and two warps per point, and meshes on either side of the lines in panels."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu

MESHES = {56: (7, 3, 1), 126: (9, 4, 2), 1040: (20, 21, 3)}  # panels: n_theta, n_z, n_r


def mesh(lib, P):
    nth, nz, nr = MESHES[P]
    m = lib.tube_mesh(1.0, lib.uniform_z(0.0, 4.0, nz), nth, nr)
    assert m.P == P
    return m


def points(n, far):
    rng = np.random.default_rng(n)
    if far:
        return 40.0 * rng.normal(size=(n, 3))
    r, t, z = 0.97 * np.sqrt(rng.uniform(size=n)), rng.uniform(0, 2 * np.pi, n), rng.uniform(0.01, 3.99, n)
    return np.stack([r * np.cos(t), r * np.sin(t), z], 1)


@pytest.fixture(scope="module")
def fields(oracle):
    """The oracle's velocities at 1215 points, computed once per mesh and place."""
    out = {}
    for P in MESHES:
        rng = np.random.default_rng(P)
        u, f = rng.normal(size=(P, 3)), rng.normal(size=(P, 3))
        for far in (False, True):
            pts = points(1215, far)
            out[P, far] = u, f, pts, oracle.velocity_at(mesh(oracle, P), u, f, 1.3, pts)
    return out


@pytest.mark.parametrize("P", list(MESHES))
@pytest.mark.parametrize("far", [False, True])
@pytest.mark.parametrize("n", [37, 38, 39, 76, 77, 114, 115, 152, 153, 228, 229, 304, 305, 307, 456, 457, 608, 609, 911,
                               912, 913, 1214, 1215])
def test_lines_between_the_forms(fields, P, far, n):
    u, f, pts, ref = fields[P, far]
    m, scale = mesh(sqbem, P), np.abs(ref).max()
    a = sqbem.velocity_at(m, u, f, 1.3, pts[:n])
    assert np.abs(a - ref[:n]).max() <= 1e-12 * scale
    b = sqbem.velocity_at(m, u, f, 1.3, pts[:n], sqbem.MIXED)
    assert np.abs(b - ref[:n]).max() <= P * 2.0 ** -22 * scale  # FP32 kernel sums
    np.testing.assert_array_equal(b, sqbem.velocity_at(m, u, f, 1.3, pts[:n], sqbem.MIXED))


@pytest.mark.parametrize("n", [5, 60, 120, 200, 250, 400, 500, 700, 1000])
@pytest.mark.parametrize("precision", [sqbem.FP64, sqbem.MIXED])
def test_a_bad_point_is_alone_in_every_form(n, precision):
    m, pts = mesh(sqbem, 126), points(n, False)
    rng = np.random.default_rng(n)
    u, f = rng.normal(size=(m.P, 3)), rng.normal(size=(m.P, 3))
    ref = sqbem.velocity_at(m, u, f, 1.3, pts, precision)
    for index, bad in ((0, (np.nan, 0.1, 0.2)), (1, (0.1, np.inf, 0.2)), (n - 1, (1e30, 0.0, 0.0))):
        p = pts.copy()
        p[index] = bad
        got = sqbem.velocity_at(m, u, f, 1.3, p, precision)
        other = np.arange(n) != index
        np.testing.assert_array_equal(got[other], ref[other])


def test_more_near_panels_than_the_list_holds_is_an_error():
    # 300 copies of a panel under every point: the list of 256 near panels per point runs over in every form
    m = mesh(sqbem, 56)
    V = np.concatenate([m.V] + [m.V[:1]] * 300)
    crowd = sqbem.Mesh(V, np.concatenate([m.tags, np.full(300, m.tags[0])]))
    u = np.ones((crowd.P, 3))
    p = m.centroid[:1] - 0.2 * m.normal[:1]
    for n in (5, 60, 120, 250, 400, 500, 700, 1000, 1300, 4900):
        with pytest.raises(sqbem.BEMError):
            sqbem.velocity_at(crowd, u, u, 1.0, np.repeat(p, n, 0))


@pytest.mark.parametrize("n", [1, 60, 120, 200, 250, 400, 500, 700, 1000, 1300, 4900])
@pytest.mark.parametrize("precision", [sqbem.FP64, sqbem.MIXED])
def test_no_panels_no_velocity(n, precision):
    m = sqbem.Mesh(np.zeros((0, 9)), np.zeros(0, int))
    got = sqbem.velocity_at(m, np.zeros((0, 3)), np.zeros((0, 3)), 1.0, points(n, False), precision)
    np.testing.assert_array_equal(got, np.zeros((n, 3)))
