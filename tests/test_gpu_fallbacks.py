"""Branches that ordinary meshes do not enter: what the Fourier blocks of the FP64 tube and duct
cannot take goes through the general solve, a factor with row exchanges is not reused, and
the mixed kernels' forms for few members, many members and odd sizes agree."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def swim(R, L, nth, nr, mu=1.0, precision=sqbem.FP64):
    c, e = np.array([0.4 * (R - 1.0), 0.0, 0.0]), np.array([0.6, 0.0, 0.8])
    tube = sqbem.Tube(R, L, 1.0, nth, nr, mu, precision)
    s = sqbem.SwimmerSolver(tube, sqbem.icosphere(1.0, 1, c), c, mu, precision)
    x = s.solve_free([s.slip(e, 1.0, 0.0), s.slip(e, 0.0, 1.0)])
    return (np.stack([np.concatenate([y.U, y.Om]) for y in x]), np.stack([y.f_sphere for y in x]) / mu,
            np.stack([y.f_tube for y in x]) / mu)


def flow(L, nth, nz, nr, mu=1.0):
    d = sqbem.DuctFlow(1.0, L, nth, nz, nr, mu)
    x = d.solve(1.5, -0.25)
    return np.atleast_1d(x.Q) * mu, x.u * mu, x.f


# Viscosities for which the entries leave FP32's range, so that the FP32 inverse that the iteration
# starts from is no inverse.  Powers of two scale every FP64 number exactly: the general
# path, as at mu = 1 without the Fourier blocks.
@pytest.mark.parametrize("mu", [2.0 ** 150, 2.0 ** -150, 2.0 ** 128, 2.0 ** -131])
def test_tube_whose_blocks_have_no_fp32_inverse(monkeypatch, mu):
    a = swim(2.5, 6.0, 10, 2, mu)
    b = swim(2.5, 6.0, 10, 2)
    for x, y in zip(a, b):
        assert rel(x, y) <= 1e-11
    monkeypatch.setenv("SQBEM_TUBE_FOURIER", "0")
    for x, y in zip(a, swim(2.5, 6.0, 10, 2, mu)):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("mu", [2.0 ** 150, 2.0 ** -150])
def test_duct_of_any_viscosity(monkeypatch, mu):
    a = flow(4.0, 8, 6, 2, mu)
    monkeypatch.setenv("SQBEM_TUBE_FOURIER", "0")
    for x, y in zip(a, flow(4.0, 8, 6, 2)):
        assert rel(x, y) <= 1e-11


def at_threshold(mesh_of, lo, hi, steps=24):
    """A parameter between lo and hi at which a pair of panels lies on a quadrature threshold."""
    def ratio(x, i, p):
        m = mesh_of(x)
        return np.linalg.norm(m.centroid[p] - m.centroid[i]) / m.h[p]
    xs = np.linspace(lo, hi, steps)
    m0 = mesh_of(xs[0])
    P = m0.P
    d = np.linalg.norm(m0.centroid[None] - m0.centroid[:, None], axis=2) / m0.h[None]
    for x1 in xs[1:]:
        m1 = mesh_of(x1)
        if m1.P != P:
            break
        d1 = np.linalg.norm(m1.centroid[None] - m1.centroid[:, None], axis=2) / m1.h[None]
        for t in (3.0, 1.5):
            hit = np.argwhere((d - t) * (d1 - t) < 0)
            if len(hit):
                i, p = hit[0]
                a, b = xs[0], x1
                for _ in range(100):
                    c = 0.5 * (a + b)
                    if (ratio(c, i, p) - t) * (ratio(a, i, p) - t) <= 0:
                        b = c
                    else:
                        a = c
                assert abs(ratio(b, i, p) / t - 1) <= 1e-13
                return b
    raise AssertionError("no pair crosses a threshold")


def test_duct_with_a_pair_on_a_threshold(monkeypatch):
    L = at_threshold(lambda L: sqbem.tube_mesh(1.0, sqbem.uniform_z(0.0, L, 6), 9, 2), 3.9, 4.1)
    a, b = flow(L, 9, 6, 2), flow(L * (1 + 1e-7), 9, 6, 2)
    monkeypatch.setenv("SQBEM_TUBE_FOURIER", "0")
    # the general path itself, which the duct next to it does not take
    for x, y in zip(a, flow(L, 9, 6, 2)):
        np.testing.assert_array_equal(x, y)
    c = flow(L * (1 + 1e-7), 9, 6, 2)
    assert any(not np.array_equal(x, y) for x, y in zip(b, c))
    for x, y in zip(b, c):
        assert rel(x, y) <= 1e-11


def test_tube_with_a_pair_on_a_threshold(monkeypatch):
    R = at_threshold(lambda R: sqbem.swimmer_tube_mesh(R, 6.0, 1.0, 10, 2), 2.45, 2.55)
    a = swim(R, 6.0, 10, 2)
    monkeypatch.setenv("SQBEM_TUBE_FOURIER", "0")
    for x, y in zip(a, swim(R, 6.0, 10, 2)):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("tube", [False, True])
def test_towed_after_a_factor_with_exchanges(tube):
    # a copy of a panel 1e-6 above it: a quadrature node lies at the copy's centroid, and the entry
    # below the diagonal exceeds it
    m = sqbem.icosphere(1.0, 1)
    V = np.concatenate([m.V, m.V[:1] + np.tile(1e-6 * m.normal[0], 3)])
    mesh = sqbem.Mesh(V, np.concatenate([m.tags, m.tags[:1]]))
    near, _ = sqbem.panel_integrals(V[:1], mesh.centroid[-1:], 0)
    own, _ = sqbem.panel_integrals(V[:1], mesh.centroid[:1], 1)
    assert abs(near[0, 0]) > 2 * abs(own[0, 0])
    t = sqbem.Tube(2.5, 6.0, 1.0, 8, 2) if tube else None
    U, Om, e = np.array([0.1, -0.2, 1.0]), np.array([0.3, 0.0, -0.1]), np.array([0.0, 0.6, 0.8])
    fresh = sqbem.SwimmerSolver(t, mesh, np.zeros(3)).solve_prescribed(U, Om)
    s = sqbem.SwimmerSolver(t, mesh, np.zeros(3))
    s.solve_free([s.slip(e, 1.0, 0.0)])
    after = s.solve_prescribed(U, Om)
    np.testing.assert_array_equal(after.f_sphere, fresh.f_sphere)
    # without exchanges: the leading block of the larger factor
    s = sqbem.SwimmerSolver(t, m, np.zeros(3))
    fresh = s.solve_prescribed(U, Om)
    s.solve_free([s.slip(e, 1.0, 0.0)])
    assert rel(s.solve_prescribed(U, Om).f_sphere, fresh.f_sphere) <= 1e-12


# 1: triangular solves on clusters of 16 and pairs of CTAs per LU leaf, 12: the narrow clusters, 20:
# one CTA per leaf too
@pytest.mark.parametrize("n", [2, 12, 20])
@pytest.mark.parametrize("nth,level", [(11, 2), (24, 1)])
def test_mixed_members_of_a_group_match_one_alone(n, nth, level):
    ins = dict(a_over_R=0.4, beta=0.3, L_over_R=3.0, e=(0.6, 0.0, 0.8), n_theta=nth, n_r=3, sphere_level=level, towed=1)
    one, _, fs, ft = sqbem.kinematics_batch([ins], sqbem.MIXED, tractions=True)
    many, _, gs, gt = sqbem.kinematics_batch([ins] * n, sqbem.MIXED, tractions=True)
    for k in range(n):
        np.testing.assert_array_equal(many[k, :13], one[0, :13])
        np.testing.assert_array_equal(gs[k], fs[0])
        np.testing.assert_array_equal(gt[k], ft[0])


@pytest.mark.parametrize("nth", [None, 9, 24])
def test_mixed_sphere_with_an_odd_number_of_panels(nth):
    # one triangle cut in two: 81 panels, odd leading dimensions
    m = sqbem.icosphere(1.0, 1)
    a, b, c = m.V[0, :3], m.V[0, 3:6], m.V[0, 6:]
    h = 0.5 * (a + b)
    V = np.concatenate([m.V[1:], [np.concatenate([a, h, c]), np.concatenate([h, b, c])]])
    mesh = sqbem.Mesh(V, np.full(81, m.tags[0]))
    e = np.array([0.6, 0.0, 0.8])

    def run(precision):
        t = sqbem.Tube(2.5, 6.0, 1.0, nth, 2, 1.0, precision) if nth else None
        s = sqbem.SwimmerSolver(t, mesh, np.zeros(3), 1.0, precision)
        x = s.solve_free([s.slip(e, 1.0, 0.0), s.slip(e, 0.0, 1.0)])
        y = s.solve_prescribed((0.1, 0.2, 1.0), (0.0, 0.3, 0.0))
        return (np.stack([np.concatenate([z.U, z.Om]) for z in x]), np.stack([z.f_sphere for z in x] + [y.f_sphere]))
    # FP32 blocks: entries good to 2^-22 or so
    for x, y in zip(run(sqbem.MIXED), run(sqbem.FP64)):
        assert rel(x, y) <= 1e-5
