"""Mixed triangular solves by size and number of columns: wide clusters, two columns at a time, or
narrow ones with two or up to eight (mixed.cu)."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu

E = np.array([0.6, 0.0, 0.8])


def sphere(panels):
    if panels != 240:
        return sqbem.icosphere(1.0, {20: 0, 80: 1, 320: 2, 1280: 3}[panels])
    m = sqbem.icosphere(1.0, 1)  # every triangle cut in three: 720 unknowns
    a, b, c = m.V[:, :3], m.V[:, 3:6], m.V[:, 6:]
    g = (a + b + c) / 3
    V = np.concatenate([np.hstack([a, b, g]), np.hstack([b, c, g]), np.hstack([c, a, g])])
    return sqbem.Mesh(V, np.tile(m.tags, 3))


def solver(panels):
    return sqbem.SwimmerSolver(None, sphere(panels), np.zeros(3), 1.0, sqbem.MIXED)


def launches(s, slips):
    s.solve_free(slips)
    sqbem.kernel_stats_enable(True)
    s.solve_free(slips)
    n = sqbem.kernel_stats("trsv")[0]
    sqbem.kernel_stats_enable(False)
    return n


@pytest.mark.parametrize("panels", [20, 80, 320, 1280])
def test_eight_columns_take_one_pass(panels):
    s = solver(panels)
    two = [s.slip(E, 1.0, 0.0), s.slip(E, 0.0, 1.0)]
    assert launches(s, two * 4) == launches(s, two)


@pytest.mark.parametrize("panels", [20, 80, 240, 320, 1280])
@pytest.mark.parametrize("r", [1, 2, 3, 4, 5, 6, 7, 8])
def test_columns_match_one_at_a_time(panels, r):
    s = solver(panels)
    slips = [s.slip(E, np.cos(k), np.sin(k)) for k in range(r)]
    got = s.solve_free(slips)
    for k in range(r):
        one = s.solve_free(slips[k:k + 1])[0]
        # refined to a relative residual of 1e-8 or better either way
        scale = np.abs(one.f_sphere).max()
        np.testing.assert_allclose(got[k].f_sphere, one.f_sphere, rtol=0, atol=1e-7 * scale)
        np.testing.assert_allclose(got[k].U, one.U, rtol=0, atol=1e-7)


# seven members' wide clusters fit the GPU at once, eight do not; 20: one CTA per leaf too
@pytest.mark.parametrize("n", [7, 8, 9, 20])
@pytest.mark.parametrize("level", [2, 3])
def test_members_of_a_group_match_one_alone(n, level):
    ins = dict(a_over_R=0.4, beta=0.3, L_over_R=3.0, e=tuple(E), n_theta=9, n_r=2, sphere_level=level, towed=1)
    one, _, fs, ft = sqbem.kinematics_batch([ins], sqbem.MIXED, tractions=True)
    many, _, gs, gt = sqbem.kinematics_batch([ins] * n, sqbem.MIXED, tractions=True)
    for k in range(n):
        np.testing.assert_array_equal(many[k, :13], one[0, :13])
        np.testing.assert_array_equal(gs[k], fs[0])
        np.testing.assert_array_equal(gt[k], ft[0])
