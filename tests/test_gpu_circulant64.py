"""FP64 solves through the Fourier blocks of the tube and of the duct (circulant64.cu) against
the LU of the directly assembled matrix (SQBEM_TUBE_FOURIER=0)."""
import numpy as np
import pytest

sqbem = pytest.importorskip("sqbem")

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def swimmer(R, L, nth, nr):
    c = np.array([0.4 * (R - 1.0), 0.0, 0.0])
    e = np.array([0.6, 0.0, 0.8])
    tube = sqbem.Tube(R, L, 1.0, nth, nr)
    s = sqbem.SwimmerSolver(tube, sqbem.icosphere(1.0, 1, c), c)
    slips = [s.slip(e, 1.0, 0.0), s.slip(e, 0.0, 1.0)]
    m = s.solve_free(slips)
    many = s.solve_free([np.roll(slips[k % 2], k, axis=0) for k in range(9)])  # more than eight columns
    d = s.adjoint(slips)
    return (np.stack([np.concatenate([x.U, x.Om]) for x in m]), np.stack([x.f_sphere for x in m]),
            np.stack([x.f_tube for x in m]), np.stack([x.f_tube for x in many]), d[2], d[3])


# sectors: odd, twice an odd number, multiples of four, the largest handled, one past it;
# n_r: the block order (up to 3 nb = 256, and one past it)
@pytest.mark.parametrize("R,L,nth,nr", [(2.5, 6.0, 3, 1), (2.5, 6.0, 7, 2), (2.5, 6.0, 9, 4), (2.5, 6.0, 10, 3),
                                        (2.5, 6.0, 12, 2), (2.5, 6.0, 24, 4), (2.0, 5.0, 36, 2), (2.0, 5.0, 37, 2),
                                        (2.0, 30.0, 17, 2)])
def test_tube_through_fourier_blocks_matches_lu(monkeypatch, R, L, nth, nr):
    a = swimmer(R, L, nth, nr)
    monkeypatch.setenv("SQBEM_TUBE_FOURIER", "0")
    b = swimmer(R, L, nth, nr)
    # the blocks' condition (below 1e4) times FP64 rounding, with a factor of ten
    for x, y in zip(a, b):
        assert rel(x, y) <= 1e-11


@pytest.mark.parametrize("nth,nz,nr", [(3, 4, 1), (7, 5, 2), (8, 6, 3), (24, 24, 6), (36, 8, 2), (37, 8, 2), (9, 43, 2)])
def test_duct_from_one_sector_matches_the_whole_system(monkeypatch, nth, nz, nr):
    def run():
        d = sqbem.DuctFlow(1.0, 4.0, nth, nz, nr)
        s = [d.solve(1.5, 0.0), d.solve(2.0, -0.5)]
        return [np.array([x.Q for x in s]), np.stack([x.u for x in s]), np.stack([x.f for x in s])]
    a = run()
    monkeypatch.setenv("SQBEM_TUBE_FOURIER", "0")
    for x, y in zip(a, run()):
        assert rel(x, y) <= 1e-11
