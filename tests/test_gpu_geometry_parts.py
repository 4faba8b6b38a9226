"""The ray tracer's plain path at the ends of its parts (64 lines of the major
axis), the rays it must hand on (corners met at 30 and 60 degrees, lines
followed closely, axis-aligned ones) and images too large for a listed ray's
block: structure and values bit for bit equal to the oracle's.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(A, R):
    vA, IA, JA = A.arrays()
    assert np.array_equal(IA, R.IA)
    assert np.array_equal(JA, R.JA)
    assert np.array_equal(vA, R.vA)


@pytest.mark.parametrize("n,p", [(2, 4), (62, 90), (63, 89), (64, 92), (65, 93), (127, 181), (128, 182),
                                 (129, 37), (5200, 6)])
def test_parallel_parts(fair, oracle, n, p):
    th = np.array([0.0, np.pi / 6, np.pi / 4, np.pi / 3, np.pi / 2, 2 * np.pi / 3, 3 * np.pi / 4, 0.3, 2.9,
                   1e-12, 1e-9, 1e-6, np.pi / 2 - 1e-9, np.arctan(0.5), np.arctan(2.0)])
    same(fair.paralleltomo(fair.Data(n=n, p=p, nth=len(th), theta=th)),
         oracle.paralleltomo(n, len(th), p, th))


@pytest.mark.parametrize("n,p,r,fix", [(64, 91, 2.0, True), (65, 94, 1.0, False), (96, 140, 0.8, False),
                                       (33, 50, 20.0, False)])
def test_fan_parts(fair, oracle, n, p, r, fix):
    nth = 25
    th = np.concatenate([[0.0, np.pi / 6, np.pi / 2, np.pi], 2 * np.pi * np.arange(1, nth - 3) / nth])
    d = fair.Data(n=n, p=p, nth=nth, r=r, dw=1.4, sd=2.0, theta=th)
    same(fair.fanlineartomo(d, geometry_fix=fix),
         oracle.fanlineartomo(n, nth, p, r, 1.4, 2.0, th, geometry_fix=fix))
