"""The fan backprojector's tiles (32 x 16 pixels, pieces of 64 rays per angle,
128 angles per window batch, shares of the angles) at the sizes where they
end: images smaller than a tile, one pixel past it, more rays per pixel than
the unrolled test takes (a fine detector), rays more than two pixels apart (a
coarse one), a source close to the image. Against the oracle's stored matrix:
FP64 to the 1e-12 of the operator's other tests, FP32 to their 1e-5.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

CASES = [  # N, angles, bins, detector width / N, source radius / N, geometry_fix
    (15, 150, 24, 1.6, 2.0, 0),    # below the index-range form; two window batches
    (16, 20, 24, 1.5, 2.0, 0),
    (17, 40, 27, 1.6, 2.0, 1),
    (33, 130, 402, 1.5, 2.0, 0),   # several pieces and candidates per pixel and angle
    (40, 24, 20, 1.5, 2.0, 0),     # bins three pixels apart
    (49, 33, 71, 1.45, 2.0, 0),    # odd p: the lower half of the bins past the image
    (35, 30, 52, 1.6, 1.2, 0),     # keys are angles
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("prec,tol", [("f64", 1e-12), ("f32", 1e-5)])
def test_backprojection_at_tile_edges(fair, oracle, case, prec, tol):
    n, nth, p, dw, r, fix = case
    th = 2 * np.pi * np.arange(nth) / nth + 0.013
    M = fair.MatrixFree(fair.Data(n=n, p=p, nth=nth, r=r, dw=dw, sd=2.0, theta=th), prec,
                        beam="fan", geometry_fix=fix)
    R = oracle.fanlineartomo(n, nth, p, r, dw, 2.0, th, geometry_fix=bool(fix))
    y = np.random.default_rng(n).random(R.m)
    assert rel_err(M.backproject(y), oracle.transvecmul(R, y)) < tol
    # one ray at a time at the window's ends: nothing outside it, nothing lost
    for j in (0, p // 2, p - 1):
        e = np.zeros(R.m)
        e[(nth // 3) * p + j] = 1.0
        assert np.array_equal(M.backproject(e) > 0, oracle.transvecmul(R, e) > 0)
    M.close()
