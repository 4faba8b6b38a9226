"""FP32 matrix-free passes at angles a rounding away from the axes: the sine or
cosine is 1 in fixed point and the other not 0.

Bins on the pixel centres: over N columns a ray drifts by at most N 2^-20, so it keeps
clear of its neighbours' pixels, and every entry is that of the FP64 operator, 1 to
2^-24, but for the cut of the distance, none on the flat of the chord.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OFF = [2.0 ** -24, 4.4e-8, 1e-9, 2.0 ** -46, 1e-16, 2.0 ** -20]


@pytest.mark.parametrize("n,p", [(33, 47), (40, 58)])
def test_close_to_the_axes(fair, n, p):
    th = [a * np.pi / 2 + s * e for a in (0, 1, 2) for e in OFF for s in (1, -1)]
    th += [float(np.float32(a * np.pi / 2)) for a in (1, 2)]
    d = fair.Data(n=n, p=p, nth=len(th), theta=np.array(th))
    M, D = fair.MatrixFree(d, "f32"), fair.MatrixFree(d, "f64")
    rng = np.random.default_rng(n)
    x, y = rng.random(n * n), rng.random(len(th) * p)
    # sums of up to n (and 2 per angle) entries of 1 with n 2^-24 relative error
    for got, want, terms in ((M.project(x), D.project(x), n), (M.backproject(y), D.backproject(y), 2 * len(th))):
        assert want.max() > 1.0
        assert np.abs(got - want).max() <= 2 * terms * 2.0 ** -24 * want.max()
    M.close()
    D.close()
