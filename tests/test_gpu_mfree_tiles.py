"""FP32 matrix-free passes at the edges of their tiles and warps.

The projector walks 32 adjacent rays in step, the parallel backprojector takes
32 x 32 pixel tiles and batches of 8 angles; both must sum the entries of the
FP64 operator. An FP32 entry differs from the FP64 one by the cut of the
distance (2^-31) and its roundings, (1/c) (2^-31 / s + 3 2^-24 w), a sum of q
of them by q 2^-24 more: with s > 1e-2 on the tested angles (or 0), entries of
about 1 and at most 2 x 95 of them, below 2e-5 of the largest sum.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-5
SHAPES = [(1, 2, 1), (2, 31, 7), (3, 32, 8), (8, 33, 9), (31, 47, 16), (32, 64, 17), (33, 65, 5),
          (63, 95, 24), (64, 96, 25), (95, 134, 11)]  # N, p, angles


def op(fair, beam, n, p, nth, prec):
    if beam == "par":
        th = np.pi * np.arange(nth) / nth + np.where(np.arange(nth) % 5 == 0, 0.0, 0.02)
        return fair.MatrixFree(fair.Data(n=n, p=p, nth=nth, theta=th), prec)
    th = 2 * np.pi * np.arange(nth) / nth + 0.02
    return fair.MatrixFree(fair.Data(n=n, p=p, nth=nth, r=2.0, dw=p / n, sd=2.0, theta=th), prec, beam="fan")


@pytest.mark.parametrize("beam", ["par", "fan"])
@pytest.mark.parametrize("shape", SHAPES)
def test_products_match_fp64(fair, beam, shape):
    n, p, nth = shape
    M, D = op(fair, beam, n, p, nth, "f32"), op(fair, beam, n, p, nth, "f64")
    rng = np.random.default_rng(n * p)
    for x in (rng.random(n * n), rng.standard_normal(n * n)):
        ref = D.project(x)
        scale = np.abs(D.project(np.abs(x))).max() + 1e-30
        assert np.abs(M.project(x) - ref).max() <= TOL * scale
    for y in (rng.random(nth * p), rng.standard_normal(nth * p)):
        ref = D.backproject(y)
        scale = np.abs(D.backproject(np.abs(y))).max() + 1e-30
        assert np.abs(M.backproject(y) - ref).max() <= TOL * scale
    M.close()
    D.close()


@pytest.mark.parametrize("beam", ["par", "fan"])
def test_entries_bit_identical(fair, beam):
    """Column j of the projector and row r of the backprojector hold the same
    bits, the angles 0, pi/4 and pi/2 of a parallel beam included."""
    n, p, nth = 9, 14, 8
    M = op(fair, beam, n, p, nth, "f32") if beam == "fan" else fair.MatrixFree(
        fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth), "f32")
    A = np.stack([M.project(e) for e in np.eye(n * n)], axis=1)
    B = np.stack([M.backproject(e) for e in np.eye(nth * p)], axis=0)
    assert A.max() > 0.9
    assert np.array_equal(A, B)
    M.close()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("beam", ["par", "fan"])
def test_nonfinite_reaches_its_own_entries_only(fair, beam, bad):
    """An Inf or NaN in x (or y) reaches exactly the rays (pixels) with an
    entry there; all others keep their values."""
    n, p, nth = 40, 58, 12
    M = op(fair, beam, n, p, nth, "f32")
    rng = np.random.default_rng(5)
    x, y = rng.random(n * n), rng.random(nth * p)
    q, r = 17 * n + 23, 3 * p + 27
    hit = M.project(np.eye(1, n * n, q)[0]) > 0
    x0, xb = x.copy(), x.copy()
    x0[q], xb[q] = 0.0, bad
    g, ref = M.project(xb), M.project(x0)
    assert hit.any() and not np.isfinite(g[hit]).any()
    assert np.abs(g[~hit] - ref[~hit]).max() <= 1e-6 * ref.max()
    hit = M.backproject(np.eye(1, nth * p, r)[0]) > 0
    y0, yb = y.copy(), y.copy()
    y0[r], yb[r] = 0.0, bad
    g, ref = M.backproject(yb), M.backproject(y0)
    assert hit.any() and not np.isfinite(g[hit]).any()
    assert np.abs(g[~hit] - ref[~hit]).max() <= 1e-6 * ref.max()
    M.close()
