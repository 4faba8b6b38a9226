"""The adjoint on matrices whose squared row norms lie where their reciprocals
overflow: Cimmino does not change when A and b are scaled together, nor do its
gradients but for the scale.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problem(fair, m, n):
    rng = np.random.default_rng(0)
    D = rng.uniform(0.1, 1.0, (m, n)) * (rng.random((m, n)) < 0.4)
    IA = np.concatenate([[0], np.cumsum((D != 0).sum(1))])
    JA = (np.nonzero(D)[1] + 1).astype(np.int32)
    return fair.CSRMatrix.construct(m, n, D[D != 0], IA, JA)


# weights m |a_i|^2 of about 2^-131 in FP32 (unit 2^-149: 2^-18 of them) and 2^-1030
# in FP64 (unit 2^-1074; squares of entries from 2^-1045 on, 2^-30 of them each): a
# few steps grow neither by more than a factor of 20
@pytest.mark.parametrize("prec,shift,tol", [("f32", 70, 20 * 2.0 ** -18), ("f64", 519, 20 * 2.0 ** -30)])
@pytest.mark.parametrize("n", [49, 51])  # an image of 7 x 7 pixels (tiled products with A) and none
@pytest.mark.parametrize("nrhs", [1, 3])
def test_subnormal_weights(fair, prec, shift, tol, n, nrhs):
    A, S = problem(fair, 70, n), problem(fair, 70, n)
    s = 2.0 ** -shift
    S.multiply_by_scalar(s)
    A.set_precision(prec)
    S.set_precision(prec)
    rng = np.random.default_rng(nrhs)
    b, gx, lam = rng.random((A.m, nrhs)), rng.standard_normal((A.n, nrhs)), rng.uniform(0.5, 1.3, nrhs)
    want = fair.airms.sirt_adjoint("cimmino", A, b, 4, lam, gx)
    got = fair.airms.sirt_adjoint("cimmino", S, b * s, 4, lam, gx)
    got = (got[0], got[1] * s, got[2], got[3])
    for g, w in zip(got, want):
        assert np.isfinite(w).all() and np.abs(w).max() > 0
        assert np.linalg.norm(g - w) <= tol * np.linalg.norm(w)
    A.close()
    S.close()
