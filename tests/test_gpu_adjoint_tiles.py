"""The adjoint's products on the tiled copies (32 x 32 tiles, 1, 4, 8 or 16
interleaved right-hand sides) at the edges of tiles, angle blocks and groups
of right-hand sides, on a matrix that has no image (the row engine), and
after the matrix changes. FP64 to the adjoint's 1e-10 against the oracle's,
FP32 to the operators' 1e-5.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

GEOMETRIES = [("par", 20, 30, 28), ("par", 33, 50, 47), ("fan", 65, 24, 92)]


def matrices(fair, oracle, beam, n, nth, p):
    if beam == "par":
        th = np.pi * np.arange(nth) / nth
        return (fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=th)),
                oracle.paralleltomo(n, nth, p, th))
    th = 2 * np.pi * np.arange(nth) / nth
    return (fair.fanlineartomo(fair.Data(n=n, p=p, nth=nth, r=2.0, dw=p / n, sd=2.0, theta=th)),
            oracle.fanlineartomo(n, nth, p, 2.0, p / n, 2.0, th))


def compare(fair, oracle, A, R, method, nrhs, prec, tol):
    rng = np.random.default_rng(nrhs)
    B, GX = rng.random((R.m, nrhs)), rng.standard_normal((R.n, nrhs))
    lam, K = rng.uniform(0.5, 1.3, nrhs), 5
    lb = 0.0 if prec == "f64" else None  # in FP32 a value at the bound may fall on either side
    A.set_precision(prec)
    out = fair.airms.sirt_adjoint(method, A, B, K, lam, GX, opts=fair.airms.options(lbound=lb))
    for c in range(nrhs):
        ref = oracle.sirt_adjoint(method, R, B[:, c], K, lam[c], GX[:, c], opts=oracle.options(lbound=lb))
        for got, want in zip(out[:3], ref[:3]):
            assert rel_err(got[:, c], want) < tol
        assert abs(out[3][c] - ref[3]) <= tol * max(abs(ref[3]), np.linalg.norm(GX[:, c]))


@pytest.mark.parametrize("geometry", GEOMETRIES)
@pytest.mark.parametrize("nrhs", [1, 3, 5, 9, 17])
@pytest.mark.parametrize("prec,tol", [("f64", 1e-10), ("f32", 1e-5)])
def test_adjoint_at_tile_edges(fair, oracle, geometry, nrhs, prec, tol):
    A, R = matrices(fair, oracle, *geometry)
    compare(fair, oracle, A, R, "sart", nrhs, prec, tol)
    A.close()


@pytest.mark.parametrize("nrhs", [1, 4, 6, 16])
@pytest.mark.parametrize("prec,tol", [("f64", 1e-10), ("f32", 1e-5)])
def test_adjoint_without_an_image(fair, oracle, nrhs, prec, tol):
    m, n = 70, 51
    rng = np.random.default_rng(0)
    D = rng.uniform(0.1, 1.0, (m, n)) * (rng.random((m, n)) < 0.4)
    IA = np.concatenate([[0], np.cumsum((D != 0).sum(1))])
    JA = (np.nonzero(D)[1] + 1).astype(np.int32)
    A = fair.CSRMatrix.construct(m, n, D[D != 0], IA, JA)
    R = oracle.OracleCSR(m, n, IA, JA, D[D != 0])
    compare(fair, oracle, A, R, "cimmino", nrhs, prec, tol)
    A.close()


def test_adjoint_after_the_matrix_changes(fair, oracle):
    A, _ = matrices(fair, oracle, "par", 33, 50, 47)
    B, _ = matrices(fair, oracle, "par", 33, 50, 47)
    rng = np.random.default_rng(1)
    b, gx = rng.random((A.m, 4)), rng.standard_normal((A.n, 4))
    call = lambda M: fair.airms.sirt_adjoint("cimmino", M, b, 4, 1.0, gx)  # noqa: E731
    before = call(A)
    A.multiply_by_scalar(1.5)
    B.multiply_by_scalar(1.5)
    for got, want, old in zip(call(A), call(B), before):
        assert np.array_equal(got, want)
        assert old is not got
    assert not np.array_equal(call(A)[1], before[1])
    A.transpose()
    A.transpose()
    for got, want in zip(call(A), call(B)):
        assert np.array_equal(got, want)
    A.close()
    B.close()
