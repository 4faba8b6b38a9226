"""The adjoint after its matrix is scaled: every output that must change does, to
the oracle's values on the scaled matrix."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("f64", 1e-10), ("f32", 1e-5)])
def test_scaled_matrix(fair, oracle, prec, tol):
    n, p, nth, K, nrhs, c = 33, 47, 50, 4, 3, 1.5
    th = np.pi * np.arange(nth) / nth
    A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=th))
    R = oracle.paralleltomo(n, nth, p, th)
    A.set_precision(prec)
    rng = np.random.default_rng(1)
    b, gx = rng.random((A.m, nrhs)), rng.standard_normal((A.n, nrhs))
    lam = rng.uniform(0.5, 1.3, nrhs)
    before = fair.airms.sirt_adjoint("cimmino", A, b, K, lam, gx)
    A.set_precision("f64")
    A.multiply_by_scalar(c)
    A.set_precision(prec)
    R = oracle.OracleCSR(R.m, R.n, R.IA, R.JA, c * R.vA)
    after = fair.airms.sirt_adjoint("cimmino", A, b, K, lam, gx)
    for i in (0, 1):  # x and dL/db scale with 1 / c; dL/dx0 does not change
        assert not np.array_equal(before[i], after[i])
    for q in range(nrhs):
        ref = oracle.sirt_adjoint("cimmino", R, b[:, q], K, lam[q], gx[:, q], opts=oracle.options())
        for got, want in zip(after[:3], ref[:3]):
            assert rel_err(got[:, q], want) < tol
    A.close()
