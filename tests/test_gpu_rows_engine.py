"""The row engine (rows.cuh) at the ends of its steps: rows of 0 to 3 steps of
32 entries, starting at every alignment, beside rows whose values or columns
must not reach them (infinities next door), and its one-round and 32-row
chunks. Row sums within len * 2^-52 (FP64) or len * 2^-23 (FP32) of the sum of
magnitudes, the bound of any order of summation.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 3, 4, 5, 29, 30, 31, 32, 33, 34, 35, 61, 63, 64, 65, 67, 95, 96, 97, 100, 0, 0]


def matrix(fair, repeats, seed=0):
    rng = np.random.default_rng(seed)
    n = 130
    lens = rng.permutation(np.tile(LENGTHS, repeats))
    IA = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    JA = np.concatenate([rng.permutation(n - 1)[:k] + 1 for k in lens]).astype(np.int32)  # never column n
    vA = rng.uniform(0.1, 1.0, JA.size)
    return n, lens, IA, JA, vA


def dense(lens, n, IA, JA, vA):
    D = np.zeros((lens.size, n))
    for i in range(lens.size):
        D[i, JA[IA[i]:IA[i + 1]] - 1] = vA[IA[i]:IA[i + 1]]
    return D


@pytest.mark.parametrize("repeats", [1, 40])
@pytest.mark.parametrize("prec,eps", [("f64", 2.0 ** -52), ("f32", 2.0 ** -23)])
def test_products_at_step_ends(fair, repeats, prec, eps):
    n, lens, IA, JA, vA = matrix(fair, repeats)
    A = fair.CSRMatrix.construct(lens.size, n, vA, IA, JA)
    A.set_precision(prec)
    D = dense(lens, n, IA, JA, vA)
    x = np.random.default_rng(1).standard_normal(n)
    bound = (lens + 2) * eps * (np.abs(D) @ np.abs(x)) + 1e-300
    assert np.all(np.abs(A.matvecmul(x) - D @ x) <= bound)
    assert np.allclose(A.row_norms(1), np.abs(D).sum(1), rtol=1e-13, atol=0)
    assert np.allclose(A.row_norms(2), np.sqrt((D * D).sum(1)), rtol=1e-13, atol=0)
    assert np.allclose(A.row_norms(3), (D ** 3).sum(1) ** (1 / 3), rtol=1e-13, atol=0)
    A.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_infinite_neighbours_stay_out(fair, prec):
    n, lens, IA, JA, vA = matrix(fair, 3, seed=2)
    sick = np.arange(1, lens.size, 3)  # every third row holds an infinite value
    for i in sick:
        if lens[i]:
            vA[IA[i]:IA[i + 1]] = np.inf
    A = fair.CSRMatrix.construct(lens.size, n, vA, IA, JA)
    A.set_precision(prec)
    x = np.random.default_rng(3).uniform(0.5, 1.0, n)
    x[n - 1] = np.inf  # no row has this column
    w = A.matvecmul(x)
    well = np.ones(lens.size, bool)
    well[sick] = False
    D = dense(lens, n, IA, JA, np.where(np.isfinite(vA), vA, 0.0))
    assert np.allclose(w[well], D[well, :-1] @ x[:-1], rtol=1e-5 if prec == "f32" else 1e-13, atol=0)
    assert np.all(np.isinf(w[sick][lens[sick] > 0]))
    A.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("bounds", [(None, None), (0.0, None), (-0.25, 0.25)])
def test_sirt_chunks_and_bounds(fair, oracle, monkeypatch, prec, bounds):
    n, lens, IA, JA, vA = matrix(fair, 20, seed=4)
    A = fair.CSRMatrix.construct(lens.size, n, vA, IA, JA)
    A.set_precision(prec)
    R = oracle.OracleCSR(lens.size, n, IA, JA, vA)
    b = np.random.default_rng(5).standard_normal(lens.size)
    x0 = np.random.default_rng(6).standard_normal(n)
    lo, up = bounds
    o = fair.airms.options(relaxpar=1.0, lbound=lo, ubound=up)
    x = fair.airms.sirt("cimmino", A, b, 8, x0=x0, opts=o)
    xr = oracle.sirt("cimmino", R, b, 8, x0=x0, opts=oracle.options(relaxpar=1.0, lbound=lo, ubound=up))
    assert np.linalg.norm(x - xr) <= (1e-10 if prec == "f64" else 1e-5) * np.linalg.norm(xr)
    monkeypatch.setenv("FAIR_ROWS_BY_GROUP", "0")
    assert np.array_equal(fair.airms.sirt("cimmino", A, b, 8, x0=x0, opts=o), x)
    A.close()
