"""The 6-entry tiled records (layout code 14) at chunk lengths of 1 to about 25
slots, where the inner slots' plain fetch begins and ends: images of 1 to 72
pixels a side (one tile, segments of up to 2N entries) and rows whose slots have
no step code (a random matrix), against code 9 (the same terms, the sums in
another order) and the oracle with the bars of the 2-byte forms.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def sirt(fair, A, b, prec, code):
    from fortran_airtools_gb300._clib import check, lib
    A.set_precision(prec)
    check(lib().fair_sirt_set_lanes(A.handle, (C.c_int32 * 4)(8, 8, code, code)))
    return fair.airms.sirt("sart", A, b, 6, opts=fair.airms.options())


@pytest.mark.parametrize("prec,tol", [("q16", 1e-4), ("f16", 5e-3)])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 7, 9, 12, 13, 18, 19, 24, 37, 72])
def test_chunk_lengths(fair, oracle, n, prec, tol):
    nth, p = 24, n + 3
    th = np.pi * np.arange(nth) / nth + 0.02
    A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=th))
    R = oracle.paralleltomo(n, nth, p, th)
    b = oracle.matvecmul(R, np.random.default_rng(n).random(n * n))
    x = sirt(fair, A, b, prec, 14)
    assert rel_err(x, sirt(fair, A, b, prec, 9)) < 2e-6
    assert rel_err(x, oracle.sirt("sart", R, b, 6)) < tol


def test_slots_without_codes(fair, oracle):
    rng = np.random.default_rng(8)
    n, m = 60, 200
    A0 = np.zeros((m, n * n))
    for i, q in enumerate(rng.integers(1, 90, m)):
        # a run of neighbouring pixels with a jump now and then
        cols = (np.cumsum(np.where(rng.random(q) < 0.02, 400, 1)) + rng.integers(0, 300)) % (n * n)
        A0[i, cols] = rng.random(q) + 0.2
    A0[:, 0] += 0.1
    IA = np.concatenate([[0], np.cumsum((A0 > 0).sum(1))]).astype(np.int64)
    JA = (np.nonzero(A0)[1] + 1).astype(np.int32)
    vA = A0[A0 > 0]
    A = fair.CSRMatrix.construct(m, n * n, vA, IA, JA)
    R = oracle.OracleCSR(m, n * n, IA, JA, vA)
    b = oracle.matvecmul(R, rng.random(n * n))
    x, x9 = sirt(fair, A, b, "q16", 14), sirt(fair, A, b, "q16", 9)
    xr = oracle.sirt("sart", R, b, 6)
    hit = np.isfinite(xr)  # SART divides by the column sums: NaN where no row has an entry
    assert hit.sum() > 1000
    assert np.array_equal(hit, np.isfinite(x)) and np.array_equal(hit, np.isfinite(x9))
    assert rel_err(x[hit], x9[hit]) < 2e-6
    assert rel_err(x[hit], xr[hit]) < 1e-4
