"""Small FP64 SIRT problems in one launch (a warp's first rows in registers, a grid
barrier between passes): bit for bit the passes launched one by one, which
FAIR_ROWS_BY_GROUP=1 selects, and within 1e-10 of the oracle.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

# N, angles, bins: one group of rows to just past two blocks per SM (152 SMs x 16 warps x 4 rows)
# and several groups per warp
SHAPES = [(1, 1, 2), (2, 3, 5), (7, 9, 12), (24, 20, 35), (40, 60, 58), (90, 70, 130), (98, 70, 139),
          (64, 180, 91), (128, 60, 181)]


def sirt(fair, A, b, method, K, **kw):
    return fair.airms.sirt(method, A, b, K, opts=fair.airms.options(**kw))


@pytest.mark.parametrize("method", ["sart", "cimmino"])
@pytest.mark.parametrize("shape", SHAPES)
def test_equals_passes_and_oracle(fair, oracle, monkeypatch, shape, method):
    n, nth, p = shape
    th = np.pi * np.arange(nth) / nth + 0.1
    A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=th))
    R = oracle.paralleltomo(n, nth, p, th)
    b = oracle.matvecmul(R, np.random.default_rng(n).random(n * n))
    for K, kw in ((2, {}), (5, dict(lbound=0.0, ubound=0.7)), (20, dict(lbound=0.1))):
        x = [sirt(fair, A, b, method, K, **kw) for _ in range(2)]  # the barrier's counter ends as it began
        with monkeypatch.context() as mp:
            mp.setenv("FAIR_ROWS_BY_GROUP", "1")
            y = sirt(fair, A, b, method, K, **kw)
        assert np.array_equal(x[0], y, equal_nan=True)
        assert np.array_equal(x[1], y, equal_nan=True)
        xr = oracle.sirt(method, R, b, K, opts=oracle.options(**kw))
        f = np.isfinite(xr)
        assert np.array_equal(f, np.isfinite(y))
        assert rel_err(y[f], xr[f]) < 1e-10


@pytest.mark.parametrize("m", [150, 12001])
@pytest.mark.parametrize("lanes", [4, 8, 16, 32])
def test_lanes_per_row_and_long_rows(fair, oracle, monkeypatch, lanes, m):
    """Rows from empty to past the entries held in registers."""
    from fortran_airtools_gb300._clib import check, lib
    rng = np.random.default_rng(lanes)
    n = 700
    lens = rng.integers(0, 300, m)
    lens[:8] = 0
    IA = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    JA = np.concatenate([np.sort(rng.choice(n, q, replace=False)) for q in lens]).astype(np.int32) + 1
    vA = rng.random(JA.size) + 0.1
    R = oracle.OracleCSR(m, n, IA, JA, vA)
    A = fair.CSRMatrix.construct(m, n, vA, IA, JA)
    check(lib().fair_sirt_set_lanes(A.handle, (C.c_int32 * 4)(lanes, lanes, 0, 0)))
    b = oracle.matvecmul(R, rng.random(n))
    x = sirt(fair, A, b, "cimmino", 6)
    xr = oracle.sirt("cimmino", R, b, 6)
    monkeypatch.setenv("FAIR_ROWS_BY_GROUP", "1")
    assert np.array_equal(x, sirt(fair, A, b, "cimmino", 6))
    assert rel_err(x, xr) < 1e-10
