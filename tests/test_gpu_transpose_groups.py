"""transposition (sparse_matrices.f90:395-411, reorder :492-570) at the edges
of its row groups: columns with few and with many entries per group (sorted by
a warp, by a block in shared memory, in global memory), rows that repeat a
column (source order kept), empty rows and columns, keys too wide for 32 bits.
Bit for bit equal to a stable sort by column on the host.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(fair, m, n, rows, cols):
    order = np.argsort(rows, kind="stable")
    rows, cols = rows[order], cols[order]
    vals = np.random.default_rng(7).standard_normal(rows.size)
    IA = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]).astype(np.int64)
    A = fair.CSRMatrix.construct(m, n, vals, IA, (cols + 1).astype(np.int32))
    A.transpose()
    v, ia, ja = A.arrays()
    t = np.argsort(cols, kind="stable")
    assert A.m == n and A.n == m
    assert np.array_equal(ia, np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]))
    assert np.array_equal(ja, rows[t] + 1)
    assert np.array_equal(v, vals[t])
    A.close()


@pytest.mark.parametrize("m,n,nnz", [(1, 1, 1), (1, 40, 25), (40, 1, 33), (300, 7, 2000), (500, 400, 9000),
                                     (4000, 90, 60000)])
def test_random_matrices(fair, m, n, nnz):
    rng = np.random.default_rng(m + n)
    check(fair, m, n, rng.integers(0, m, nnz), rng.integers(0, n, nnz))  # repeats a column in some rows


@pytest.mark.parametrize("heavy", [33, 700, 4096, 4097, 9000])
def test_a_heavy_column(fair, heavy):
    rng = np.random.default_rng(heavy)
    m, n = 10000, 500
    rows = np.concatenate([rng.integers(0, m, 20000), rng.permutation(m)[:heavy]])
    cols = np.concatenate([rng.integers(3, n, 20000), np.full(heavy, 1)])  # columns 0 and 2 empty
    check(fair, m, n, rows, cols)


def test_wide_keys(fair):
    rng = np.random.default_rng(0)
    m, n = 70000, 140000
    rows = np.concatenate([np.full(131100, 5), rng.integers(0, m, 70000)])
    cols = np.concatenate([rng.permutation(n)[:131100], rng.integers(0, n, 70000)])
    check(fair, m, n, rows, cols)
