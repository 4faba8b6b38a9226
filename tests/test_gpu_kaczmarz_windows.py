"""GPU parity of the Kaczmarz sweep's level set-up at the edges of its windows.

The levels are computed in windows of 128, 64 or 32 steps (the widest whose
entries fit shared memory), and a backward sweep takes the forward sweep's
levels in reverse. The iterate must equal the oracle's (basic_sweep,
AIRMs.f90:813-858) within 1e-10: a sum of q products rounded in any order is
off by about sqrt(q) 1.1e-16 of |a||x| (1e-14 at q = 7201), each of at most
560 projections adds that much and none enlarges the error of x.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL64 = 1e-10


def both(fair, oracle, A, R, b, method, K, order=None, **kw):
    X = fair.airms.art(method, A, b, K, order=order, opts=fair.airms.options(**kw))
    Xr = oracle.art(method, R, b, K, order=order, opts=oracle.options(**kw))
    return rel_err(X, Xr)


@pytest.mark.parametrize("cluster", ["", "1", "16"])
@pytest.mark.parametrize("steps", [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257])
def test_window_edges(fair, oracle, monkeypatch, steps, cluster):
    """Sweeps of `steps` rows in a shuffled order, forwards and back."""
    monkeypatch.setenv("FAIR_SWEEP_LEVELS_ALWAYS", "1")
    if cluster:  # unset: the sweep without barriers, levels on a grid
        monkeypatch.setenv("FAIR_SWEEP_CLUSTER", cluster)
    n, nth, p = 24, 9, 34
    th = oracle.linspace(0.0, np.pi, nth)
    A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=th))
    R = oracle.paralleltomo(n, nth, p, th)
    b = oracle.matvecmul(R, oracle.shepplogan(n))
    rows = np.flatnonzero(np.diff(R.IA) > 0) + 1
    order = np.random.default_rng(steps).permutation(rows)[:steps].astype(np.int32)
    assert order.size == steps
    for method in ("kaczmarz", "symkaczmarz"):
        assert both(fair, oracle, A, R, b, method, [2], order, relaxpar=0.7, lbound=0.0) < TOL64


@pytest.mark.parametrize("cluster", ["", "1", "16"])
@pytest.mark.parametrize("longest", [1655, 1656, 3528, 3529, 7200, 7201])
def test_window_widths(fair, oracle, monkeypatch, longest, cluster):
    """Longest rows on both sides of each window width's limit of shared
    memory (past the last, the sweep runs without levels)."""
    monkeypatch.setenv("FAIR_SWEEP_LEVELS_ALWAYS", "1")
    if cluster:  # unset: the sweep without barriers, levels on a grid
        monkeypatch.setenv("FAIR_SWEEP_CLUSTER", cluster)
    rng = np.random.default_rng(longest)
    m, n = 140, 8000
    lens = rng.integers(1, 60, m)
    lens[::47] = longest
    IA = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    JA = np.concatenate([np.sort(rng.choice(n, q, replace=False)) for q in lens]).astype(np.int32) + 1
    vA = rng.random(JA.size) + 0.1
    R = oracle.OracleCSR(m, n, IA, JA, vA)
    A = fair.CSRMatrix.construct(m, n, vA, IA, JA)
    b = oracle.matvecmul(R, rng.random(n))
    assert both(fair, oracle, A, R, b, "symkaczmarz", [4], relaxpar=0.9) < TOL64
