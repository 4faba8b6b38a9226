"""GPU parity of the Kaczmarz sweep without barriers with the oracle.

Every step waits for its own columns, so group sizes and block counts change
nothing but the order of independent steps: the iterate equals the oracle's
(basic_sweep, AIRMs.f90:813-858) within 1e-10 as on the other paths, and an Inf
or NaN in b reaches the same pixels.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL64 = 1e-10


@pytest.fixture(scope="module")
def fan(fair, oracle):
    n, nth, p = 48, 120, 69
    th = 2 * np.pi * np.arange(nth) / nth
    A = fair.fanlineartomo(fair.Data(n=n, p=p, nth=nth, r=2.0, dw=p / n, sd=2.0, theta=th))
    R = oracle.fanlineartomo(n, nth, p, 2.0, p / n, 2.0, th)
    return A, R, oracle.matvecmul(R, oracle.shepplogan(n))


@pytest.mark.parametrize("blocks", ["1", "3", "40", ""])
@pytest.mark.parametrize("group", ["1", "2", "4", "8", "16"])
def test_groups_and_blocks(fan, fair, oracle, monkeypatch, group, blocks):
    """Rows of up to 96 entries on 1 to 16 warps (entries in registers and past
    them), 1 to 640 steps in flight, both directions."""
    monkeypatch.setenv("FAIR_SWEEP_GROUP", group)
    if blocks:
        monkeypatch.setenv("FAIR_SWEEP_GRID_BLOCKS", blocks)
    A, R, b = fan
    for method, K, kw in (("kaczmarz", [1, 3], dict(relaxpar=0.25, lbound=0.0, ubound=1.0)),
                          ("symkaczmarz", [4], dict(relaxpar=0.5, lbound=0.0))):
        X = fair.airms.art(method, A, b, K, opts=fair.airms.options(**kw))
        Xr = oracle.art(method, R, b, K, opts=oracle.options(**kw))
        assert rel_err(X, Xr) < TOL64, method


def test_equals_barrier_sweep_with_long_rows(fair, oracle, monkeypatch):
    """Rows of up to 1400 entries (44 chunks: past the registers of 16 warps)
    against the sweep with barriers and the oracle."""
    rng = np.random.default_rng(4)
    m, n = 300, 2500
    lens = rng.integers(1, 90, m)
    lens[::31] = 1400
    IA = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    JA = np.concatenate([np.sort(rng.choice(n, q, replace=False)) for q in lens]).astype(np.int32) + 1
    vA = rng.random(JA.size) + 0.1
    R = oracle.OracleCSR(m, n, IA, JA, vA)
    A = fair.CSRMatrix.construct(m, n, vA, IA, JA)
    b = oracle.matvecmul(R, rng.random(n))
    monkeypatch.setenv("FAIR_SWEEP_LEVELS_ALWAYS", "1")
    kw = dict(relaxpar=0.8, lbound=0.0)
    Xf = fair.airms.art("kaczmarz", A, b, [3], opts=fair.airms.options(**kw))
    monkeypatch.setenv("FAIR_SWEEP_FLOW", "0")
    Xb = fair.airms.art("kaczmarz", A, b, [3], opts=fair.airms.options(**kw))
    Xr = oracle.art("kaczmarz", R, b, [3], opts=oracle.options(**kw))
    assert rel_err(Xf, Xr) < TOL64
    assert rel_err(Xb, Xr) < TOL64


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_nonfinite_data(fan, fair, oracle, bad):
    A, R, b = fan
    b = b.copy()
    rows = np.flatnonzero(np.diff(R.IA) > 20)
    b[rows[-40]] = bad  # late in the order: some pixels stay finite
    kw = dict(relaxpar=0.5)
    X = fair.airms.art("kaczmarz", A, b, [1], opts=fair.airms.options(**kw))
    Xr = oracle.art("kaczmarz", R, b, [1], opts=oracle.options(**kw))
    f = np.isfinite(Xr)
    assert f.any() and not f.all()
    assert np.array_equal(f, np.isfinite(X))
    assert rel_err(X[f], Xr[f]) < TOL64
