"""Host threads on handles of their own, images of different sizes: Kaczmarz
sweeps (with and without barriers) and one-launch SIRT at once give the bits
they give alone.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flow", ["0", "1"])
def test_threads_equal_alone(fair, monkeypatch, flow):
    monkeypatch.setenv("FAIR_SWEEP_FLOW", flow)
    probs = []
    for i in range(4):
        n, nth, p = 40 + 8 * i, 60, 70 + 6 * i
        A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth + 0.1))
        probs.append((A, A.matvecmul(np.random.default_rng(i).random(n * n))))
    oa, os_ = fair.airms.options(relaxpar=0.5, lbound=0.0), fair.airms.options()

    def work(i, out, times):
        A, b = probs[i]
        for _ in range(times):
            out.append((fair.airms.art("symkaczmarz", A, b, [4], opts=oa).copy(),
                        fair.airms.sirt("sart", A, b, 20, opts=os_).copy()))

    alone = [[] for _ in probs]
    for i in range(4):
        work(i, alone[i], 1)
    outs = [[] for _ in probs]
    threads = [threading.Thread(target=work, args=(i, outs[i], 12)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(4):
        assert len(outs[i]) == 12  # no thread ended with an error
        for x, y in outs[i]:
            assert np.array_equal(x, alone[i][0][0])
            assert np.array_equal(y, alone[i][0][1])
