"""Where cooperative launches are refused, SIRT, Kaczmarz sweeps and twin ART run
on their other kernels."""
import pytest

import fake_cuda

pytestmark = pytest.mark.gpu


def test_without_cooperative_launches(tmp_path):
    """The one-launch SIRT and its passes give the same bits; sweeps on other
    groups of warps agree to 1e-10, as each does with the oracle. Fan N = 128: levels that
    a cooperative grid takes by default."""
    fake_cuda.run(tmp_path, """
o = fair.airms.options(relaxpar=0.5, lbound=0.0)
for n, nth, p in ((40, 60, 58), (128, 90, 182)):
    A = fair.fanlineartomo(fair.Data(n=n, p=p, nth=nth, r=2.0, dw=p / n, sd=2.0, theta=2 * np.pi * np.arange(nth) / nth))
    b = A.matvecmul(np.random.default_rng(n).random(A.n))
    def runs():
        return (fair.airms.sirt("sart", A, b, 10, opts=o), fair.airms.art("kaczmarz", A, b, [2], opts=o),
                fair.airms.art("symkaczmarz", A, b, [4], opts=o))
    want, before = runs(), fake.fake_refused()
    fake.fake_no_cooperative(1)
    for flow in ("1", "0"):
        os.environ["FAIR_SWEEP_FLOW"] = flow
        got = runs()
        assert fake.fake_refused() > before
        assert np.array_equal(got[0], want[0])
        for g, w in zip(got[1:], want[1:]):
            assert np.linalg.norm(g - w) <= 1e-10 * np.linalg.norm(w)
    os.environ["FAIR_SWEEP_FLOW"] = "1"
    fake.fake_no_cooperative(0)
    A.close()
""")
