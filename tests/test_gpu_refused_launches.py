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


def test_without_room_for_the_sweeps_copies(tmp_path):
    """Memory for the level schedule but not for the copies of the entries beside
    it: the sweep with barriers runs, with its own bits."""
    fake_cuda.run(tmp_path, """
n, nth, p = 64, 90, 92
def handle():
    A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth + 0.01))
    fair.airms.sirt("cimmino", A, b, 1)
    return A
b = np.random.default_rng(0).random(nth * p)
run = lambda: fair.airms.art("kaczmarz", A, b, [3], opts=fair.airms.options(relaxpar=0.5))
os.environ["FAIR_SWEEP_FLOW"] = "0"
A = handle()
run()
fake.fake_peak(1)
barriers = run()
need = fake.fake_peak(1)
os.environ["FAIR_SWEEP_LEGACY"] = "1"
legacy = run()
del os.environ["FAIR_SWEEP_LEGACY"], os.environ["FAIR_SWEEP_FLOW"]
flow = run()
assert not np.array_equal(flow, barriers) and not np.array_equal(legacy, barriers)  # told apart by their bits
for room in (need, need + 8 * A.nnz, need + 12 * A.nnz):  # the copies: 12 bytes per entry, 16 per pixel
    fake.fake_limit(room)
    before = fake.fake_refused()
    got = run()
    assert fake.fake_refused() > before
    assert np.array_equal(got, barriers), room - need
fake.fake_limit(0)
assert np.array_equal(run(), flow)
""")
