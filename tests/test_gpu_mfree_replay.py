"""Matrix-free SIRT captured in a CUDA graph: a replay gives the bits of a direct
call for whatever x holds when it runs, Inf and NaN among it, also when other
passes of the operator ran in between.
"""
import numpy as np
import pytest

from fortran_airtools_gb300._clib import check, lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beam", ["par", "fan"])
def test_replay_with_nonfinite_x(fair, beam):
    n, p, nth, K = 40, 58, 12, 1
    th = (1 if beam == "par" else 2) * np.pi * np.arange(nth) / nth + 0.02
    if beam == "par":
        M = fair.MatrixFree(fair.Data(n=n, p=p, nth=nth, theta=th), "f32")
    else:
        M = fair.MatrixFree(fair.Data(n=n, p=p, nth=nth, r=2.0, dw=p / n, sd=2.0, theta=th), "f32", beam="fan")
    rng = np.random.default_rng(5)
    good = rng.random(n * n)
    bad = good.copy()
    bad[17 * n + 23] = np.inf
    st = torch.cuda.Stream()
    check(lib().fair_mf_set_stream(M._h, st.cuda_stream))
    d_b = torch.from_numpy(rng.random(nth * p)).cuda()
    d_x = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    check(lib().fair_mf_sirt_prepare(M._h, b"sart", None))

    def direct(x):
        d_x.copy_(torch.from_numpy(x))
        torch.cuda.synchronize()
        check(lib().fair_mf_sirt_run_device(M._h, d_b.data_ptr(), d_x.data_ptr(), K))
        torch.cuda.synchronize()
        return d_x.cpu().numpy()

    want = {k: direct(x) for k, x in (("good", good), ("bad", bad))}
    # the rays through the Inf reach some pixels and leave others alone
    assert 0 < np.isfinite(want["bad"]).sum() < n * n and np.isfinite(want["good"]).all()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        check(lib().fair_mf_sirt_run_device(M._h, d_b.data_ptr(), d_x.data_ptr(), K))
    for kind, x in (("good", good), ("bad", bad), ("bad", bad), ("good", good), ("bad", bad)):
        assert np.array_equal(direct(bad), want["bad"], equal_nan=True)  # a later pass that met an Inf
        d_x.copy_(torch.from_numpy(x))
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(d_x.cpu().numpy(), want[kind], equal_nan=True), kind
    M.close()
