"""Device-resident SIRT in the reduced forms with two rounds of rows per chunk.

How rows are cut into chunks changes no sum: the same bits as in chunks of 32
rows, as with one round per chunk on the host call, at row counts on either side
of the line (2 x 5 x 8 chunks per SM) and with remainders.
"""
import numpy as np
import pytest

from fortran_airtools_gb300._clib import check, lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f16", "q16"])
@pytest.mark.parametrize("n,nth,p", [(313, 219, 445), (320, 300, 453)])  # rows 97,455 and 135,900
def test_same_bits_as_other_cuts(fair, monkeypatch, prec, n, nth, p):
    A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth + 0.003))
    A.set_precision(prec)
    b = np.random.default_rng(1).random(A.m)
    d_b = torch.from_numpy(b).cuda()

    def device():
        d_x = torch.zeros(A.n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        check(lib().fair_sirt_prepare(A.handle, b"sart", None))
        check(lib().fair_sirt_run_device(A.handle, d_b.data_ptr(), d_x.data_ptr(), 4))
        torch.cuda.synchronize()
        return d_x.cpu().numpy()

    got = device()
    assert np.array_equal(got, fair.airms.sirt("sart", A, b, 4, opts=fair.airms.options()))
    monkeypatch.setenv("FAIR_ROWS_BY_GROUP", "0")
    assert np.array_equal(got, device())
    A.close()
