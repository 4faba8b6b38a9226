"""Work units of a tiled batch at the edges of a CTA's rounds of 16 chunks.

The units of all problems are cut together (whole rounds, at most 128 chunks);
how they are cut changes no sum, so every problem must come out bit for bit as
alone in its batch, and within 1e-10 (FP64) or 1e-5 (FP32) of the oracle.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

# N, angles, bins: 1, 15, 16, 17, 128, 129 chunks of 32 rays over one image tile
# and 1, 8, 17, 32 chunks per pixel tile; N = 100: 4 image tiles, 16 pixel tiles
SHAPES = [(4, 2, 4), (32, 15, 32), (16, 16, 32), (23, 17, 32), (32, 128, 32), (32, 129, 32), (100, 40, 140)]


@pytest.mark.parametrize("prec,tol", [("f64", 1e-10), ("f32", 1e-5)])
def test_units_together_and_alone(fair, oracle, prec, tol):
    o = fair.airms.options(lbound=0.0)
    probs = []
    for n, nth, p in SHAPES:
        th = np.pi * np.arange(nth) / nth + 0.01
        A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=th))
        R = oracle.paralleltomo(n, nth, p, th)
        probs.append((A, R, oracle.matvecmul(R, fair.phantomgallery.grains(n, 12, seed=n + nth))))

    def run(sel):
        B = fair.Batch(prec, layout="tiled")
        for A, _, _ in sel:
            B.add(A)
        X = B.sirt("sart", np.concatenate([b for _, _, b in sel]), 8, opts=o)
        _, co = B.offsets()
        B.close()
        return [X[co[i]:co[i + 1]] for i in range(len(sel))]

    for x, q in zip(run(probs), probs):
        assert np.array_equal(x, run([q])[0])
        xr = oracle.sirt("sart", q[1], q[2], 8, opts=oracle.options(lbound=0.0))
        assert rel_err(x, xr) < tol
