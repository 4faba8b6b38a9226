"""A batch used again and again: calls with other options, methods, vectors and
problems give the bits of a batch made for that call.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(20, 15, 29), (33, 24, 47)]  # N, angles, bins


def make(fair, prec, layout, shapes=SHAPES):
    B = fair.Batch(prec, layout=layout)
    for n, nth, p in shapes:
        A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth + 0.01))
        B.add(A, take=True)
        A.close()
    return B


def data(shapes=SHAPES):
    rng = np.random.default_rng(3)
    return rng.random(sum(nth * p for _, nth, p in shapes))


CALLS = [("sart", dict()), ("sart", dict(relaxpar=0.5)), ("sart", dict(relaxpar=0.5, lbound=0.4)),
         ("sart", dict(relaxpar=0.5, lbound=0.4, ubound=0.7)), ("cimmino", dict(relaxpar=0.5, lbound=0.4, ubound=0.7)),
         ("sart", dict())]


@pytest.mark.parametrize("layout", ["packed", "tiled"])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_options_of_each_call(fair, prec, layout):
    """The same vectors and number of iterations, other options: no call may
    run the captured passes of an earlier one."""
    B, b = make(fair, prec, layout), data()
    for method, kw in CALLS:
        F = make(fair, prec, layout)
        want = F.sirt(method, b, 4, opts=fair.airms.options(**kw))
        F.close()
        assert np.array_equal(B.sirt(method, b, 4, opts=fair.airms.options(**kw)), want), (method, kw)
    B.close()
