"""A batch used again and again: calls with other options, methods, vectors and
problems give the bits of a batch made for that call.
"""
import numpy as np
import pytest

import fake_cuda

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


@pytest.mark.parametrize("layout", ["packed", "tiled"])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_vectors_methods_and_problems_of_each_call(fair, prec, layout):
    """Device runs that change the vectors, the method, the number of iterations
    and the problems, in an order where each is the only change once."""
    torch = pytest.importorskip("torch")
    B, shapes = make(fair, prec, layout), list(SHAPES)
    bufs = {}

    def vectors(key, rows, cols):
        if (key, rows) not in bufs:
            g = torch.Generator().manual_seed(hash(key) % 1000 + rows)
            bufs[key, rows] = (torch.rand(rows, generator=g, dtype=torch.float64).cuda(),
                               torch.empty(cols, dtype=torch.float64, device="cuda"))
        return bufs[key, rows]

    def run(batch, vec, method, K):
        info = batch.info()
        d_b, d_x = vectors(vec, info["rows"], info["cols"])
        d_x.zero_()
        torch.cuda.synchronize()
        batch.prepare(method, fair.airms.options(lbound=0.0))
        batch.run_device(d_b.data_ptr(), d_x.data_ptr(), K)
        torch.cuda.synchronize()
        return d_x.cpu().numpy().copy()

    for add, vec, method, K in ((False, 0, "sart", 3), (False, 1, "sart", 3), (False, 1, "cimmino", 3),
                                (False, 1, "cimmino", 4), (False, 0, "sart", 3), (True, 0, "sart", 3),
                                (False, 0, "sart", 3), (False, 1, "cimmino", 2)):
        if add:
            shapes.append((26, 11, 37))
            n, nth, p = shapes[-1]
            A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth + 0.01))
            B.add(A)
            A.close()
        F = make(fair, prec, layout, shapes)
        want = run(F, vec, method, K)
        F.close()
        got = run(B, vec, method, K)
        assert np.isfinite(got).any() and np.array_equal(got, want, equal_nan=True), (add, vec, method, K)
    B.close()


@pytest.mark.parametrize("layout", ["packed", "tiled"])
def test_repeated_calls_copy_no_tables(tmp_path, layout):
    """After the first call on a set of problems the tables that these settle, and
    on the same vectors all tables, stay: no blocking copy, no allocation."""
    fake_cuda.run(tmp_path, f"""
B = fair.Batch("f32", layout="{layout}")
for n, nth, p in ((20, 15, 29), (33, 24, 47)):
    A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth + 0.01))
    B.add(A, take=True)
    A.close()
b = np.random.default_rng(3).random(B.info()["rows"])
first = B.sirt("sart", b, 3)
copies, allocs = fake.fake_copies(), fake.fake_allocs()
for K in (3, 3, 5, 3):
    x = B.sirt("sart", b, K)
assert np.array_equal(x, first, equal_nan=True)
assert (fake.fake_copies(), fake.fake_allocs()) == (copies, allocs)
""")
