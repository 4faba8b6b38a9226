"""What the adjoint holds on the device, seen by its allocations."""
import pytest

import fake_cuda

pytestmark = pytest.mark.gpu

GEOMETRY = """
n, nth, p, nrhs = 33, 50, 47, 4
A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth))
rng = np.random.default_rng(1)
b, gx = rng.random((A.m, nrhs)), rng.standard_normal((A.n, nrhs))
call = lambda K: fair.airms.sirt_adjoint("sart", A, b, K, 1.0, gx)
"""


def test_vectors_grow_with_the_root_of_the_steps(tmp_path):
    """400 steps: 20 segments of 20, 21 checkpoints and 40 vectors of a segment;
    16 steps: 5 and 8. Everything else, the sums of the gradient with respect to
    lambda among it, is less than one more vector of n x nrhs."""
    fake_cuda.run(tmp_path, GEOMETRY + """
call(16)
few = fake.fake_used()
call(400)
vector = 8 * A.n * nrhs
assert fake.fake_used() - few <= (61 - 13 + 1) * vector, (fake.fake_used() - few, vector)
""")


@pytest.mark.parametrize("K", [6, 400])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_runs_without_room_for_the_tiled_copies(tmp_path, K, prec):
    """The copies take at least 10 (FP64) or 6 bytes per nonzero of A and of A'; with
    nearly that much less memory the row engine gives the same gradients, to the
    tolerances of the two engines against the oracle."""
    fake_cuda.run(tmp_path, GEOMETRY + f"""
K, prec, per_nonzero, tol = {K}, "{prec}", {dict(f64=9, f32=5)[prec]}, {dict(f64=1e-10, f32=1e-5)[prec]}
""" + """
def start():
    global A
    A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth))
    A.set_precision(prec)
    A.transvecmul(b[:, 0])
    return fake.fake_used()
A.close()
base = start()
want = call(K)
held = fake.fake_used() - base
A.close()
base = start()
fake.fake_limit(base + held - 2 * per_nonzero * A.nnz)
for again in range(2):
    got = call(K)
    assert fake.fake_refused() > 0
    for g, w in zip(got, want):
        assert np.linalg.norm(g - w) <= tol * K * np.linalg.norm(w)
fake.fake_limit(0)
for g, w in zip(call(K), want):
    assert np.array_equal(g, w)
""")


def test_later_calls_take_the_memory(tmp_path):
    """No memory left but what the adjoint keeps on the handle: other calls on it
    run as on a fresh one."""
    fake_cuda.run(tmp_path, GEOMETRY + """
want = fair.airms.sirt("cimmino", A, b[:, 0], 5), fair.airms.art("kaczmarz", A, b[:, 0], [2])
A.close()
A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth))
grad = call(200)
fake.fake_limit(fake.fake_used())
got = fair.airms.sirt("cimmino", A, b[:, 0], 5), fair.airms.art("kaczmarz", A, b[:, 0], [2])
assert fake.fake_refused() > 0
for g, w in zip(got, want):
    assert np.array_equal(g, w)
fake.fake_limit(0)
for g, w in zip(call(200), grad):
    assert np.array_equal(g, w)
""")


def test_matrix_moved_to_a_batch(tmp_path):
    """A batch holds the same for a matrix whose handle has run the adjoint."""
    fake_cuda.run(tmp_path, GEOMETRY + """
def held(adjoint):
    global A
    A = fair.paralleltomo(fair.Data(n=n, p=p, nth=nth, theta=np.pi * np.arange(nth) / nth))
    if adjoint:
        call(4)
    B = fair.Batch("f64")
    B.add(A, take=True)
    A.close()
    used = fake.fake_used()
    B.close()
    return used
A.close()
assert held(False) == held(True)
""")
