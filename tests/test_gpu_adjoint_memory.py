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
