"""Quotients and roots of the ray tracer's plain path, bit for bit those of IEEE
arithmetic: next to ties and powers of two, where a neighbour's rounding decides,
and from estimates as far off as ray parameters of some thousand pixels leave them.
"""
import ctypes as C
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
#include "exact_round.cuh"
__global__ void k(const double *a, const double *b, double *out, int n, int root) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = root ? fair::sqrt_near(a[i], b[i]) : fair::div_by(a[i], b[i], __drcp_rn(b[i]));
}
extern "C" int run(const double *a, const double *b, double *out, int n, int root) {
    double *d = nullptr;
    if (cudaMalloc(&d, 3 * sizeof(double) * n) != cudaSuccess) return 1;
    cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
    k<<<256, 256>>>(d, d + n, d + 2 * n, n, root);
    const cudaError_t e = cudaMemcpy(out, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    from fortran_airtools_gb300 import build
    d = tmp_path_factory.mktemp("round")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([build.nvcc_path(), "-shared", "-o", str(d / "t.so"), str(d / "t.cu"), "-cudart", "shared"] +
                   build.common_flags(), check=True)
    f = C.CDLL(str(d / "t.so")).run

    def call(a, b, root):
        a, b, out = np.ascontiguousarray(a), np.ascontiguousarray(b), np.empty(a.size)
        p = [v.ctypes.data_as(C.c_void_p) for v in (a, b, out)]
        assert f(*p, C.c_int(a.size), C.c_int(root)) == 0
        return out
    return call


def mantissas(rng, n):
    """A quarter each: just above a power of two, just below one, two of any kind."""
    m = rng.integers(0, 1 << 52, n)
    m[::4] = rng.integers(0, 8, m[::4].size)
    m[1::4] = (1 << 52) - 1 - rng.integers(0, 8, m[1::4].size)
    return m


def number(exponent, mantissa):
    return ((np.asarray(exponent, np.int64) << 52) | mantissa).view(np.float64)


def nudge(x, k):
    return (x.view(np.int64) + k).view(np.float64)


N = 4_000_000


def test_quotients(device):
    rng = np.random.default_rng(0)
    a = number(rng.integers(965, 1024, N), rng.permutation(mantissas(rng, N)))  # direction components
    q = number(rng.integers(1010, 1036, N), mantissas(rng, N))
    n = nudge(a * q, rng.integers(-2, 3, N)) * rng.choice([-1.0, 1.0], N)
    n[::5] = 0.5 * rng.integers(-4000, 4000, n[::5].size)
    a *= rng.choice([-1.0, 1.0], N)
    assert np.array_equal(device(n, a, 0), n / a)


def test_roots(device):
    rng = np.random.default_rng(1)
    s = number(rng.integers(1009, 1024, N), mantissas(rng, N))
    v = nudge(s * s, rng.integers(-3, 4, N))
    # segments between crossings at parameters up to 2^13: each off by 2^-41 or less
    s0 = np.abs(np.sqrt(v) + rng.integers(-1000, 1001, N) * rng.choice([2.0 ** -52, 2.0 ** -50], N))
    assert np.array_equal(device(v, s0, 1), np.sqrt(v))


def test_roots_next_to_powers_of_two(device):
    """A step that lands one and a half units above a power of two, and one and a half
    units off a tie."""
    e = np.repeat(np.arange(1011, 1024), 4000)  # s = 2^(e - 1023)
    rng = np.random.default_rng(2)
    s = number(e, np.zeros(e.size, np.int64))
    s = nudge(s, rng.integers(-2, 3, e.size))
    v = nudge(s * s, rng.integers(-3, 4, e.size))
    s0 = s * (1.0 + rng.integers(-4000, 4001, e.size) * 2.0 ** -42)
    assert np.array_equal(device(v, s0, 1), np.sqrt(v))
