"""The FP64 terms of the preconditioner's sum z.M z (csrc/device_common.cuh), over pairs in
the ranges a solve meets (divisors are 1/den stored in FP32), at the clamp that stands
in for the zero of a fixed cell, and at numerators of zero.  krylov_solve adds quot, the
correctly rounded quotient; the pipelined solve's add_quot is the exact product with the
correctly rounded reciprocal, rounded once with the sum.  The header is compiled here
for the test; its functions are inline in the kernels."""
import ctypes as ct
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from dhara_b200 import build

pytestmark = pytest.mark.gpu

N = 1 << 24
SOURCE = """
#include "device_common.cuh"
__global__ void k(const double *a, const double *b, double *q, long long n, int add) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) q[i] = add ? add_quot(q[i], a[i], b[i]) : quot(a[i], b[i]);
}
extern "C" int run(const double *a, const double *b, double *q, long long n, int add) {
    double *d = nullptr;
    if (cudaMalloc((void **)&d, 3 * n * sizeof(double)) != cudaSuccess) return 1;
    int rc = cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
             cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
             cudaMemcpy(d + 2 * n, q, n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess;
    if (!rc) {
        k<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, d + 2 * n, n, add);
        rc = cudaGetLastError() != cudaSuccess ||
             cudaMemcpy(q, d + 2 * n, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess;
    }
    cudaFree(d);
    return rc;
}
"""


@pytest.fixture(scope="module")
def quot(gpu, tmp_path_factory):
    d = tmp_path_factory.mktemp("quot")
    src, lib = d / "quot.cu", d / "libquot.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I", os.path.join(build.HERE, "csrc"), "-shared", str(src), "-o",
                    str(lib)], check=True)
    fn = ct.CDLL(str(lib)).run

    def call(a, b, add_to=None):
        q = np.zeros_like(a) if add_to is None else add_to.copy()
        assert fn(*(x.ctypes.data_as(ct.c_void_p) for x in (a, b, q)), ct.c_longlong(a.size), add_to is not None) == 0
        return q
    return call


def pairs(n, lo=-149, hi=128):
    """Numerators (squares of z) and divisors (up to the largest FP32), then the edges."""
    r = np.random.default_rng(7)
    a, b = (np.ldexp(1.0 + r.random(n), r.integers(lo, hi, n)) for _ in range(2))
    edge = np.array([1e-300, np.ldexp(1.0, hi), np.ldexp(2.0, lo)])
    return np.concatenate([a, np.zeros(len(edge)), np.ones(len(edge))]), np.concatenate([b, edge, edge])


def test_fp64_is_correctly_rounded(quot):
    a, b = pairs(N)
    assert np.array_equal(quot(a, b), a / b)


def test_pipelined_term(quot):
    a, b = pairs(N)
    one = np.ones_like(b)
    assert np.array_equal(quot(one, b, add_to=np.zeros_like(b)), one / b)  # the reciprocal
    a, b = pairs(20000)
    # sums from far below the term to far above it (the clamp's own terms are huge)
    r = np.random.default_rng(8)
    s = np.minimum(a / b, 1e200) * np.ldexp(1.0 + r.random(a.size), r.integers(-60, 60, a.size))
    exact = [float(Fraction(x) * Fraction(1.0 / y) + Fraction(t)) for x, y, t in zip(a, b, s)]
    assert np.array_equal(quot(a, b, add_to=s), np.array(exact))
