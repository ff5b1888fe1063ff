"""The FP64 division of the preconditioner's sum z.M z (quot, csrc/device_common.cuh),
which both 3D solvers use: the correctly rounded quotient, over 2^24 pairs in the ranges
a solve meets (divisors are 1/den stored in FP32), at the clamp that stands in for the
zero of a fixed cell, and at numerators of zero.  The header is compiled here for the
test; its functions are inline in the kernels."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

from dhara_b200 import build

pytestmark = pytest.mark.gpu

N = 1 << 24
SOURCE = """
#include "device_common.cuh"
__global__ void k(const double *a, const double *b, double *q, long long n) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) q[i] = quot(a[i], b[i]);
}
extern "C" int run(const double *a, const double *b, double *q, long long n) {
    double *d = nullptr;
    if (cudaMalloc((void **)&d, 3 * n * sizeof(double)) != cudaSuccess) return 1;
    int rc = cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
             cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess;
    if (!rc) {
        k<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, d + 2 * n, n);
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

    def call(a, b):
        q = np.empty_like(a)
        assert fn(*(x.ctypes.data_as(ct.c_void_p) for x in (a, b, q)), ct.c_longlong(a.size)) == 0
        return q
    return call


def test_fp64_is_correctly_rounded(quot):
    # squares of z in a, divisors up to the largest FP32
    r, lo, hi = np.random.default_rng(7), -149, 128
    a, b = (np.ldexp(1.0 + r.random(N), r.integers(lo, hi, N)) for _ in range(2))
    edge = np.array([1e-300, np.ldexp(1.0, hi), np.ldexp(2.0, lo)])
    a = np.concatenate([a, np.zeros(len(edge)), np.ones(len(edge))])
    b = np.concatenate([b, edge, edge])
    assert np.array_equal(quot(a, b), a / b)
