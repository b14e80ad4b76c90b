"""exact.cuh at its edges: zero numerators of either sign, reciprocals next to a tie."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HARNESS = r"""
#include <cuda_runtime.h>
#include "exact.cuh"
template <typename R> __global__ void k(const R *a, const R *b, R *q, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if constexpr (sizeof(R) == 8)
        q[i] = psst::lin_quot(a[i], b[i], psst::lin_recip(b[i]));
    else
        q[i] = psst::rn_div(a[i], b[i]);
}
template <typename R> int run(const R *a, const R *b, R *q, int n) {
    R *d;
    if (cudaMalloc(&d, 3 * sizeof(R) * n)) return 1;
    cudaMemcpy(d, a, n * sizeof(R), cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, n * sizeof(R), cudaMemcpyHostToDevice);
    k<R><<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, n);
    const int e = cudaMemcpy(q, d + 2 * n, n * sizeof(R), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
extern "C" int run64(const double *a, const double *b, double *q, int n) { return run(a, b, q, n); }
extern "C" int run32(const float *a, const float *b, float *q, int n) { return run(a, b, q, n); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact")
    (d / "h.cu").write_text(HARNESS)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "supersonicflowsolver_b200", "csrc")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I", csrc, "-shared",
                    "-Xcompiler", "-fPIC", str(d / "h.cu"), "-o", str(d / "h.so")], check=True)
    return ctypes.CDLL(str(d / "h.so"))


def quotient(lib, a, b):
    q = np.empty_like(a)
    assert getattr(lib, "run64" if a.dtype == np.float64 else "run32")(
        *(v.ctypes.data_as(ctypes.c_void_p) for v in (a, b, q)), len(a)) == 0
    return q


def same_bits(x, y):
    i = np.int64 if x.dtype == np.float64 else np.int32
    return np.array_equal(x.view(i), y.view(i))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_zero_over_a_positive_number_keeps_its_sign(lib, dtype):
    b = np.concatenate([2.0 ** np.arange(-50, 50), 10.0 ** np.random.default_rng(0).uniform(-15, 15, 1000)]).astype(dtype)
    b = np.concatenate([b, b])
    a = np.zeros_like(b)
    a[len(a) // 2:] = -0.0
    q = quotient(lib, a, b)
    assert same_bits(q, a / b) and np.signbit(q[len(a) // 2:]).all()


def test_quotients_by_mantissas_of_ones(lib):
    """b = 2^k - ulp: 1 / b lies next to the middle between two FP32 numbers."""
    rng = np.random.default_rng(1)
    k = np.arange(1, 126)
    b = np.nextafter((2.0 ** k).astype(np.float32), np.float32(0))
    one, two = np.ones_like(b), np.full_like(b, 2.0)
    b = np.concatenate([b, b, np.tile(b, 100)])
    a = np.concatenate([one, two, rng.choice([-1.0, 1.0], 100 * len(one)) * rng.uniform(1.0, 87.0, 100 * len(one))])
    a = a.astype(np.float32)
    assert same_bits(quotient(lib, a, b), a / b)


def test_quotients_of_small_numerators(lib):
    """z / (1 + e^-z) for |z| down to 2^-120: the divisor is 2 from 2^-24 on."""
    rng = np.random.default_rng(2)
    z = (rng.choice([-1.0, 1.0], 1 << 18) * 2.0 ** rng.uniform(-120.0, 0.0, 1 << 18)).astype(np.float32)
    b = (np.float32(1) + np.exp(-z)).astype(np.float32)
    assert same_bits(quotient(lib, z, b), z / b)
