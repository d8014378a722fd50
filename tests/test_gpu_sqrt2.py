"""The pipelines' pairwise square root (sqrt2 in csrc/cell.cuh) against sqrtf, bit for bit: every
float in [1, 4), and every exponent it takes with the mantissas nearest a power of four. A small
kernel is compiled for this, as no entry point hands the function out."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "cell.cuh"
__global__ void check(unsigned first, unsigned count, unsigned *bad) {
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const float x = __uint_as_float(first + k), y = __uint_as_float(first + (k ^ 1u));
        bool odd = false;
        const float2 s = sbs::sqrt2(make_float2(x, y), odd);
        if (odd || __float_as_uint(s.x) != __float_as_uint(sqrtf(x)) || __float_as_uint(s.y) != __float_as_uint(sqrtf(y)))
            atomicAdd(bad, 1u);
    }
}
__global__ void refused(const float *x, int n, unsigned *odd_count) {
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        bool odd = false;
        sbs::sqrt2(make_float2(x[k], 1.f), odd);
        if (odd) atomicAdd(odd_count, 1u);
    }
}
extern "C" int run_check(unsigned first, unsigned count, unsigned *out) {
    unsigned *d;
    if (cudaMalloc(&d, 4) != cudaSuccess) return 1;
    cudaMemset(d, 0, 4);
    check<<<1024, 256>>>(first, count, d);
    const int rc = (int)cudaMemcpy(out, d, 4, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return rc;
}
extern "C" int run_refused(const float *x, int n, unsigned *out) {
    unsigned *d;
    float *dx;
    if (cudaMalloc(&d, 4) != cudaSuccess || cudaMalloc(&dx, 4 * n) != cudaSuccess) return 1;
    cudaMemset(d, 0, 4);
    cudaMemcpy(dx, x, 4 * n, cudaMemcpyHostToDevice);
    refused<<<1, 32>>>(dx, n, d);
    const int rc = (int)cudaMemcpy(out, d, 4, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(dx);
    return rc;
}
"""


@pytest.fixture(scope="module")
def lib(sbs, tmp_path_factory):
    from soap_bubble_simulation_gb300 import build

    d = tmp_path_factory.mktemp("sqrt2")
    src, so = str(d / "sqrt2.cu"), str(d / "sqrt2.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build.nvcc_path(), "-shared", *build.NVCC_FLAGS, "-I", os.path.join(build.CSRC), src, "-o", so],
                   check=True)
    return ctypes.CDLL(so)


def test_every_mantissa_rounds_as_sqrtf(lib):
    out = ctypes.c_uint()
    assert lib.run_check(ctypes.c_uint(0x3F800000), ctypes.c_uint(1 << 24), ctypes.byref(out)) == 0
    assert out.value == 0
    for e in range(127 - 96, 127 + 126):  # the edges of every binade sqrt2 takes
        for first in (e << 23, (e << 23) + (1 << 23) - 4096):
            assert lib.run_check(ctypes.c_uint(first), ctypes.c_uint(4096), ctypes.byref(out)) == 0
            assert out.value == 0


def test_zero_is_taken_and_the_rest_is_left_to_sqrtf(lib):
    def refused(*x):
        a, out = (ctypes.c_float * len(x))(*x), ctypes.c_uint()
        assert lib.run_refused(a, len(x), ctypes.byref(out)) == 0
        return out.value

    assert refused(0.0, 2.0**-96, 1e30) == 0
    odd = (2.0**-97, 1e-40, 2.0**126, float("inf"), float("nan"), -1.0)
    assert refused(*odd) == len(odd)
