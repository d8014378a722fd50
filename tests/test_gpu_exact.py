"""The branch-free root, reciprocal and quotient of csrc/exact.cuh against the operators, bit for bit:
every float in [1, 4) as the root's operand (the exponent only scales the rest), the reciprocals of
the root and of its square, and quotients by both. A small kernel is compiled for this, as no entry
point hands the functions out."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "exact.cuh"
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__global__ void check(unsigned first, unsigned count, unsigned *bad) {
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const float x = __uint_as_float(first + k);
        float r;
        const float d = sbs::sqrt_near(x, r);
        if (!same(d, sqrtf(x))) atomicAdd(bad, 1u);
        r = sbs::recip_near(d, r);
        if (!same(r, 1.0f / d)) atomicAdd(bad + 1, 1u);
        const float dd = d * d, rr = sbs::recip_near(dd, r * r);
        if (!same(rr, 1.0f / dd)) atomicAdd(bad + 2, 1u);
        unsigned h = (first + k) * 2654435761u;
        for (int t = 0; t < 4; ++t) {
            h = h * 1664525u + 1013904223u;
            const float a = __uint_as_float((h & 0x807fffffu) | ((90u + (h >> 27)) << 23));
            if (!same(sbs::quotient(a, d, r), a / d) || !same(sbs::quotient(a, dd, rr), a / dd)) atomicAdd(bad + 3, 1u);
        }
    }
}
extern "C" int run_check(unsigned first, unsigned count, unsigned *out) {
    unsigned *d;
    if (cudaMalloc(&d, 16) != cudaSuccess) return 1;
    cudaMemset(d, 0, 16);
    check<<<1024, 256>>>(first, count, d);
    const int rc = (int)cudaMemcpy(out, d, 16, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return rc;
}
"""


@pytest.fixture(scope="module")
def lib(sbs, tmp_path_factory):
    from soap_bubble_simulation_gb300 import build

    d = tmp_path_factory.mktemp("exact")
    src, so = str(d / "exact.cu"), str(d / "exact.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build.nvcc_path(), "-shared", *build.NVCC_FLAGS, "-I", os.path.join(build.CSRC), src, "-o", so],
                   check=True)
    return ctypes.CDLL(so)


def test_every_mantissa_rounds_as_the_operators(lib):
    out = (ctypes.c_uint * 4)()
    assert lib.run_check(ctypes.c_uint(0x3F800000), ctypes.c_uint(1 << 24), out) == 0
    assert list(out) == [0, 0, 0, 0]


@pytest.mark.parametrize("exponent", [-94, -41, -40, -39, 0, 60, 122])
def test_binade_edges_round_as_the_operators(lib, exponent):
    out = (ctypes.c_uint * 4)()
    e = 127 + exponent
    for first in (e << 23, (e << 23) + (1 << 23) - 4096):
        assert lib.run_check(ctypes.c_uint(first), ctypes.c_uint(4096), out) == 0
        assert list(out) == [0, 0, 0, 0]
