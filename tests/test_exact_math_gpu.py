"""The short forms of division and square root the kernels use (tfx_exact_math.cuh) against the general
operators on the device: the roots and reciprocal roots of every float of the range, and quotients of all
2^23 divisor significands by numerator significands spread over the whole range, with both ends.  The two
are the same operation, so every bit has to agree."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include "tfx_exact_math.cuh"
using namespace tfx;
__global__ void roots(unsigned long long* bad) {
    const unsigned lo = 0x0D800000u, hi = 0x71800000u;
    for (unsigned long long k = lo + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k <= hi;
         k += (unsigned long long)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((unsigned)k), r = __fsqrt_rn(x);
        float s, i;
        sqrt_inv_ranged(x, s, i);
        if (s != r || sqrt_ranged(x) != r || !sqrt_in_range(x)) atomicAdd(bad, 1ull);
        const bool inv = sqrt_inv_in_range(x);
        if (inv && i != __fdiv_rn(1.0f, r)) atomicAdd(bad + 1, 1ull);
        if (!inv && (k & 0xfffffeu) != 0x7ffffeu) atomicAdd(bad + 2, 1ull);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned out[6] = {lo - 1, hi + 1, 0u, 0x7f800000u, 0x7fc00000u, 0x80000001u};
        for (unsigned u : out)
            if (sqrt_in_range(__uint_as_float(u)) || sqrt_inv_in_range(__uint_as_float(u))) atomicAdd(bad + 2, 1ull);
    }
}
__global__ void quotients(unsigned step, unsigned long long* bad) {
    const float b = __uint_as_float(0x3f800000u | (blockIdx.x * blockDim.x + threadIdx.x)), y = __fdiv_rn(1.0f, b);
    unsigned c = 0;
    for (unsigned a = 0; a < (1u << 23); a += step) c += div_by(__uint_as_float(0x3f800000u | a), b, y) != __fdiv_rn(__uint_as_float(0x3f800000u | a), b);
    for (unsigned k = 0; k < 512; ++k) {   // both ends
        const float p = __uint_as_float(0x3f800000u | k), q = __uint_as_float(0x3fffffffu - k);
        c += (div_by(p, b, y) != __fdiv_rn(p, b)) + (div_by(-q, b, y) != __fdiv_rn(-q, b));
    }
    if (c) atomicAdd(bad + 3, (unsigned long long)c);
}
extern "C" int run(unsigned long long* out) {
    unsigned long long* d;
    if (cudaMalloc(&d, 32) != cudaSuccess || cudaMemset(d, 0, 32) != cudaSuccess) return 1;
    roots<<<2048, 256>>>(d);
    quotients<<<(1 << 23) / 256, 256>>>(2039, d);
    const cudaError_t e = cudaMemcpy(out, d, 32, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
"""


def test_short_forms_equal_the_operators(tmp_path):
    from tressfx_gb300 import build as B
    src, lib = tmp_path / "exact.cu", tmp_path / "libexact.so"
    src.write_text(SOURCE)
    subprocess.run([str(B._cuda_home() / "bin" / "nvcc"), *B.nvcc_flags(), "-shared", "-o", str(lib), str(src)], check=True)
    out = (C.c_ulonglong * 4)()
    assert C.CDLL(str(lib)).run(out) == 0
    assert list(out) == [0, 0, 0, 0], f"roots {out[0]}, reciprocal roots {out[1]}, range {out[2]}, quotients {out[3]}"
