"""The short exact division (tfx_exact_math.cuh) over its stated ranges: every pair of a numerator's and a divisor's
exponent at and inside the ends of kDivMin..kDivMax and kDivisorMin..kDivisorMax, with spread significands, both
signs and the range's end points themselves, against the operator, bit for bit."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include "tfx_exact_math.cuh"
using namespace tfx;
__device__ int exponent(float x) { return (int)(__float_as_uint(x) >> 23); }
__global__ void ranges(unsigned long long* out) {
    const int ea = exponent(kDivMin) + blockIdx.x, eb = exponent(kDivisorMin) + blockIdx.y;
    unsigned long long bad = 0, done = 0;
    for (unsigned k = threadIdx.x; k < 16384; k += blockDim.x) {
        const unsigned h = (k * 2654435761u) ^ (blockIdx.x * 40503u + blockIdx.y * 9973u);
        const unsigned ma = k < 64 ? k & 7 : k < 128 ? 0x7fffffu - (k & 7) : h & 0x7fffffu;
        const unsigned mb = k < 64 ? (k >> 3) & 7 : k < 128 ? 0x7fffffu - ((k >> 3) & 7) : (h * 747796405u >> 9);
        float a = __uint_as_float(((unsigned)ea << 23) | ma), b = __uint_as_float(((unsigned)eb << 23) | mb);
        if (a < kDivMin || a > kDivMax || b < kDivisorMin || b > kDivisorMax) continue;
        if (k & 1) a = -a;
        if (k & 2) b = -b;
        const float q = div_by(a, b, __fdiv_rn(1.0f, b)), r = __fdiv_rn(a, b);
        bad += __float_as_uint(q) != __float_as_uint(r);
        ++done;
    }
    atomicAdd(out, bad);
    atomicAdd(out + 1, done);
}
extern "C" int run(unsigned long long* out) {
    unsigned long long* d;
    if (cudaMalloc(&d, 16) != cudaSuccess || cudaMemset(d, 0, 16) != cudaSuccess) return 1;
    ranges<<<dim3(NA, 81), 128>>>(d);   // every exponent of a's range, every one of b's
    const cudaError_t e = cudaMemcpy(out, d, 16, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
"""


def test_quotients_at_the_ends_of_the_ranges(tmp_path):
    from tressfx_gb300 import build as B
    src, lib = tmp_path / "ranges.cu", tmp_path / "libranges.so"
    src.write_text(SOURCE)
    subprocess.run([str(B._cuda_home() / "bin" / "nvcc"), *B.nvcc_flags(), "-DNA=141", "-shared", "-o", str(lib), str(src)], check=True)
    out = (C.c_ulonglong * 2)()
    assert C.CDLL(str(lib)).run(out) == 0
    assert out[1] > 150_000_000 and out[0] == 0, f"{out[0]} of {out[1]} quotients differ"
