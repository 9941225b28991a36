"""The branch-free square root, reciprocal and quotient of vmath.cuh against
CUDA's built-in ones, bit for bit over the ranges they are used in: every
mantissa for the square root (two exponent parities) and the reciprocal, and
for the quotient random operands and divisors with extreme mantissas.  The
kernel that compares them is compiled here from the header itself."""
import ctypes as C
import subprocess

import pytest

from seevr_b200.build import ARCH, CSRC, NVCC

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
#include "vmath.cuh"
using namespace seevr;
__device__ unsigned next(unsigned& s) { s ^= s << 13; s ^= s >> 17; s ^= s << 5; return s; }
__global__ void k_compare(unsigned long long* bad) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, n = gridDim.x * blockDim.x;
    // root: 2^-67 .. 2^63, both parities (a root's mantissa lies in [1, 1.41) or
    // [1.41, 2) with the parity); reciprocals: 2^-27 .. 2^23
    const unsigned exps[6] = {60u, 100u, 126u, 127u, 150u, 189u};
    for (unsigned m = t; m < (1u << 23); m += n)
        for (unsigned e : exps) {
            const float a = __uint_as_float((e << 23) | m);
            const float r = rsqrt_approx(a), root = sqrtf(a);
            if (root_of(a, r) != root) atomicAdd(&bad[0], 1ull);
            if (e >= 90u && e <= 160u) {
                if (recip_of(a, rcp_approx(a)) != 1.0f / a) atomicAdd(&bad[1], 1ull);
                if (recip_of(root, rcp_approx(root)) != 1.0f / root) atomicAdd(&bad[2], 1ull);
            }
        }
    unsigned s = 2654435761u * (t + 1u);
    for (int i = 0; i < 4096; ++i) {
        // x in 2^[-82, 82], y in 2^[-39, 39]; every eighth divisor or dividend
        // has the mantissa 1.11..1 or 1.00..0
        const unsigned xs = next(s), ys = next(s), k = next(s);
        unsigned xm = xs & 0x7fffffu, ym = ys & 0x7fffffu;
        if ((k & 7u) == 0u) ym = (k & 8u) ? 0x7fffffu : 0u;
        if ((k & 7u) == 1u) xm = (k & 8u) ? 0x7fffffu : 0u;
        const float x = __uint_as_float((xs & 0x80000000u) | ((45u + (k >> 8) % 165u) << 23) | xm);
        const float y = __uint_as_float(((88u + (k >> 20) % 78u) << 23) | ym);
        const float q = div_by(x, y, recip_of(y, rcp_approx(y)));
        const bool ok = size_key(x) >= kNumMinKey && fabsf(x) <= kNumMax;
        if (ok && q != x / y) atomicAdd(&bad[3], 1ull);
        if (ok != (fabsf(x) >= kNumMin && fabsf(x) <= kNumMax)) atomicAdd(&bad[4], 1ull);
    }
    const float z = div_by(-0.0f, 3.0f, recip_of(3.0f, rcp_approx(3.0f)));
    if (__float_as_uint(z) != 0x80000000u || size_key(-0.0f) < kNumMinKey ||
        size_key(0.0f) < kNumMinKey || size_key(kNumMin) != kNumMinKey ||
        size_key(1e-30f) >= kNumMinKey)
        atomicAdd(&bad[5], 1ull);
}
extern "C" int compare(unsigned long long out[6]) {
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, 48) != cudaSuccess || cudaMemset(d, 0, 48) != cudaSuccess) return 1;
    k_compare<<<592, 256>>>(d);
    const int e = cudaMemcpy(out, d, 48, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
"""


def test_branch_free_root_and_quotient_equal_the_builtin_ones(cuda, tmp_path):
    src, lib = tmp_path / "compare.cu", tmp_path / "compare.so"
    src.write_text(SOURCE)
    subprocess.run([NVCC, *ARCH, "-O3", "-std=c++17", "-fmad=false", "-I", str(CSRC), "-shared",
                    "-Xcompiler", "-fPIC", "-o", str(lib), str(src)], check=True)
    bad = (C.c_ulonglong * 6)()
    assert C.CDLL(str(lib)).compare(bad) == 0
    assert list(bad) == [0] * 6, "root, reciprocal, reciprocal of a root, quotient, range, zeros"
