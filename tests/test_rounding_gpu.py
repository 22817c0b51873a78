"""The quotients and roots of csrc/internal.cuh against CUDA's correctly rounded ones.

They decide where footprints begin and end, so a last bit matters. A reciprocal or a root has one
operand: all of the declared range is compared. A corrected quotient can only go wrong next to a
rounding midpoint, where random operands hardly ever fall: the numerators that lie 1, 2, ... units
from one are computed for every odd 24-bit denominator.
"""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "internal.cuh"
using namespace elsa_b200;
typedef unsigned long long u64;

static __device__ void differ(float got, float want, u64* count)
{
    if (__float_as_uint(got) != __float_as_uint(want))
        atomicAdd(count, 1ull);
}

// every float in [2^-40, 2^40]; count[0..3]: reciprocals, pairs of them, roots, pairs of roots
static __global__ void unary(u64* count)
{
    const u64 all = 80ull << 23, first = 87ull << 23; // 2^-40
    for (u64 i = blockIdx.x * (u64) blockDim.x + threadIdx.x; i <= all;
         i += (u64) gridDim.x * blockDim.x) {
        const float v = __uint_as_float((unsigned) (first + i));
        const float y = refineRcp(v, rcpApprox(v));
        differ(y, __frcp_rn(v), count);
        const float2 y2 = refineRcp2(make_float2(v, -v),
                                     make_float2(rcpApprox(v), rcpApprox(-v)));
        differ(y2.x, y, count + 1);
        differ(y2.y, -y, count + 1);
        differ(root(v), __fsqrt_rn(v), count + 2);
        const float2 r = root2(make_float2(v, v));
        differ(r.x, __fsqrt_rn(v), count + 3);
        differ(r.y, __fsqrt_rn(v), count + 3);
    }
}

static __device__ void quotients(float a, float b, u64* count)
{
    const float want = __fdiv_rn(a, b);
    differ(quotient(a, b, refineRcp(b, rcpApprox(b))), want, count);
    const float y = rcpApprox(b);
    const float2 q = quotient2(make_float2(a, -a), make_float2(b, b),
                               refineRcp2(make_float2(b, b), make_float2(y, y)));
    differ(q.x, want, count + 1);
    if (a != 0.0f) // (a numerator of -0 gives +0)
        differ(q.y, -want, count + 1);
    // the denominator as a root (b^2 rounded has the root b, or one next to it)
    float norm;
    const float q1 = overRoot(a, b * b, norm);
    differ(q1, __fdiv_rn(a, __fsqrt_rn(b * b)), count + 2);
}

// denominators B = 2^23 + 1, + 3, ...; numerators A with A 2^25 = M B + r: for odd M the quotient
// A / B is |r| / (2^25 B) from a midpoint
static __global__ void midpoints(int scaleA, int scaleB, u64* count)
{
    for (u64 k = blockIdx.x * (u64) blockDim.x + threadIdx.x; k < (1ull << 22);
         k += (u64) gridDim.x * blockDim.x) {
        const u64 B = (1ull << 23) + 2 * k + 1;
        u64 inverse = 1; // of 2^25 modulo B
        for (int i = 0; i < 25; ++i)
            inverse = inverse % 2 ? (inverse + B) / 2 : inverse / 2;
        for (int r = -6; r <= 6; ++r) {
            u64 A = r >= 0 ? r * inverse % B : B - (-r) * inverse % B;
            if (A == 0 || A >= B)
                continue;
            while (A < (1ull << 23)) // the same quotient, doubled
                A *= 2;
            quotients(ldexpf((float) A, scaleA - 23), ldexpf((float) B, scaleB - 23), count);
        }
    }
}

// random operands of the declared range, and denominators next to 2 (all-ones significands)
static __global__ void anything(u64 seed, u64* count)
{
    u64 s = seed + (blockIdx.x * (u64) blockDim.x + threadIdx.x) * 0x9E3779B97F4A7C15ull;
    auto next = [&] {
        s += 0x9E3779B97F4A7C15ull;
        u64 z = (s ^ (s >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    };
    for (int i = 0; i < 512; ++i) {
        const u64 x = next(), w = next();
        const float a = __uint_as_float((unsigned) ((87 + x % 80) << 23 | (x >> 40 & 0x7FFFFF)));
        unsigned m = (unsigned) (w >> 40) & 0x7FFFFF;
        if (i % 3 == 0)
            m = 0x7FFFFF - m % 64;
        // (the square of a root's operand stays in the range)
        const float b = __uint_as_float((unsigned) ((107 + w % 40) << 23 | m));
        quotients(a, b, count);
        quotients(0.0f, b, count);
    }
}

extern "C" int run(u64* host) // 7 counts; returns a CUDA error code
{
    u64* count;
    cudaError_t e = cudaMalloc(&count, 7 * sizeof(u64));
    if (e != cudaSuccess)
        return e;
    cudaMemset(count, 0, 7 * sizeof(u64));
    unary<<<148 * 8, 256>>>(count);
    for (int scale = -20; scale <= 20; scale += 10) {
        midpoints<<<148 * 8, 256>>>(0, scale, count + 4);
        midpoints<<<148 * 8, 256>>>(-2 * scale, 0, count + 4);
    }
    anything<<<148 * 16, 256>>>(1, count + 4);
    e = cudaMemcpy(host, count, 7 * sizeof(u64), cudaMemcpyDeviceToHost);
    cudaFree(count);
    return e;
}
"""


def test_quotients_and_roots_are_correctly_rounded(cuda, tmp_path):
    from elsa_b200 import build
    src, lib = tmp_path / "rounding.cu", tmp_path / "librounding.so"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, *build.ARCH, *build.CUDA_FLAGS, "--fmad=false",
                    "-I" + build.CSRC, "-shared", str(src), "-o", str(lib), "-lcudart"],
                   check=True, capture_output=True)
    counts = (ctypes.c_ulonglong * 7)()
    assert ctypes.CDLL(str(lib)).run(counts) == 0
    rcp, rcp2, roots, roots2, scalar, pairs, of_root = counts
    assert rcp == 0 and rcp2 == 0 and roots == 0 and roots2 == 0
    assert scalar == 0 and pairs == 0 and of_root == 0
