"""The branch-free square root, reciprocal, quotient and arc cosine of
tangle_b200/csrc/common.cuh round as the general operators do.

A small program built from that header checks, on the GPU: the square root
and the reciprocal of every float in [2^-80, 2^81); acos_plain against
acos_f32 on every float of [-1, 1]; and quotients (general operator against
div_plain) of 2 x 10^9 operand pairs, half of them with the quotient next to
a rounding boundary, one in seven with a divisor's significand near 2.
Whole numbers of mismatches, no tolerance: each must be 0.
"""

import os
import subprocess

import pytest

from tangle_b200.build import ROOT, nvcc

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "tangle_b200/csrc/common.cuh"
using namespace tgl;
typedef unsigned long long u64;
__device__ inline float pack(unsigned exponent, unsigned significand) {
    return __uint_as_float((exponent << 23) | (significand & 0x7fffffu));
}
__global__ void roots(u64 *bad) {
    for (u64 i = blockIdx.x * 256ull + threadIdx.x; i < (161ull << 23); i += gridDim.x * 256ull) {
        const float a = pack((unsigned)(i >> 23) + 47u, (unsigned)i);
        if (__float_as_uint(sqrt_plain(a)) != __float_as_uint(sqrtf(a))) atomicAdd(bad, 1ull);
        if (__float_as_uint(reciprocal_plain(a)) != __float_as_uint(__frcp_rn(a))) atomicAdd(bad + 1, 1ull);
    }
}
__device__ inline u64 mix(u64 x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__global__ void quotients(u64 pairs, u64 *bad) {
    for (u64 i = blockIdx.x * 256ull + threadIdx.x; i < pairs; i += gridDim.x * 256ull) {
        const u64 h = mix(i);
        const unsigned m = (unsigned)(h >> 23) & 0x7fffffu;
        float b = pack((unsigned)((h >> 46) % 120) + 67u, (unsigned)h);
        if (i % 7 == 0) b = __uint_as_float(__float_as_uint(b) | 0x7fff00u);
        float a = pack((unsigned)((h >> 53) % 120) + 67u, m);
        if (h >> 63) a = -a;
        if (i & 1) a = (float)(((double)__uint_as_float(0x3f800000u | m) + 5.9604644775390625e-08) * (double)b);
        if (__float_as_uint(div_plain(a, b, reciprocal_plain(b))) != __float_as_uint(a / b)) atomicAdd(bad, 1ull);
    }
}
__global__ void arcs(u64 *bad) {
    for (unsigned i = blockIdx.x * 256u + threadIdx.x; i <= 0x3f800000u; i += gridDim.x * 256u) {
        const float x = __uint_as_float(i);
        if (__float_as_uint(acos_plain(x)) != __float_as_uint(acos_f32(x)) ||
            __float_as_uint(acos_plain(-x)) != __float_as_uint(acos_f32(-x)))
            atomicAdd(bad, 1ull);
    }
}
int main() {
    u64 *d, h[4];
    cudaMalloc(&d, sizeof(h));
    cudaMemset(d, 0, sizeof(h));
    roots<<<1184, 256>>>(d);
    quotients<<<1184, 256>>>(2000000000ull, d + 2);
    arcs<<<1184, 256>>>(d + 3);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("%llu %llu %llu %llu\n", h[0], h[1], h[2], h[3]);
    return 0;
}
"""


def test_plain_operations_round_as_the_general_ones(tmp_path):
    source = tmp_path / "plain_math.cu"
    source.write_text(PROGRAM)
    program = str(tmp_path / "plain_math")
    subprocess.run([nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-ftz=false", "-I", ROOT, "-o", program, str(source)],
                   check=True, capture_output=True, env=dict(os.environ))
    out = subprocess.run([program], check=True, capture_output=True, text=True).stdout
    assert [int(v) for v in out.split()] == [0, 0, 0, 0], "square roots, reciprocals, quotients, arc cosines that differ"
