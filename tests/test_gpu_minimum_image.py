"""minimum_image shifts each axis as the division alone would.

A small program built from tangle_b200/csrc/common.cuh compares the second
segment that minimum_image moves, and whether it reports a move, with
roundf(separation / length) box lengths taken off axis by axis: every mix of
periodic and walled axes, separations near half and whole numbers of boxes
(where all three axes divide), up to 5,000 boxes, zeros, infinities and NaN.
The bits must be equal.
"""

import subprocess

import pytest

from tangle_b200.build import ROOT, nvcc

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "tangle_b200/csrc/common.cuh"
using namespace tgl;
typedef unsigned long long u64;
__device__ inline u64 mix(u64 x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__device__ inline float unit(u64 h) { return (float)(h >> 40) * 5.9604645e-8f; }
__device__ inline float separation(u64 h, float length) {
    const float boxes = floorf((unit(h) - 0.5f) * 10000.0f), near = boxes * length, small = (unit(mix(h)) - 0.5f) * 4.0e-6f;
    switch ((mix(h + 1) >> 20) % 10) {
        case 0: return (boxes + 0.5f) * length * (1.0f + small);
        case 1: return near * (1.0f + small);
        case 2: return (floorf((unit(h) - 0.5f) * 8.0f) + 0.5f) * length * (1.0f + small);
        case 3: return length * small;
        case 4: return (mix(h + 2) & 1) ? 0.0f : -0.0f;
        case 5: return (mix(h + 2) & 255) ? near : (mix(h + 2) & 256) ? INFINITY : NAN;
        default: return (unit(h) - 0.5f) * 8.0f * length;
    }
}
__global__ void compare(u64 cases, u64 *bad) {
    for (u64 i = blockIdx.x * 256ull + threadIdx.x; i < cases; i += gridDim.x * 256ull) {
        const u64 h = mix(i);
        Grid g{};
        float p1[3], q1[3], p2[3], q2[3], want_p[3], want_q[3];
        bool moved = false;
        for (int a = 0; a < 3; ++a) {
            g.length[a] = 1.0e-5f * (1.0f + 300.0f * unit(mix(h + 10 + a)));
            g.inv_length[a] = 1.0f / g.length[a];
            g.periodic[a] = (h >> a) & 1;
            p1[a] = (unit(mix(h + 20 + a)) - 0.5f) * g.length[a];
            q1[a] = p1[a] + 0.01f * g.length[a];
            const float d = separation(mix(h + 30 + a), g.length[a]);
            p2[a] = p1[a] + d;
            q2[a] = (h & 64) ? q1[a] + d : p2[a];
            if (h & 128) p1[a] = q1[a] = 0.0f, p2[a] = q2[a] = d;
            want_p[a] = p2[a], want_q[a] = q2[a];
            const float between = 0.5f * (p2[a] + q2[a] - p1[a] - q1[a]);
            if (g.periodic[a]) {
                const float images = roundf(between / g.length[a]);
                want_p[a] -= images * g.length[a];
                want_q[a] -= images * g.length[a];
                moved |= images != 0.0f;
            }
        }
        const bool got = minimum_image(p1[0], p1[1], p1[2], q1[0], q1[1], q1[2], p2[0], p2[1], p2[2], q2[0], q2[1], q2[2], g);
        bool same = got == moved;
        for (int a = 0; a < 3; ++a)
            same = same && (isnan(want_p[a]) ? isnan(p2[a]) : __float_as_uint(p2[a]) == __float_as_uint(want_p[a])) &&
                   (isnan(want_q[a]) ? isnan(q2[a]) : __float_as_uint(q2[a]) == __float_as_uint(want_q[a]));
        if (!same) atomicAdd(bad, 1ull);
        if (moved) atomicAdd(bad + 1, 1ull);
    }
}
int main() {
    u64 *d, h[2];
    cudaMalloc(&d, sizeof(h));
    cudaMemset(d, 0, sizeof(h));
    compare<<<1184, 256>>>(200000000ull, d);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("%llu %llu\n", h[0], h[1]);
    return 0;
}
"""


def test_minimum_image_matches_the_division_on_every_axis(tmp_path):
    source = tmp_path / "minimum_image.cu"
    source.write_text(PROGRAM)
    program = str(tmp_path / "minimum_image")
    subprocess.run([nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-ftz=false", "-I", ROOT, "-o", program, str(source)],
                   check=True, capture_output=True)
    different, moved = subprocess.run([program], check=True, capture_output=True, text=True).stdout.split()
    assert int(different) == 0 and int(moved) > 10_000_000
