"""Fibers whose edges have components that are exactly zero.

Planar fibers, staircases along the axes and straight ones put exact zeros
into the sweeps' quotients. div_plain keeps the sign of a zero numerator (a
small program checks every divisor of its range), and positions are the
oracle's bit for bit for planes across each axis, at a positive, a zero and a
negative zero height, sharply bent and staircase, periodic and between walls.
"""

import subprocess

import numpy as np
import pytest

from tangle_b200.assembly import Cell, FiberAssembly, PackedAssembly
from tangle_b200.build import ROOT, nvcc
from tangle_b200.settings import CellListConfig, RelaxationConfig

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "tangle_b200/csrc/common.cuh"
using namespace tgl;
__global__ void zeros(unsigned long long *bad) {
    for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < (160ull << 23); i += gridDim.x * 256ull) {
        const float b = __uint_as_float(((unsigned)(i >> 23) + 47u) << 23 | ((unsigned)i & 0x7fffffu)), y = reciprocal_plain(b);
        if (__float_as_uint(div_plain(0.0f, b, y)) != 0u || __float_as_uint(div_plain(-0.0f, b, y)) != 0x80000000u)
            atomicAdd(bad, 1ull);
    }
}
int main() {
    unsigned long long *d, h;
    cudaMalloc(&d, sizeof(h));
    cudaMemset(d, 0, sizeof(h));
    zeros<<<1184, 256>>>(d);
    if (cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("%llu\n", h);
    return 0;
}
"""


def test_quotients_of_zero_keep_their_sign(tmp_path):
    source = tmp_path / "zeros.cu"
    source.write_text(PROGRAM)
    program = str(tmp_path / "zeros")
    subprocess.run([nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-ftz=false",
                    "-prec-div=true", "-prec-sqrt=true", "-I", ROOT, "-o", program, str(source)], check=True, capture_output=True)
    assert int(subprocess.run([program], check=True, capture_output=True, text=True).stdout) == 0


@pytest.mark.parametrize("lanes", [4, 8, 32])
@pytest.mark.parametrize("periodic", ["xyz", "xy", ""])
@pytest.mark.parametrize("shape", ["bent", "stairs", "straight"])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_planar_fibers_match_the_oracle(axis, shape, periodic, lanes, cuda_lib):
    from oracle import OracleWorld
    from tangle_b200.device import DeviceWorld

    rng = np.random.default_rng(axis + 10 * lanes)
    step, side = 2.0e-5, 4.0e-4
    assembly = FiberAssembly(Cell([side] * 3, periodic, origin=[-0.5 * side] * 3))
    heights = [0.0, -0.0, 1.3e-5, -2.7e-5, 6.1e-5]
    for k in range(20):
        n = int(rng.integers(3, 45))
        in_plane = np.zeros((n - 1, 3))
        first, second = [a for a in range(3) if a != axis]
        if shape == "bent":
            in_plane[:, first], in_plane[:, second] = rng.normal(1.0, 0.7, n - 1), rng.normal(0.0, 0.7, n - 1)
        elif shape == "stairs":
            turn = np.arange(n - 1) % 2 == 1
            in_plane[~turn, first], in_plane[turn, second] = 1.0, rng.choice([-1.0, 1.0])
        else:
            in_plane[:, first] = 1.0
        in_plane *= step / np.linalg.norm(in_plane, axis=1)[:, None]
        points = np.concatenate([np.zeros((1, 3)), np.cumsum(in_plane, axis=0)]) + rng.uniform(-0.4, 0.4, 3) * side
        for a, name in enumerate("xyz"):
            if name not in periodic:
                points[:, a] = np.abs((points[:, a] + 1.5 * side) % (2.0 * 0.9 * side) - 0.9 * side) - 0.45 * side
        points[:, axis] = heights[k % len(heights)]
        assembly.add_fiber(points, radius=0.25 * step, min_bend_radius=2.5 * step)
    packed = PackedAssembly.from_assembly(assembly)
    cells = CellListConfig(neighbor_capacity=128, max_list_bytes=1 << 28)
    config = RelaxationConfig(penetration_tolerance=1.0e-8, force_full_iterations=True, max_step=1.0e-6,
                              constraint_iterations=2, curvature_cleanup_sweeps=3, cell_list=cells)
    dev, orc = DeviceWorld(packed, cells, config.max_step), OracleWorld(packed, cells, config.max_step)
    dev.set_launch_params(dict(dev.launch_params(), lanes_per_fiber=lanes))
    for batch in (1, 5):
        assert dev.run_batch(config, batch).max_curvature_ratio == orc.run_batch(config, batch).max_curvature_ratio
        np.testing.assert_array_equal(dev.download_positions().view(np.uint32), orc.download_positions().view(np.uint32))
        np.testing.assert_array_equal(dev.wall_reactions().view(np.uint32), orc.wall_reactions().view(np.uint32))
    dev.close()
    orc.close()
