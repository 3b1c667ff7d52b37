"""The curvature sweeps' strips at the sizes where they can go wrong.

Fibers of every length around the ends of strips and of the lanes that share
a fiber (a strip holds 5 to 29 triplets; 4, 8, 16 or 32 lanes; up to 930
vertices in the grouped kernel, longer ones in the one-warp kernel), bent
far past their limit so that most triplets act and strips hand moved
vertices on, with pinned and straight stretches, in a periodic box and
between walls. Positions and wall reactions are the oracle's bit for bit.
"""

import numpy as np
import pytest

from tangle_b200.assembly import Cell, FiberAssembly, PackedAssembly
from tangle_b200.settings import CellListConfig, RelaxationConfig

pytestmark = pytest.mark.gpu

LENGTHS = {
    "short": [2, 3, 4, 6, 7, 8, 12, 13, 22, 31],
    "strips": [41, 42, 43, 47, 58, 59, 82, 83, 106, 118, 119],
    "raised_16": [162, 163, 226, 234, 235, 236],
    "raised_32": [290, 466, 467],
    "longest": [898, 930],
    "one_warp": [931],
}


def bent_fibers(lengths, periodic, seed):
    """Random walks of 2 d steps: sharp bends on the first fiber of each
    length, a straight middle third on the second."""
    rng = np.random.default_rng(seed)
    d = 1.0e-5
    side = 4.0e-4
    assembly = FiberAssembly(Cell([side, side, 0.3 * side], periodic))
    for n in lengths:
        for kind in range(2):
            turn = rng.normal(scale=0.5, size=(n - 1, 3))
            if kind == 1:
                turn[(n - 1) // 3: 2 * (n - 1) // 3] = 0.0
            steps = np.array([1.0, 0.2, 0.1]) + turn
            steps *= 2.0 * d / np.linalg.norm(steps, axis=1)[:, None]
            points = np.concatenate([np.zeros((1, 3)), np.cumsum(steps, axis=0)])
            points[:, 2] = 0.15 * side + 0.13 * side * np.sin(points[:, 2] / (4.0 * d))
            points[:, :2] += rng.uniform(0.0, side, 2)
            if "x" not in periodic:
                points[:, :2] = d + np.abs((points[:, :2] - d) % (2.0 * (side - 2.0 * d)) - (side - 2.0 * d))
            assembly.add_fiber(points, radius=0.5 * d, min_bend_radius=5.0 * d)
    return assembly


@pytest.mark.parametrize("lanes", [2, 4, 8, 32])
@pytest.mark.parametrize("periodic", ["xyz", "xy", ""])
@pytest.mark.parametrize("lengths", list(LENGTHS), ids=list(LENGTHS))
def test_strips_match_the_serial_sweep(lengths, periodic, lanes, cuda_lib):
    from oracle import OracleWorld
    from tangle_b200.device import DeviceWorld

    packed = PackedAssembly.from_assembly(bent_fibers(LENGTHS[lengths], periodic, seed=len(periodic) + 7))
    rng = np.random.default_rng(3)
    packed.vertex_pinned[rng.integers(0, packed.vertex_count, packed.vertex_count // 16)] = 1
    packed.vertex_max_curvature[rng.integers(0, packed.vertex_count, packed.vertex_count // 16)] = 0.0
    cells = CellListConfig(neighbor_capacity=128, max_list_bytes=1 << 30)
    config = RelaxationConfig(penetration_tolerance=1.0e-8, force_full_iterations=True, max_step=1.0e-6,
                              constraint_iterations=1 + lanes % 3, curvature_cleanup_sweeps=3, cell_list=cells)
    dev = DeviceWorld(packed, cells, config.max_step)
    dev.set_launch_params(dict(dev.launch_params(), lanes_per_fiber=lanes))
    orc = OracleWorld(packed, cells, config.max_step)
    for batch in (1, 4):
        assert dev.run_batch(config, batch).max_curvature_ratio == orc.run_batch(config, batch).max_curvature_ratio
        np.testing.assert_array_equal(dev.download_positions().view(np.uint32),
                                      orc.download_positions().view(np.uint32))
        np.testing.assert_array_equal(dev.wall_reactions().view(np.uint32), orc.wall_reactions().view(np.uint32))
    dev.close()
    orc.close()
