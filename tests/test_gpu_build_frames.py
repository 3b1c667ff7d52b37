"""The Verlet build's staged spheres, in the home cell's frame, lose no pair.

The sphere test takes a candidate's image from its stencil cell where every
periodic axis has at least four cells, and the nearest image with three; the
scan joins neighboring cells and queues two rounds at a time. Lists of short
random fibers, unwrapped by up to three box lengths, with 2 to 6 cells per
axis and crowded and empty cells, equal the oracle's.
"""

import numpy as np
import pytest

from tangle_b200.assembly import Cell, FiberAssembly, PackedAssembly
from tangle_b200.settings import CellListConfig

pytestmark = pytest.mark.gpu

RADIUS = 0.5e-5


def scattered(cells, periodic, count, seed):
    rng = np.random.default_rng(seed)
    width = 8.0 * RADIUS  # a segment of four radii, its capsule's ends and the skin
    lengths = np.array(cells) * width * 1.02
    assembly = FiberAssembly(Cell(list(lengths), periodic))
    for k in range(count):
        n = int(rng.integers(2, 5))
        steps = rng.normal(size=(n - 1, 3))
        steps *= 4.0 * RADIUS / np.linalg.norm(steps, axis=1)[:, None]
        points = np.concatenate([np.zeros((1, 3)), np.cumsum(steps, axis=0)])
        points += rng.uniform(0.0, 1.0, 3) ** (1 + k % 2) * lengths  # half of them crowd one corner
        for axis, name in enumerate("xyz"):
            if name in periodic:
                points[:, axis] += rng.integers(-3, 4) * lengths[axis]
            else:
                points[:, axis] = np.clip(points[:, axis], RADIUS, lengths[axis] - RADIUS)
        assembly.add_fiber(points, radius=RADIUS, min_bend_radius=1.0e-6)
    return assembly


@pytest.mark.parametrize("count", [1, 33, 700])
@pytest.mark.parametrize("periodic", ["xyz", "xy", ""])
@pytest.mark.parametrize("cells", [(2, 3, 4), (3, 3, 3), (4, 4, 4), (5, 3, 6), (6, 5, 4)], ids=str)
def test_lists_equal_the_oracles(cells, periodic, count, cuda_lib):
    from oracle import OracleWorld
    from tangle_b200.device import DeviceWorld

    packed = PackedAssembly.from_assembly(scattered(cells, periodic, count, sum(cells) + count))
    config = CellListConfig(neighbor_capacity=2048, max_list_bytes=1 << 30)
    step = 1.0e-7
    dev, orc = DeviceWorld(packed, config, step), OracleWorld(packed, config, step)
    dev.debug_rebuild()
    orc.debug_rebuild()
    (counts, lists), (oracle_counts, oracle_lists) = dev.debug_neighbor_lists(), orc.debug_neighbor_lists()
    np.testing.assert_array_equal(counts, oracle_counts)
    for mine, theirs in zip(lists, oracle_lists):
        np.testing.assert_array_equal(mine, theirs)
    dev.close()
    orc.close()
