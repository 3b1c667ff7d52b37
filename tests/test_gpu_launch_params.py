"""Launch parameters read from a world describe the plan it runs.

Setting what launch_params() reports must leave the contact pass's grid and
the sharing of its batches as they are. A world of b batches of 32 segments
shares each among four warps while b is at most half the resident warps (8
per block, p blocks per SM; all of them with lists of fewer than 64 entries),
in min(ceil(4 b / 8 or b / 8), p x SMs) blocks; untuned, p is 3. The least p
with the same plan is reported, and again once it has been set.
"""

import numpy as np
import pytest

from tangle_b200.assembly import Cell, FiberAssembly, PackedAssembly
from tangle_b200.settings import CellListConfig

pytestmark = pytest.mark.gpu


def straight_pairs(segments):
    assembly = FiberAssembly(Cell([4.0e-3] * 3, "xyz"))
    starts = np.random.default_rng(1).uniform(0.0, 4.0e-3, (segments // 40, 3))
    for start in starts:
        points = start + np.linspace([0.0, 0.0, 0.0], [8.0e-4, 0.0, 0.0], 41)
        assembly.add_fiber(points, radius=5.0e-6, min_bend_radius=1.0e-4)
    return PackedAssembly.from_assembly(assembly)


@pytest.mark.parametrize("batches", [5, 295, 300, 590, 940, 1180, 1190, 2400, 3600, 4800])
@pytest.mark.parametrize("capacity", [16, 64])
def test_set_of_get_leaves_the_contact_plan(batches, capacity, cuda_lib):
    import torch

    from tangle_b200.device import DeviceWorld

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    world = DeviceWorld(straight_pairs(batches * 32), CellListConfig(neighbor_capacity=capacity, max_list_bytes=1 << 28), 1.0e-6)
    b = (world.segment_count + 31) // 32

    def plan(p):
        shared = 4 if (1 if capacity < 64 else 2) * b <= 8 * p * sms else 1
        return min(-(-b * shared // 8), p * sms), shared

    params = world.launch_params()
    least = min(p for p in (1, 2, 3) if plan(p) == plan(3))
    assert params["contact_blocks_per_sm"] == least
    world.set_launch_params(params)
    assert world.launch_params() == params
    world.close()
