"""The autotuner times each plan once.

Different parameters can give one plan: 2 and 4 lanes per fiber are the same
kernel, a fiber too long for its strips raises them all to 32, and a small
world's contact pass has one grid for every count of blocks per SM. A search
tries 4, 8 and 32 lanes, five chunks, four skins and three block sizes of the
update, one parameter at a time from a world that has one of each.
"""

import numpy as np
import pytest

from tangle_b200.assembly import Cell, FiberAssembly, PackedAssembly
from tangle_b200.settings import CellListConfig, RelaxationConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vertices, lanes", [(20, 3), (500, 1)])
def test_trials_are_of_different_plans(vertices, lanes, cuda_lib):
    from tangle_b200.device import DeviceWorld

    side = 2.0e-5 * vertices
    assembly = FiberAssembly(Cell([max(side, 4.0e-4), 4.0e-4, 4.0e-4], "xyz"))
    for k in range(4):
        points = np.arange(vertices)[:, None] * np.array([2.0e-5, 0.0, 0.0]) + [0.0, 9.0e-6 * k, 1.0e-5]
        assembly.add_fiber(points, radius=5.0e-6, min_bend_radius=5.0e-5)
    cells = CellListConfig(neighbor_capacity=64, max_list_bytes=1 << 28)
    config = RelaxationConfig(penetration_tolerance=1.0e-9, max_step=5.0e-7, cell_list=cells)
    world = DeviceWorld(PackedAssembly.from_assembly(assembly), cells, config.max_step)
    _, report = world.autotune_trials(config, 4)
    assert report["trials"] == 1 + (lanes - 1) + (5 - 1) + (4 - 1) + (3 - 1)
    world.close()
