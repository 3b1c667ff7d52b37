"""Compaction of a periodic axis past the contact lists' single-image bounds.

With half lengths H, radii r and a contact skin s the lists hold while every
periodic edge L keeps L / 2 > 2 H + 2 r + s (less 0.1 % of H). A cell that
leaves room for the narrow skin (a tenth of the neighbor skin) but not for
the wide one (2.5 times that) keeps narrow lists: nearly still fibers refresh
them once, not in every pass. In a cell without room for either every pass
is a refresh while a segment is too long. Positions are the oracle's.
"""

import numpy as np
import pytest

from tangle_b200.assembly import Cell, FiberAssembly, PackedAssembly
from tangle_b200.formation import CompactionKinematics
from tangle_b200.settings import CellListConfig, RelaxationConfig

pytestmark = pytest.mark.gpu

RADIUS, STEP = 5.0e-6, 2.0e-5
EDGE = 2.0 * (STEP / 0.999 + 2.0 * RADIUS)  # without a skin
NARROW = 2.0 * RADIUS * 0.1                 # neighbor skin: two radii


def bundle(edge):
    rng = np.random.default_rng(8)
    assembly = FiberAssembly(Cell([edge, 3.0e-4, 3.0e-4], "xyz"))
    for _ in range(60):
        turn = rng.normal(scale=0.1, size=(9, 3)) * [0.3, 1.0, 1.0]
        steps = np.array([0.05, 1.0, 0.4]) + turn
        steps *= STEP / np.linalg.norm(steps, axis=1)[:, None]
        points = np.concatenate([np.zeros((1, 3)), np.cumsum(steps, axis=0)])
        assembly.add_fiber(points + rng.uniform(0.0, 1.0, 3) * [edge, 3.0e-4, 3.0e-4], radius=RADIUS,
                           min_bend_radius=2.0e-5)
    return PackedAssembly.from_assembly(assembly)


@pytest.mark.parametrize("room, refreshes", [(6.0 * NARROW, 2), (2.0 * 1.7 * NARROW, 2), (2.0 * 0.5 * NARROW, 13)],
                         ids=["wide", "narrow", "neither"])
def test_lists_after_a_compaction(room, refreshes, cuda_lib):
    from oracle import OracleWorld
    from tangle_b200.device import DeviceWorld

    packed = bundle(EDGE + 10.0 * NARROW)
    cells = CellListConfig(neighbor_capacity=512, max_list_bytes=1 << 28)
    config = RelaxationConfig(penetration_tolerance=1.0e-9, force_full_iterations=True, max_step=1.0e-9, cell_list=cells)
    dev, orc = DeviceWorld(packed, cells, config.max_step), OracleWorld(packed, cells, config.max_step)
    assert dev.contact_list_info()["skin"] > 0.0
    for world in (dev, orc):
        world.run_batch(config, 2)
        world.compact_cell([0.0, 0.0, 0.0], [EDGE + room, 3.0e-4, 3.0e-4], CompactionKinematics.RIGID_FIBER_CENTERS)
    before = dev.contact_list_info()["refreshes"]
    for world in (dev, orc):
        world.run_batch(config, 12)
    info = dev.contact_list_info()  # 12 iterations, 13 passes
    assert info["skin"] > 0.0 and 1 <= info["refreshes"] - before <= refreshes
    np.testing.assert_array_equal(dev.download_positions().view(np.uint32), orc.download_positions().view(np.uint32))
    dev.close()
    orc.close()
