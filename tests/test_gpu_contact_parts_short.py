"""Shared batches whose segments scan their cells: the oracle's bits.

With Verlet lists of fewer than 64 entries, four warps share a batch while
the batches are at most the resident warps, and take the parts from the
counter once those are more than the warps. Worlds on each side of both
lines, with lists of 8 entries that nearly all overflow.
"""

import numpy as np
import pytest

from tangle_b200.assembly import PackedAssembly
from tangle_b200.generate import mid_size_specimen
from tangle_b200.settings import CellListConfig, RelaxationConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fibers", [60, 250, 600, 1000, 1100])
def test_scanned_parts_match_the_oracle(fibers, cuda_lib):
    from oracle import OracleWorld
    from tangle_b200.device import DeviceWorld

    packed = PackedAssembly.from_assembly(mid_size_specimen(scale=(fibers / 20000.0) ** (1.0 / 3.0), seed=fibers))
    cells = CellListConfig(neighbor_capacity=8, max_list_bytes=1 << 30)
    config = RelaxationConfig(penetration_tolerance=1.0e-9, force_full_iterations=True, max_step=1.0e-6, cell_list=cells)
    dev, orc = DeviceWorld(packed, cells, config.max_step), OracleWorld(packed, cells, config.max_step)
    assert dev.run_batch(config, 2).max_penetration == orc.run_batch(config, 2).max_penetration
    counts, _ = dev.debug_neighbor_lists_raw()
    assert (counts > 8).mean() > 0.5
    np.testing.assert_array_equal(dev.download_positions().view(np.uint32), orc.download_positions().view(np.uint32))
    dev.close()
    orc.close()
