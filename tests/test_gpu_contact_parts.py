"""A contact batch's segments taken by one warp or shared by four: same bits.

Four warps share a batch of 32 segments while the batches number at most the
resident warps, so a world takes either way as the blocks per SM change (900
fibers: one, one, four) and as fibers are added; with Verlet lists of 8
entries the segments take the cell scan. Positions and penetration are the
oracle's.
"""

import numpy as np
import pytest

from tangle_b200.assembly import PackedAssembly
from tangle_b200.generate import mid_size_specimen
from tangle_b200.settings import CellListConfig, RelaxationConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fibers, capacity", [(40, 8), (40, 256), (900, 256), (2000, 256), (3500, 256)])
def test_shared_batches_match_the_oracle(fibers, capacity, cuda_lib):
    from oracle import OracleWorld
    from tangle_b200.device import DeviceWorld

    packed = PackedAssembly.from_assembly(mid_size_specimen(scale=(fibers / 20000.0) ** (1.0 / 3.0), seed=fibers))
    cells = CellListConfig(neighbor_capacity=capacity, max_list_bytes=1 << 31)
    config = RelaxationConfig(penetration_tolerance=1.0e-9, force_full_iterations=True, max_step=1.0e-6, cell_list=cells)
    orc = OracleWorld(packed, cells, config.max_step)
    want_status = orc.run_batch(config, 3)
    want = orc.download_positions().view(np.uint32)
    orc.close()
    for blocks in (1, 2, 3):
        dev = DeviceWorld(packed, cells, config.max_step)
        dev.set_launch_params(dict(dev.launch_params(), contact_blocks_per_sm=blocks))
        status = dev.run_batch(config, 3)
        assert status.max_penetration == want_status.max_penetration
        np.testing.assert_array_equal(dev.download_positions().view(np.uint32), want)
        dev.close()
