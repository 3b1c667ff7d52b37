"""Contact lists are wide while the packing moves fast, and narrow else.

A refresh takes a skin of 2.5 times the narrow one unless the lists before
lasted seven passes. Lists of a fresh packing hold more entries than narrow
ones made at the same positions; once it hardly moves, refreshes (forced here
by new Verlet lists) keep the width they find, and lists that end by a move
after many passes are narrow again.
"""

import numpy as np
import pytest

from tangle_b200.assembly import PackedAssembly
from tangle_b200.generate import mid_size_specimen
from tangle_b200.settings import RelaxationConfig, RelaxationSettings

pytestmark = pytest.mark.gpu


def test_lists_follow_the_motion(cuda_lib):
    from tangle_b200.device import CONTACT_USE_VERLET, DeviceWorld

    assembly = mid_size_specimen(scale=0.3, seed=2)
    config = RelaxationSettings(penetration_tolerance=1.0e-3 * assembly.smallest_diameter(), neighbor_capacity=256,
                                max_list_bytes=1 << 30).to_config(assembly.smallest_diameter())
    fast = RelaxationConfig(**{**config.__dict__, "force_full_iterations": True})
    still = RelaxationConfig(**{**fast.__dict__, "max_step": 1.0e-13, "stretch_stiffness": 0.0, "bend_stiffness": 0.0,
                                "curvature_limit_stiffness": 0.0})
    packed = PackedAssembly.from_assembly(assembly)

    def entries(world):
        states = world.debug_contact_states()
        assert (states < CONTACT_USE_VERLET).all()
        return int(states.sum())

    world = DeviceWorld(packed, config.cell_list, config.max_step)
    world.run_batch(fast, 12)
    wide, positions = entries(world), world.download_positions()
    fresh = DeviceWorld(packed, config.cell_list, config.max_step)
    fresh.upload_positions(positions)
    fresh.run_batch(still, 1)
    narrow = entries(fresh)
    assert wide > 1.3 * narrow
    # New Verlet lists: the same width again.
    world.debug_rebuild()
    world.run_batch(still, 40)
    assert entries(world) > 1.3 * narrow
    # The lists have served 40 passes when a move that leaves the Verlet lists
    # (less than half the neighbor skin) ends them: narrow ones.
    world.upload_positions(positions + np.float32(0.15 * world.neighbor_skin))
    world.run_batch(still, 1)
    assert entries(world) < 1.05 * narrow
    world.close()
    fresh.close()
