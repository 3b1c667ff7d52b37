"""Launch shapes applied to an arena refresh every specimen's contact lists.

The lists' single-image bound is that of the skin in force, so lists made
with another skin must not outlive it: as for a single world, the next batch
makes them anew. Vertices that barely move keep every other cause of a
refresh away; lists of a wide skin, then of a narrow one, are those of an
arena that had the narrow skin throughout.
"""

import numpy as np
import pytest

from tangle_b200.assembly import PackedAssembly
from tangle_b200.generate import batched_specimens
from tangle_b200.settings import RelaxationConfig, RelaxationSettings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide, narrow", [(0.5, 0.02), (0.25, 0.1)])
def test_specimens_refresh_their_lists_after_new_launch_shapes(wide, narrow, cuda_lib):
    from tangle_b200.device import DeviceWorld

    packs = [PackedAssembly.from_assembly(a) for a in batched_specimens(count=4, seed=3, max_fibers=200)]
    config = RelaxationSettings(penetration_tolerance=1.0e-8, neighbor_capacity=256,
                                max_list_bytes=1 << 30).to_config(7.0e-6)
    still = RelaxationConfig(**{**config.__dict__, "force_full_iterations": True, "max_step": 1.0e-13,
                                "stretch_stiffness": 0.0, "bend_stiffness": 0.0, "curvature_limit_stiffness": 0.0})
    states = []
    for fractions in ((wide, narrow), (narrow, narrow)):
        arena = DeviceWorld.arena(packs, config.cell_list, config.max_step)
        for fraction in fractions:
            arena.set_launch_params(dict(arena.launch_params(), contact_skin_fraction=fraction))
            arena.run_batch(still, 2)
        states.append(arena.debug_contact_states())
        arena.close()
    np.testing.assert_array_equal(states[0], states[1])
