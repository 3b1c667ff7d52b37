"""Worlds of many short fibers: the update's default lanes, and its results.

From 72 fibers per SM, fibers of 3 to 32 vertices (24 in an arena) take four
lanes each by default (eight before); worlds of two-vertex fibers, which have nothing to
sweep, run a kernel without the sweeps. Positions and curvature maxima are
the oracle's bit for bit, in a periodic box and between walls, and an
arena's are those of its specimens alone.
"""

import numpy as np
import pytest

from tangle_b200.assembly import Cell, FiberAssembly, PackedAssembly
from tangle_b200.settings import CellListConfig, RelaxationConfig

pytestmark = pytest.mark.gpu

RADIUS = 5.0e-6
CELLS = CellListConfig(neighbor_capacity=96, max_list_bytes=1 << 30)


def short_fibers(count, vertices, periodic="xyz", seed=1):
    rng = np.random.default_rng(seed)
    side = (count * vertices * 4.0e-14) ** (1.0 / 3.0)
    assembly = FiberAssembly(Cell([side] * 3, periodic))
    for _ in range(count):
        steps = np.array([1.0, 0.2, 0.1]) + rng.normal(scale=0.5, size=(vertices - 1, 3))
        steps *= 4.0 * RADIUS / np.linalg.norm(steps, axis=1)[:, None]
        points = np.concatenate([np.zeros((1, 3)), np.cumsum(steps, axis=0)]) + rng.uniform(0.0, side, 3)
        for axis, name in enumerate("xyz"):
            if name not in periodic:
                points[:, axis] = np.clip(points[:, axis], RADIUS, side - RADIUS)
        assembly.add_fiber(points, radius=RADIUS, min_bend_radius=10.0 * RADIUS)
    return PackedAssembly.from_assembly(assembly)


def settings():
    return RelaxationConfig(penetration_tolerance=1.0e-8, force_full_iterations=True, max_step=5.0e-7, cell_list=CELLS)


@pytest.mark.parametrize("per_sm, vertices, lanes", [(16, 8, 32), (17, 8, 8), (72, 8, 8), (73, 8, 4), (73, 3, 4), (73, 2, 8),
                                                     (73, 32, 4), (73, 33, 8)])
def test_default_lanes(per_sm, vertices, lanes, cuda_lib):
    import torch

    from tangle_b200.device import DeviceWorld

    count = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    world = DeviceWorld(short_fibers(count, vertices), CELLS, 5.0e-7)
    assert world.launch_params()["lanes_per_fiber"] == lanes
    world.close()


@pytest.mark.parametrize("periodic", ["xyz", "xy"])
@pytest.mark.parametrize("count, vertices", [(1, 2), (2500, 2), (11000, 2), (11000, 3), (11000, 7)])
def test_short_fibers_match_the_oracle(count, vertices, periodic, cuda_lib):
    from oracle import OracleWorld
    from tangle_b200.device import DeviceWorld

    packed, config = short_fibers(count, vertices, periodic), settings()
    dev, orc = DeviceWorld(packed, CELLS, config.max_step), OracleWorld(packed, CELLS, config.max_step)
    for batch in (1, 4):
        got, want = dev.run_batch(config, batch), orc.run_batch(config, batch)
        assert (got.max_penetration, got.max_curvature_ratio) == (want.max_penetration, want.max_curvature_ratio)
        np.testing.assert_array_equal(dev.download_positions().view(np.uint32), orc.download_positions().view(np.uint32))
        np.testing.assert_array_equal(dev.wall_reactions().view(np.uint32), orc.wall_reactions().view(np.uint32))
    dev.close()
    orc.close()


@pytest.mark.parametrize("vertices, lanes", [(24, 4), (25, 8)])
def test_default_lanes_of_an_arena(vertices, lanes, cuda_lib):
    import torch

    from tangle_b200.device import DeviceWorld

    count = 73 * torch.cuda.get_device_properties(0).multi_processor_count // 4
    arena = DeviceWorld.arena([short_fibers(count + 1, vertices, seed=s) for s in range(4)], CELLS, 5.0e-7)
    assert arena.launch_params()["lanes_per_fiber"] == lanes
    arena.close()


def test_two_vertex_specimens_of_an_arena(cuda_lib):
    from tangle_b200.device import DeviceWorld

    packs, config = [short_fibers(900, 2, seed=s) for s in range(4)], settings()
    arena = DeviceWorld.arena(packs, CELLS, config.max_step)
    arena.run_batch(config, 5)
    for got, packed in zip(arena.specimen_positions(), packs):
        world = DeviceWorld(packed, CELLS, config.max_step)
        world.run_batch(config, 5)
        np.testing.assert_array_equal(got.view(np.uint32), world.download_positions().view(np.uint32))
        world.close()
    arena.close()
