"""The contact graph's edges, where a segment has few, many and very many.

graph_sort_kernel ranks a segment's incoming edges in registers, 32 and then
64 of them, and sorts longer runs in memory. With a neighbor skin of many
radii every Verlet pair is an edge, and segments of a bundle have from none
to far more than 64 before them: sources ascend, edge and twin name each
other, and the records moved with their edges (a twin's parameters are its
own, exchanged, and its offset the opposite).
"""

import numpy as np
import pytest

from tangle_b200.assembly import Cell, FiberAssembly, PackedAssembly
from tangle_b200.settings import CellListConfig

pytestmark = pytest.mark.gpu


def test_edges_are_sorted_and_keep_their_records(cuda_lib):
    from tangle_b200.device import DeviceWorld
    from tangle_b200.warmstart import ContactGraph

    rng = np.random.default_rng(5)
    assembly = FiberAssembly(Cell([8.0e-4] * 3, "xyz"))
    for k in range(90):
        spread = 4.0e-5 if k < 60 else 3.0e-4
        start = np.array([4.0e-4, 4.0e-4, 4.0e-4]) + rng.normal(scale=spread, size=3)
        direction = rng.normal(size=3)
        points = start + np.arange(4)[:, None] * 2.0e-5 * direction / np.linalg.norm(direction)
        assembly.add_fiber(points, radius=5.0e-6, min_bend_radius=5.0e-5)
    packed = PackedAssembly.from_assembly(assembly)
    world = DeviceWorld(packed, CellListConfig(neighbor_skin_scale=16.0, neighbor_capacity=512, max_list_bytes=1 << 28), 1.0e-6)
    graph = ContactGraph.from_world(world, 1.0e-3)
    counts, lists = world.debug_neighbor_lists()
    world.close()
    get = lambda t: t.cpu().numpy()
    src, dst, twin, s, t = (get(getattr(graph, name)) for name in ("src", "dst", "twin", "s", "t"))
    offsets, features = get(graph.offsets), get(graph.edge_features.float())
    wanted = {(a, int(b)) for a, entries in enumerate(lists) for b in entries}
    wanted |= {(b, a) for a, b in wanted}
    assert graph.E == len(wanted) and set(zip(dst.tolist(), src.tolist())) == wanted
    before = np.zeros(packed.segment_count, dtype=int)
    for segment in range(packed.segment_count):
        low, high = offsets[segment], offsets[segment + 1]
        assert (dst[low:high] == segment).all() and (np.diff(src[low:high]) > 0).all()
        before[segment] = (src[low:high] < segment).sum()
    for low, high in ((0, 0), (1, 1), (2, 32), (33, 64), (65, 400)):
        assert ((before >= low) & (before <= high)).any(), (low, high, before.max())
    edges = np.arange(graph.E)
    assert (twin[twin] == edges).all() and (src[twin] == dst).all() and (dst[twin] == src).all()
    assert (s[twin] == t).all() and (t[twin] == s).all()
    assert (features[twin][:, :3] == -features[:, :3]).all() and (features[twin][:, 3] == features[:, 3]).all()
    assert (features[twin][:, 4] == features[:, 5]).all()
    rounded = graph.s.bfloat16().float().cpu().numpy()
    assert (features[:, 4] == rounded).all()
