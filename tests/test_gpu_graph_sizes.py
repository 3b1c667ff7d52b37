"""The message kernels' results do not depend on how a graph's size splits them.

A warp takes one vertex of a small graph and a run of eight of a large one,
and one to 32 edges.
Copies of one graph side by side, in numbers around each change of the split
and so that the copies start anywhere in a run, give each copy the bits that
the graph gives alone.
"""

import ctypes

import pytest

pytestmark = pytest.mark.gpu


def copies_of(graph, n):
    """n copies of a graph's tensors as one graph."""
    import torch

    from tangle_b200 import warmstart

    out = warmstart.ContactGraph.__new__(warmstart.ContactGraph)
    out.V, out.S, out.E = n * graph.V, n * graph.S, n * graph.E
    k = torch.arange(n, device="cuda", dtype=torch.int32)[:, None]

    def shifted(values, by):
        return torch.where(values >= 0, values + k * by, values).reshape(-1).contiguous()

    out.seg_v0 = shifted(graph.seg_v0, graph.V)
    vertices, segments = graph.links.view(-1, 4)[:, :2].reshape(-1), graph.links.view(-1, 4)[:, 2:].reshape(-1)
    out.links = torch.cat([shifted(vertices, graph.V).view(-1, 2), shifted(segments, graph.S).view(-1, 2)], 1).contiguous()
    out.offsets = torch.cat([shifted(graph.offsets[:-1], graph.E), torch.tensor([out.E], device="cuda", dtype=torch.int32)])
    out.dst, out.src, out.twin = (shifted(getattr(graph, name)[:graph.E], by)
                                  for name, by in (("dst", graph.S), ("src", graph.S), ("twin", graph.E)))
    out.s, out.t = (getattr(graph, name)[:graph.E].repeat(n) for name in ("s", "t"))
    return out


def inputs(graph, h, m):
    import torch

    from tangle_b200 import warmstart
    from tangle_b200.warmstart import _check, _p, _stream

    lib, gs = warmstart._lib(), graph.struct()
    x = torch.zeros(graph.V, 192, device="cuda", dtype=torch.bfloat16)
    xe = torch.zeros(graph.E, 80, device="cuda", dtype=torch.bfloat16)
    _check(lib.tgl_mp_node_inputs(ctypes.byref(gs), _p(h), _p(m), _p(x), _stream()))
    _check(lib.tgl_mp_edge_inputs(ctypes.byref(gs), _p(h), _p(xe), 80, _stream()))
    return x, xe


@pytest.fixture(scope="module")
def small(cuda_lib):
    import torch

    from tangle_b200 import warmstart
    from tangle_b200.assembly import PackedAssembly
    from tangle_b200.device import DeviceWorld
    from tangle_b200.generate import cpu_runnable_specimen

    assembly = cpu_runnable_specimen(seed=2)
    config = warmstart.relaxation_config(assembly)
    world = DeviceWorld(PackedAssembly.from_assembly(assembly), config.cell_list, config.max_step)
    graph = warmstart.ContactGraph.from_world(world, warmstart.graph_cutoff(world))
    world.close()
    gen = torch.Generator(device="cuda").manual_seed(3)
    h = torch.randn(graph.V, 64, device="cuda", generator=gen)
    m = torch.randn(graph.E, 64, device="cuda", generator=gen)
    return graph, h, m


@pytest.mark.parametrize("vertices", [1, 2 * 1240, 5 * 1240, 20_000, 148 * 1024, 148 * 1024 + 1240, 400_000])
def test_copies_of_a_graph_get_its_bits(vertices, small):
    import torch

    graph, h, m = small
    assert graph.V == 1240 and graph.E > 4000
    want, want_e = inputs(graph, h, m)
    n = max(vertices // graph.V, 1)
    x, xe = inputs(copies_of(graph, n), h.repeat(n, 1), m.repeat(n, 1))
    assert torch.equal(x.view(n, graph.V, 192).view(torch.int16), want.view(torch.int16).expand(n, -1, -1))
    assert torch.equal(xe.view(n, graph.E, 80).view(torch.int16), want_e.view(torch.int16).expand(n, -1, -1))
