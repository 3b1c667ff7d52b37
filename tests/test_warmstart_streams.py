"""Contact graphs are filled after the kernels that last used their memory.

`ContactGraph.from_world` allocates its tensors on torch's current stream,
whose caching allocator hands out memory that kernels already given to that
stream may still use, and fills them on the world's own non-blocking stream.
The fill has to wait for torch's stream: here in the order of the calls (on
the CPU, with fakes of both streams and of the library), and on the GPU with
kernels in flight over the very memory that the new graph is given.
"""

import numpy as np
import pytest

from tangle_b200 import warmstart

FIELDS = ("seg_v0", "links", "offsets", "dst", "src", "twin", "s", "t", "node_features", "edge_features")


def test_the_fill_waits_for_torchs_stream(monkeypatch):
    import torch

    calls = []

    class Stream:
        def __init__(self, handle, device=None):
            self.handle = handle

        def wait_stream(self, other):
            calls.append(("wait", self.handle, other))

    class Library:
        def tgl_warmstart_graph_count(self, handle, cutoff, edges):
            edges._obj.value = 3
            return 0

        def tgl_warmstart_graph_fill(self, handle, out):
            calls.append(("fill",))
            return 0

    class World:
        _handle, vertex_count, segment_count, stream_handle = None, 4, 3, 77

    allocate = warmstart.ContactGraph.__init__

    def on_the_host(self, V, S, E, device):
        calls.append(("allocate",))
        allocate(self, V, S, E, torch.device("cpu"))

    monkeypatch.setattr(warmstart, "_lib", Library)
    monkeypatch.setattr(warmstart.ContactGraph, "__init__", on_the_host)
    monkeypatch.setattr(torch.cuda, "ExternalStream", Stream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: "torch's")
    graph = warmstart.ContactGraph.from_world(World(), 1.0e-6)
    assert (graph.V, graph.S, graph.E) == (4, 3, 3)
    assert calls == [("allocate",), ("wait", 77, "torch's"), ("fill",)]


@pytest.mark.gpu
def test_a_graph_over_memory_in_use_is_the_quiet_one(cuda_lib):
    import torch

    from tangle_b200.assembly import PackedAssembly
    from tangle_b200.device import DeviceWorld
    from tangle_b200.generate import mid_size_specimen

    assembly = mid_size_specimen(scale=0.15, seed=6)
    config = warmstart.relaxation_config(assembly)
    world = DeviceWorld(PackedAssembly.from_assembly(assembly), config.cell_list, config.max_step)
    cutoff = warmstart.graph_cutoff(world)
    torch.cuda.synchronize()
    quiet = warmstart.ContactGraph.from_world(world, cutoff)
    want = {name: getattr(quiet, name).cpu() for name in FIELDS}
    del quiet
    busy = torch.ones(8192, 8192, device="cuda", dtype=torch.bfloat16)
    out = torch.empty_like(busy)
    torch.cuda.synchronize()
    for _ in range(100):
        torch.mm(busy, busy, out=out)
    again = [torch.empty(want[name].shape, dtype=want[name].dtype, device="cuda") for name in FIELDS]
    for buffer in again:
        buffer.fill_(1)
    places = {buffer.data_ptr() for buffer in again}
    del again, buffer
    graph = warmstart.ContactGraph.from_world(world, cutoff)
    assert places & {getattr(graph, name).data_ptr() for name in FIELDS}
    torch.cuda.synchronize()
    for name in FIELDS:
        np.testing.assert_array_equal(getattr(graph, name).cpu().view(torch.uint8).numpy(),
                                      want[name].view(torch.uint8).numpy(), err_msg=name)
    world.close()
