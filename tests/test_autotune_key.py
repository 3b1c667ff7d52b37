"""A cached launch shape is only taken for the kernels and worlds it was found on.

The cache's key holds what decides the best shape: beside the sizes of the
grid and the lists, the kernels themselves (a digest of their sources), the
active fibers and the longest fiber. An entry of other kernels, or one whose
key lacks any of these, is searched anew.
"""

import json
from types import SimpleNamespace

import numpy as np
import pytest

from tangle_b200 import autotune as at
from tangle_b200.settings import RelaxationConfig

PARAMS = {"lanes_per_fiber": 8, "contact_blocks_per_sm": 1, "build_chunk": 3072, "contact_skin_fraction": 0.1,
          "update_warps_per_block": 4}


def world(searched, **other):
    values = dict(vertex_count=300, segment_count=290, cell_count=27, cell_dims=(3, 3, 3), neighbor_block=256,
                  fiber_count=10, longest_fiber=30, fiber_active=np.ones(10, dtype=np.uint32),
                  contact_list_info=lambda: {"block": 32, "skin": 1.0, "refreshes": 0},
                  set_launch_params=lambda params: None,
                  autotune_trials=lambda config, n: searched.append(n) or (PARAMS, {"trials": 1}))
    return SimpleNamespace(**{**values, **other})


@pytest.mark.parametrize("other", [{"longest_fiber": 31}, {"fiber_active": np.array([1] * 9 + [0], dtype=np.uint32)},
                                   {"fiber_count": 9, "fiber_active": np.ones(9, dtype=np.uint32)}], ids=list)
def test_other_fibers_are_searched(other, tmp_path):
    searched, path = [], str(tmp_path / "cache.json")
    run = lambda w: at.autotune(w, RelaxationConfig(), path=path, gpu="B200")["cached"]
    assert [run(world(searched)), run(world(searched))] == [False, True]
    assert [run(world(searched, **other)), run(world(searched, **other))] == [False, True]
    assert len(searched) == 2


def test_entries_of_other_kernels_are_searched(tmp_path, monkeypatch):
    searched, path = [], str(tmp_path / "cache.json")
    run = lambda: at.autotune(world(searched), RelaxationConfig(), path=path, gpu="B200")["cached"]
    assert not run()
    (key, entry), = at.load(path).items()
    before = {k: v for k, v in json.loads(key).items() if k not in ("kernels", "active_fibers", "longest_fiber")}
    at.store(tmp_path / "old.json", json.dumps(before, sort_keys=True), entry)
    path = str(tmp_path / "old.json")
    assert not run() and run()
    monkeypatch.setattr(at, "kernels", lambda: "others")
    assert not run() and run()


def test_the_digest_follows_the_sources(tmp_path, monkeypatch):
    from tangle_b200 import build

    source = tmp_path / "kernels.cu"
    source.write_text("a")
    monkeypatch.setattr(build, "SOURCES", [str(source)])
    monkeypatch.setattr(build, "HEADERS", [])
    first = at.kernels()
    source.write_text("b")
    assert at.kernels() != first
    source.unlink()  # installed without its sources: the library stands for them
    library = tmp_path / "lib.so"
    library.write_bytes(b"x")
    monkeypatch.setattr(build, "LIB", str(library))
    assert at.kernels() not in (first, "")


def test_worlds_know_their_fibers():
    from tangle_b200.device import fiber_lengths

    packed = SimpleNamespace(fiber_vertex_spans=np.array([0, 4, 4, 9, 13, 2], dtype=np.uint32))
    assert fiber_lengths([packed]) == (3, 9)
    assert fiber_lengths([packed, packed]) == (6, 9)
