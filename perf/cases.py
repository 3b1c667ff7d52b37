"""Performance cases: the calls a program that relaxes fiber assemblies makes.

Each case is a dict of plain values. `prepare` builds what such a program
holds before the call (the specimen from a seed, its resident world, pinned
host buffers, a network), `run` is one pass through the public entry points,
`work` what the pass cannot do without, and `exact` the same result in 64
bits for the cases that a plain NumPy restatement finishes in seconds.

Kinds:

* "relax": one `DeviceWorld` -- positions in, `run_batch`, positions and
  status out, the cadence of a driver that owns the positions between
  batches. Specimens: "fibers30" (the CPU-runnable cube's kind: straight
  fibers of 30 segments), "mid_size" (wavy 7 and 19 um fibers, periodic
  cube), "ply" (planar plies between z walls).
* "arena": the same on many specimens packed into one arena, each stopping
  at its own gate.
* "recipe": `Recipe.run` from fibers on the host to relaxed fibers.
* "infer": positions in, `warm_start` with the trained network (contact
  graph, network forward, residuals before and after), positions out.
* "train": one training step of that network on one specimen.
"""

from __future__ import annotations

import math
import os

import numpy as np
import torch

import tangle_b200 as tangle
from tangle_b200 import warmstart
from tangle_b200.device import DeviceWorld
from tangle_b200.generate import (SplitMix64, cpu_runnable_specimen, isotropic_direction, mid_size_specimen,
                                  ply_stack_specimen)
from tangle_b200.settings import RelaxationSettings

_TRAINED = os.path.join(os.path.dirname(tangle.__file__), "warmstart_net.npz")
_AGGREGATIONS = ("uniform_average", "penetration_weighted", "deepest_only")


def listed():
    return [
        # A driver that looks at the positions every few iterations (snapshots,
        # a live view): the smallest call, all launch latency.
        {"name": "small_4", "kind": "relax", "specimen": "fibers30", "fibers": 40, "iterations": 4},
        # The CPU-runnable configuration at the default batch of 128 iterations.
        {"name": "small_128", "kind": "relax", "specimen": "fibers30", "fibers": 40, "iterations": 128},
        # The first program of the README: a few fibers, one call.
        {"name": "recipe_small", "kind": "recipe", "fibers": 20, "segments": 8, "side": 400e-6},
        # A training specimen of the learned warm start: its trajectory over 64 iterations.
        {"name": "specimen_2k_64", "kind": "relax", "specimen": "mid_size", "fibers": 2000, "beta": 1.0 / 0.3,
         "iterations": 64},
        # The same size late in its relaxation, where a long run spends most of its iterations.
        {"name": "relaxed_2k_128", "kind": "relax", "specimen": "mid_size", "fibers": 2000, "beta": 1.0 / 0.3,
         "before": 768, "iterations": 128},
        # An odd size in the z-aligned orientation, with the weighted contact aggregation and pinned ends.
        {"name": "aligned_4999_50", "kind": "relax", "specimen": "mid_size", "fibers": 4999, "beta": 0.3,
         "iterations": 50, "aggregation": 1, "pinned": True},
        # The mid-size benchmark configuration, one default batch from the initial packing: the largest call.
        {"name": "mid_size_128", "kind": "relax", "specimen": "mid_size", "fibers": 20000, "beta": 1.0 / 0.3,
         "iterations": 128},
        # Batched specimens of uneven sizes, gates on.
        {"name": "arena_48", "kind": "arena", "specimens": 48, "most": 5000, "iterations": 64},
        # Two plies between walls (wall reactions kept), the deposition configuration's fibers.
        {"name": "plies_2", "kind": "relax", "specimen": "ply", "plies": 2, "side": 1.0e-3, "length": 1.0e-3,
         "iterations": 64},
        # Fibers of several hundred segments.
        {"name": "ply_long_fibers", "kind": "relax", "specimen": "ply", "plies": 1, "side": 1.2e-3,
         "length": 2.0e-3, "iterations": 32},
        # The learned warm start's one proposal on a specimen of the training size.
        {"name": "warm_infer_2k", "kind": "infer", "fibers": 2000},
        # One step of its training.
        {"name": "warm_train_1k", "kind": "train", "fibers": 1000},
    ]


def _log_uniform(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def draw(rng):
    """A case of the same ranges: 16 to 20,000 fibers, 1 to 128 iterations,
    either orientation, fresh or partly relaxed, every aggregation and motion
    model, walls, arenas, recipes and the warm start."""
    kind = rng.choice(["relax"] * 8 + ["ply", "ply", "arena", "arena", "recipe", "infer", "train"])
    if kind == "arena":
        return {"kind": "arena", "specimens": rng.randint(3, 40), "most": int(_log_uniform(rng, 60, 3000)),
                "iterations": rng.randint(8, 64)}
    if kind == "recipe":
        return {"kind": "recipe", "fibers": rng.randint(4, 40), "segments": rng.randint(4, 24),
                "side": rng.uniform(300e-6, 600e-6)}
    if kind in ("infer", "train"):
        return {"kind": kind, "fibers": int(_log_uniform(rng, 100, 2000 if kind == "infer" else 1000))}
    if kind == "ply":
        return {"kind": "relax", "specimen": "ply", "plies": rng.randint(1, 3), "side": rng.uniform(0.3e-3, 1.2e-3),
                "length": rng.uniform(0.3e-3, 2.0e-3), "iterations": rng.randint(2, 64)}
    iterations = int(round(_log_uniform(rng, 1, 128)))
    if rng.random() < 0.3:
        return {"kind": "relax", "specimen": "fibers30", "fibers": rng.randint(10, 120), "iterations": iterations,
                "aggregation": rng.randint(0, 2), "rigid": rng.random() < 0.3}
    return {"kind": "relax", "specimen": "mid_size", "fibers": int(_log_uniform(rng, 16, 20000)),
            "beta": rng.choice([1.0 / 0.3, 0.3, 1.0]), "before": rng.choice([0, 0, 0, rng.randint(64, 512)]),
            "iterations": iterations, "aggregation": rng.choice([0, 0, 0, 1, 2]), "pinned": rng.random() < 0.2,
            "rigid": rng.random() < 0.15}


# ---------------------------------------------------------------- specimens


def _fibers30(count, seed):
    """Straight 10 um fibers, 300 um long as 30 segments, at the CPU-runnable
    configuration's density."""
    if count == 40:
        return cpu_runnable_specimen(seed=seed)
    side = 300.0e-6 * (count / 40.0) ** (1.0 / 3.0)
    assembly = tangle.FiberAssembly(tangle.Cell([side] * 3, "xyz"))
    random = SplitMix64(seed)
    steps = np.arange(31, dtype=np.float64) * 10.0e-6
    for _ in range(count):
        start = np.array([side * random.unit() for _ in range(3)])
        points = start + steps[:, None] * np.array(isotropic_direction(random))
        assembly.add_fiber(points, points, radius=5.0e-6, min_bend_radius=50.0e-6)
    return assembly


def _arena_sizes(case):
    """The fiber lengths and volume fraction of each specimen of an arena,
    from the case alone (another seed places other fibers in specimens of the
    same sizes): fiber count log-uniform from 40 (fewer in arenas of smaller
    specimens), length 0.3 to 1 mm, 5 to 25 % fiber volume."""
    sizes = np.random.RandomState(case["specimens"] + 64 * case["most"])
    least = min(40.0, 0.5 * case["most"])
    return [(sizes.uniform(0.3e-3, 1.0e-3, int(round(math.exp(sizes.uniform(math.log(least), math.log(case["most"])))))),
             sizes.uniform(0.05, 0.25)) for _ in range(case["specimens"])]


def _arena(case, seed):
    """Straight isotropic 10 um fibers in periodic cubes, segments of two
    diameters, curvature limit 1 / (5 d)."""
    d = 10.0e-6
    places = np.random.RandomState(seed % (1 << 32))
    out = []
    for lengths, fraction in _arena_sizes(case):
        side = (math.pi * (0.5 * d) ** 2 * lengths.sum() / fraction) ** (1.0 / 3.0)
        side = max(side, 1.05 * lengths.max() / 2.0)
        assembly = tangle.FiberAssembly(tangle.Cell([side] * 3, "xyz"))
        directions = places.normal(size=(lengths.size, 3))
        directions /= np.linalg.norm(directions, axis=1)[:, None]
        for length, start, direction in zip(lengths, places.uniform(0.0, side, (lengths.size, 3)), directions):
            steps = np.linspace(0.0, length, int(round(length / (2.0 * d))) + 1)
            points = start + steps[:, None] * direction
            assembly.add_fiber(points, points, radius=0.5 * d, min_bend_radius=5.0 * d)
        out.append(assembly)
    return out


def _assembly(case, seed):
    specimen = case.get("specimen", "mid_size")
    if specimen == "fibers30":
        return _fibers30(case["fibers"], seed)
    if specimen == "ply":
        return ply_stack_specimen(plies=case["plies"], side=case["side"], fiber_length=case["length"], seed=seed)
    scale = (case["fibers"] / 20000.0) ** (1.0 / 3.0)
    return mid_size_specimen(scale=scale, seed=seed, beta=case.get("beta", 1.0 / 0.3))


def _config(case, diameter):
    return RelaxationSettings(
        penetration_tolerance=1.0e-3 * diameter, neighbor_capacity=256, max_list_bytes=8 << 30,
        contact_aggregation=_AGGREGATIONS[case.get("aggregation", 0)], pin_fiber_ends=bool(case.get("pinned", False)),
        motion_model="rigid_translation" if case.get("rigid", False) else "flexible",
        force_full_iterations=case["kind"] == "relax", max_iterations=100000).to_config(diameter)


def _pinned_host(values):
    out = torch.empty(values.size, dtype=torch.float32, pin_memory=True).numpy()
    out[:] = values
    return out


def _population(case, seed):
    material = tangle.Material("fiber", diameter=10e-6)
    return tangle.FiberPopulation(material=material, count=case["fibers"], segments_per_fiber=case["segments"],
                                  seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "recipe":
        recipe = tangle.Recipe(tangle.Cell([case["side"]] * 3, periodic="xyz"))
        recipe.insert(_population(case, seed))
        return {"case": case, "recipe": recipe, "settings": RelaxationSettings(backend="cuda")}
    if kind == "arena":
        assemblies = _arena(case, seed)
        diameter = min(a.smallest_diameter() for a in assemblies)
        config = _config(case, diameter)
        packs = [tangle.PackedAssembly.from_assembly(a) for a in assemblies]
        world = DeviceWorld.arena(packs, config.cell_list, config.max_step)
        start = np.concatenate([p.positions for p in packs])
        return {"case": case, "world": world, "config": config, "start": _pinned_host(start),
                "out": _pinned_host(start)}
    assembly = _assembly(case, seed)
    config = _config(case, assembly.smallest_diameter())
    packed = tangle.PackedAssembly.from_assembly(assembly, bool(case.get("pinned", False)))
    world = DeviceWorld(packed, config.cell_list, config.max_step)
    if kind == "train":
        sample = warmstart.make_sample(world, config, 16)
        return {"case": case, "sample": sample, "net": warmstart.WarmStartNet(seed)}
    start = packed.positions
    if case.get("before", 0):
        world.run_batch(config, case["before"])
        start = world.download_positions()
    state = {"case": case, "world": world, "config": config, "start": _pinned_host(start), "out": _pinned_host(start)}
    if kind == "infer":
        state["net"] = warmstart.WarmStartNet.load(_TRAINED)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "recipe":
        result = state["recipe"].run(state["settings"])
        return {"positions": np.concatenate([f.placed for f in result.assembly.fibers]).astype(np.float32),
                "iterations": int(result.iterations)}
    if kind == "train":
        net = state["net"]
        loss = net.train_step(state["sample"].graph, state["sample"].target, 1.0e-3)
        layers = net.layers()
        return {"loss": loss, "weight_gradients": [layer.gw for layer in layers],
                "bias_gradients": [layer.gb for layer in layers], "weights": [layer.w for layer in layers]}
    world, config = state["world"], state["config"]
    world.upload_positions(state["start"])
    if kind == "infer":
        report = warmstart.warm_start(world, state["net"], config)
        return {"positions": world.download_positions(state["out"]),
                "residuals": [report.residual_before, report.residual_after], "accepted": bool(report.accepted),
                "edges": int(report.edges)}
    status = world.run_batch(config, state["case"]["iterations"])
    out = {"positions": world.download_positions(state["out"]),
           "status": [status.max_penetration, status.max_displacement, status.max_curvature_ratio],
           "iterations": int(status.batch_iterations)}
    if kind == "arena":
        out["specimen_iterations"] = np.array([s.batch_iterations for s in world.specimen_statuses(config)])
    return out


# ---------------------------------------------------------------- work


def _nodes(case):
    """Vertices of a case's specimens, from the sizes alone."""
    kind, specimen = case["kind"], case.get("specimen", "mid_size")
    if kind == "recipe":
        return case["fibers"] * (case["segments"] + 1)
    if kind == "arena":
        return sum(float(np.round(lengths / 20.0e-6).sum() + lengths.size) for lengths, _ in _arena_sizes(case))
    if specimen == "fibers30":
        return case["fibers"] * 31
    if specimen == "ply":
        nodes = 0.0
        for d in (7.0e-6, 19.0e-6):
            volume = 0.5 * 0.15 * case["side"] ** 2 * 0.1e-3
            count = volume / (math.pi * 0.25 * d * d * case["length"])
            nodes += case["plies"] * count * (case["length"] / (0.8 * d) + 1.0)
        return nodes
    return case["fibers"] * (0.88 * 108 + 0.12 * 40)


def work(case):
    """One iteration reads and writes the state once (144 bytes per node with
    the constraint data) and does about 500 operations per node: the two
    constraint passes, a curvature test and four candidate contacts. The warm
    start: its layers' products over the nodes and about 20 edges per node."""
    nodes = _nodes(case)
    if case["kind"] in ("infer", "train"):
        edges = 20.0 * nodes
        per_node = 16 * 64 + 64 * 64 + 3 * (192 * 64 + 64 * 64) + 64 * 64 + 64 * 16
        flops = 2.0 * (nodes * per_node + edges * 3 * (80 * 64 + 64 * 64))
        passes = 1.0 if case["kind"] == "infer" else 3.0
        return {"bytes": passes * (nodes * 96.0 + edges * 52.0), "flops": passes * flops}
    iterations = case.get("iterations", 32)
    return {"bytes": 24.0 * nodes + iterations * 144.0 * nodes, "flops": iterations * 500.0 * nodes}


# ---------------------------------------------------------------- 64 bits

_EXACT_SWEEPS = 60_000       # vertices x iterations, and
_EXACT_PAIRS = 160_000_000   # vertices^2 x iterations, that the NumPy restatement finishes in seconds


def exact(case, seed):
    """The relaxation in 64 bits, in plain NumPy: every pair of segments each
    iteration (no lists), then the constraint passes, the contact step and
    the serial curvature sweeps."""
    if case["kind"] != "relax" or case.get("before", 0) or case.get("rigid", False):
        return None
    nodes = _nodes(case)
    if nodes * case["iterations"] > _EXACT_SWEEPS or nodes * nodes * case["iterations"] > _EXACT_PAIRS:
        return None
    assembly = _assembly(case, seed)
    config = _config(case, assembly.smallest_diameter())
    positions, penetration = _relax64(_Fibers64(assembly, bool(case.get("pinned", False))), config,
                                      case["iterations"])
    return {"positions": positions.reshape(-1), "status": [penetration, None, None], "iterations": None}


class _Fibers64:
    """The arrays of an assembly, positions rounded to f32 as the solver gets them."""

    def __init__(self, assembly, pinned_ends):
        f32 = np.float32
        self.counts = np.array([f.placed.shape[0] for f in assembly.fibers])
        self.first = np.concatenate([[0], np.cumsum(self.counts)[:-1]])
        self.x = np.concatenate([f.placed for f in assembly.fibers]).astype(f32).astype(np.float64)
        rest = np.concatenate([f.intrinsic for f in assembly.fibers])
        rest32 = rest.astype(f32).astype(np.float64)
        V = self.x.shape[0]
        fiber = np.repeat(np.arange(len(self.counts)), self.counts)
        local = np.arange(V) - self.first[fiber]
        n = self.counts[fiber]
        self.a = np.nonzero(local < n - 1)[0]  # first vertex of every segment
        self.segment_fiber = fiber[self.a]
        radii = np.array([f32(f.radius) for f in assembly.fibers], dtype=np.float64)
        self.radius = radii[self.segment_fiber]
        self.extent = radii[fiber][:, None]
        self.rest = np.linalg.norm(rest[self.a + 1] - rest[self.a], axis=1).astype(f32).astype(np.float64)
        self.second = np.nonzero(local < n - 2)[0]  # first vertex of every second-neighbor pair
        self.chord = np.linalg.norm(rest32[self.second + 2] - rest32[self.second], axis=1)
        length = np.linalg.norm(rest32[self.a + 1] - rest32[self.a], axis=1)
        arc = np.zeros(V)
        for f0, c in zip(self.first, self.counts):
            s0 = np.searchsorted(self.a, f0)
            arc[f0 + 1: f0 + c] = np.cumsum(length[s0: s0 + c - 1])
        self.arc0, self.arc1 = arc[self.a], arc[self.a + 1]
        limits = np.array([0.0 if f.min_bend_radius is None else f32(1.0 / f.min_bend_radius)
                           for f in assembly.fibers], dtype=np.float64)
        self.limit = np.where((local > 0) & (local < n - 1), limits[fiber], 0.0)
        self.free = np.ones(V, dtype=bool)
        if pinned_ends:
            self.free[self.first] = False
            self.free[self.first + self.counts - 1] = False
        cell = assembly.cell
        self.periodic = np.array(cell.periodic)
        lower = np.array(cell.origin, dtype=np.float64)
        self.lower = lower.astype(f32).astype(np.float64)
        self.upper = (lower + np.array(cell.lengths)).astype(f32).astype(np.float64)

    def clamp(self, x, extent):
        lo = np.where(self.periodic, -np.inf, self.lower + extent)
        hi = np.where(self.periodic, np.inf, self.upper - extent)
        return np.minimum(np.maximum(x, lo), hi)


def _meeting_normals64(d1, d2, flipped):
    """A normal for segments whose axes meet: d1 x d2, or for short products a
    vector across d1's smallest component, its largest component positive as
    seen from the lower segment."""
    n = np.cross(d1, d2)
    short = np.linalg.norm(n, axis=1) <= 1.0e-7
    ax, ay, az = np.abs(d1).T
    zero = np.zeros_like(ax)
    x_least = ((ax <= ay) & (ax <= az))[:, None]
    y_least = (ay <= az)[:, None]
    across = np.where(x_least, np.stack([zero, d1[:, 2], -d1[:, 1]], axis=1),
                      np.where(y_least, np.stack([-d1[:, 2], zero, d1[:, 0]], axis=1),
                               np.stack([d1[:, 1], -d1[:, 0], zero], axis=1)))
    n = np.where(short[:, None], across, n)
    length = np.linalg.norm(n, axis=1)
    n = np.where((length > 1.0e-7)[:, None], n / np.maximum(length, 1.0e-30)[:, None], np.array([1.0, 0.0, 0.0]))
    dominant = np.take_along_axis(n, np.abs(n).argmax(axis=1)[:, None], axis=1) if n.size else n[:, :1]
    return n * np.where(dominant < 0.0, -1.0, 1.0) * np.where(flipped, -1.0, 1.0)[:, None]


def _contacts64(f, x, config):
    """Per segment: the corrections of its two ends, and the deepest penetration of all."""
    p, q = x[f.a], x[f.a + 1]
    mid, half = 0.5 * (p + q), 0.5 * np.linalg.norm(q - p, axis=1)
    S = f.a.size
    box = f.upper - f.lower
    first, second = [], []
    for i0 in range(0, S, 512):  # the pairs whose bounding spheres meet
        delta = mid[None, :, :] - mid[i0: i0 + 512, None, :]
        delta -= np.where(f.periodic, np.round(delta / box) * box, 0.0)
        reach = (half + f.radius)[None, :] + (half + f.radius)[i0: i0 + 512, None]
        i, j = np.nonzero((delta * delta).sum(axis=2) <= reach * reach)
        first.append(i + i0)
        second.append(j)
    i, j = np.concatenate(first), np.concatenate(second)
    gap = np.maximum(f.arc0[j] - f.arc1[i], f.arc0[i] - f.arc1[j])
    own = (f.segment_fiber[i] == f.segment_fiber[j]) & (gap < f.radius[i] + f.radius[j])
    i, j = i[~own], j[~own]
    shift = np.where(f.periodic, np.round((mid[j] - mid[i]) / box) * box, 0.0)
    p1, p2 = p[i], p[j] - shift
    d1, d2 = q[i] - p[i], q[j] - p[j]
    r = p1 - p2
    dot = lambda u, v: (u * v).sum(axis=1)  # noqa: E731
    a, e, ff, c, b = dot(d1, d1), dot(d2, d2), dot(d2, r), dot(d1, r), dot(d1, d2)
    den = a * e - b * b
    parallel = np.abs(den) <= 1.0e-6 * a * e

    def ends(s):
        t = (b * s + ff) / e
        s = np.where(t < 0.0, np.clip(-c / a, 0.0, 1.0), np.where(t > 1.0, np.clip((b - c) / a, 0.0, 1.0), s))
        return s, np.clip(t, 0.0, 1.0)

    s, t = ends(np.where(parallel, 0.0, np.clip((b * ff - c * e) / np.where(parallel, 1.0, den), 0.0, 1.0)))
    s1, t1 = ends(np.ones_like(s))
    near = lambda s, t: dot(*(2 * [r + d1 * s[:, None] - d2 * t[:, None]]))  # noqa: E731
    other = parallel & (near(s1, t1) < near(s, t))
    s, t = np.where(other, s1, s), np.where(other, t1, t)
    delta = (p2 + d2 * t[:, None]) - (p1 + d1 * s[:, None])
    distance = np.sqrt(dot(delta, delta))
    penetration = f.radius[i] + f.radius[j] - distance
    hit = penetration > 0.0
    i, j, s, t, d1, d2, delta, distance, penetration = (
        v[hit] for v in (i, j, s, t, d1, d2, delta, distance, penetration))
    normal = delta / np.maximum(distance, 1.0e-30)[:, None]
    meet = distance <= 1.0e-7  # the axes meet: no direction between the closest points
    normal[meet] = _meeting_normals64(d1[meet], d2[meet], (i > j)[meet])
    weight = (1.0 - s) ** 2 + s ** 2 + (1.0 - t) ** 2 + t ** 2
    magnitude = -config.correction_fraction * penetration / weight
    push = normal * magnitude[:, None]
    deepest = float(penetration.max()) if penetration.size else 0.0
    out = np.zeros((2, S, 3))
    if config.contact_aggregation == 2:
        order = np.argsort(penetration, kind="stable")
        out[0, i[order]] = (push * (1.0 - s)[:, None])[order]
        out[1, i[order]] = (push * s[:, None])[order]
        return out, deepest
    share = penetration if config.contact_aggregation == 1 else np.ones_like(penetration)
    total = np.zeros(S)
    np.add.at(total, i, share)
    np.add.at(out[0], i, push * ((1.0 - s) * share)[:, None])
    np.add.at(out[1], i, push * (s * share)[:, None])
    some = total > 1.0e-20
    out[:, some] /= total[some][None, :, None]
    return out, deepest


def _curvature64(f, x, config):
    """Serial sweeps along each fiber, all fibers side by side."""
    most = int(f.counts.max())
    for _ in range(config.curvature_cleanup_sweeps):
        for offsets in (range(most - 2), range(most - 3, -1, -1)):
            for k in offsets:
                has = f.counts > k + 2
                i0 = f.first[has] + k
                i1, i2 = i0 + 1, i0 + 2
                limit = f.limit[i1] * (1.0 - config.curvature_limit_safety_margin)
                u, v = x[i1] - x[i0], x[i2] - x[i1]
                lu, lv = np.linalg.norm(u, axis=1), np.linalg.norm(v, axis=1)
                ok = (limit > 0.0) & (lu > 1.0e-7) & (lv > 1.0e-7)
                half = 0.25 * limit * (lu + lv)
                ok &= half < 1.0
                if not ok.any():
                    continue
                un, vn = u / np.maximum(lu, 1e-30)[:, None], v / np.maximum(lv, 1e-30)[:, None]
                cosine = np.clip((un * vn).sum(axis=1), -1.0, 1.0)
                least = 1.0 - 2.0 * np.minimum(half, 1.0) ** 2
                violation = least - cosine
                sine = np.sqrt(np.maximum(1.0 - cosine * cosine, 0.0))
                violation = np.where((violation > 0.0) & (sine > 1.0e-3),
                                     (np.arccos(cosine) - np.arccos(least)) * sine, violation)
                ok &= violation > 0.0
                if not ok.any():
                    continue
                gu = (vn - cosine[:, None] * un) / np.maximum(lu, 1e-30)[:, None]
                gv = (un - cosine[:, None] * vn) / np.maximum(lv, 1e-30)[:, None]
                gc = gu - gv
                w0, w1, w2 = (f.free[i].astype(np.float64) for i in (i0, i1, i2))
                den = w0 * (gu * gu).sum(axis=1) + w1 * (gc * gc).sum(axis=1) + w2 * (gv * gv).sum(axis=1)
                ok &= den > 1.0e-12
                scale = np.where(ok, config.curvature_limit_stiffness * violation / np.where(ok, den, 1.0), 0.0)
                extent = f.extent[i1]
                for i, w, g in ((i0, w0, -gu), (i1, w1, gc), (i2, w2, gv)):
                    act = ok & (w > 0.0)
                    x[i[act]] = f.clamp(x[i[act]] + scale[act, None] * g[act], extent[act])


def _relax64(f, config, iterations):
    x = f.x.copy()
    for _ in range(iterations):
        contact, _ = _contacts64(f, x, config)
        for _ in range(config.constraint_iterations):
            move = np.zeros_like(x)
            for i, j, rest, stiffness in ((f.a, f.a + 1, f.rest, config.stretch_stiffness),
                                          (f.second, f.second + 2, f.chord, config.bend_stiffness)):
                d = x[j] - x[i]
                length = np.linalg.norm(d, axis=1)
                pull = d * (np.where(length > 1.0e-7, 0.5 * stiffness * (length - rest) /
                                     np.maximum(length, 1.0e-30), 0.0))[:, None]
                move[i] += pull
                move[j] -= pull
            x[f.free] = f.clamp(x + move, f.extent)[f.free]
        step = np.zeros_like(x)
        step[f.a] += contact[0]
        step[f.a + 1] += contact[1]
        length = np.linalg.norm(step, axis=1)
        step *= np.where(length > config.max_step, config.max_step / np.maximum(length, 1.0e-30), 1.0)[:, None]
        x[f.free] = f.clamp(x + step, f.extent)[f.free]
        _curvature64(f, x, config)
    return x, _contacts64(f, x, config)[1]
