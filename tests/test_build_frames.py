"""The Verlet build's sphere test, in the home cell's frame, passes every pair
the exact test accepts.

rb_build_kernel (tangle_b200/csrc/kernels.cu) stages each candidate's centre
wrapped in its own cell's frame and moved by the stencil offset, its radius
times 1.0002 plus 4e-6 of its coordinates, and compares with the home's
centre in its cell's frame; with three cells on an axis the separation is
wrapped once more. This restates it in f32, operation for operation, with the
cells that proxy_cell gives the midpoints, against the exact test, on the
pairs of test_build_prefilter: 0.9-1.05 of the interaction distance, nearly
parallel axes, and end to end at the interaction distance, where the sphere
bound is tight; here also midpoints on cell faces, three to nine cells per
axis, walls, and segments unwrapped by up to forty boxes.
"""

import numpy as np
import pytest

from test_build_prefilter import half_length, roundf
from test_contact_filters import as_f32, distance, dot, unit

f32 = np.float32
SKIN = f32(2.0) * f32(9.5e-6)
CELL_SIZE = 76.0e-6  # four largest radii, two radii and the skin


def fma(a, b, c):
    """RN(a b + c) of f32 values: the product is exact in f64."""
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(f32)


def exact_build_test(p1, q1, r1, p2, q2, r2, length, periodic):
    image = (f32(0.5) * (((p2 + q2).astype(f32) - p1).astype(f32) - q1).astype(f32)).astype(f32)
    shift = (roundf((image / length).astype(f32)) * length * periodic).astype(f32)
    s2, t2 = (p2 - shift).astype(f32), (q2 - shift).astype(f32)
    d1, d2 = (q1 - p1).astype(f32), (t2 - s2).astype(f32)
    interaction = (((r1 + r2).astype(f32) + SKIN).astype(f32) * f32(1.0001)).astype(f32)
    m = (f32(0.5) * (((s2 + t2).astype(f32) - p1).astype(f32) - q1).astype(f32)).astype(f32)
    other_half = np.where(np.any(shift != 0.0, axis=1), (f32(0.5) * np.sqrt(dot(d2, d2))).astype(f32), half_length(p2, q2))
    reach = ((half_length(p1, q1) + other_half).astype(f32) + interaction).astype(f32)
    return (dot(m, m) <= (reach * reach).astype(f32)) & (distance(p1, d1, s2, d2, False) <= interaction)


def cells_of(p, q, lower, width, cells, periodic):
    middle = (f32(0.5) * (p + q).astype(f32)).astype(f32)
    raw = np.floor(((middle - lower).astype(f32) / width).astype(f32)).astype(np.int64)
    return np.where(periodic, raw % cells, np.clip(raw, 0, cells - 1))


def in_frame(centre, cell, lower, width, length, inverse, periodic):
    face = (lower + (cell.astype(f32) * width).astype(f32)).astype(f32)
    p = (centre - face).astype(f32)
    wrapped = (p - (np.rint((p * inverse).astype(f32)).astype(f32) * length).astype(f32)).astype(f32)
    return np.where(periodic, wrapped, p)


@pytest.mark.parametrize("wraps", [2, 40])
@pytest.mark.parametrize("cells, walls", [((3, 3, 3), ()), ((4, 4, 4), ()), ((4, 3, 5), ()), ((9, 4, 6), ()),
                                          ((4, 5, 2), (2,)), ((5, 4, 1), (2,))], ids=str)
def test_frame_test_passes_every_exact_pair(cells, walls, wraps):
    rng = np.random.default_rng(sum(cells) + wraps)
    n = 200_000
    cells = np.array(cells)
    periodic = np.array([axis not in walls for axis in range(3)])
    lower = np.array([0.0, -1.0e-4, 3.0e-4], dtype=f32)
    length = (cells * CELL_SIZE * rng.uniform(1.0, 1.1, 3)).astype(f32)
    inverse, width = (f32(1.0) / length).astype(f32), (length / cells.astype(f32)).astype(f32)
    r1, r2 = rng.choice([3.5e-6, 9.5e-6], size=n), rng.choice([3.5e-6, 9.5e-6], size=n)
    u1, u2 = unit(rng.normal(size=(n, 3))), unit(rng.normal(size=(n, 3)))
    tilt = unit(np.cross(u1, rng.normal(size=(n, 3))))
    angle = rng.uniform(0.005, 0.05, size=n)[:, None]
    u2 = np.where((rng.random(n) < 0.4)[:, None], unit(u1 * np.cos(angle) + tilt * np.sin(angle)), u2)
    d1, d2 = u1 * (4.0 * r1)[:, None], u2 * (4.0 * r2)[:, None]
    middle = lower + rng.uniform(0.0, 1.0, size=(n, 3)) * length
    on_face = rng.random((n, 3)) < 0.2
    middle = np.where(on_face, lower + np.round((middle - lower) / width) * width, middle)
    p1 = middle - 0.5 * d1
    x1 = p1 + d1 * rng.random(n)[:, None]
    interaction = (r1 + r2 + float(SKIN)) * 1.0001
    sep = unit(rng.normal(size=(n, 3))) * (interaction * rng.uniform(0.9, 1.05, size=n))[:, None]
    p2 = x1 + sep - d2 * rng.random(n)[:, None]
    chain = (rng.random(n) < 0.4)[:, None]
    bend = rng.uniform(0.0, 0.01, size=n)[:, None]
    p2 = np.where(chain, p1 + d1 + u1 * (interaction * rng.uniform(0.9999, 1.0, size=n))[:, None], p2)
    d2 = np.where(chain, unit(u1 * np.cos(bend) + tilt * np.sin(bend)) * (4.0 * r2)[:, None], d2)
    wrap1, wrap2 = (np.where(periodic, rng.integers(-wraps, wraps + 1, size=(n, 3)) * length.astype(np.float64), 0.0)
                    for _ in range(2))
    p1, q1, p2, q2 = p1 + wrap1, p1 + d1 + wrap1, p2 + wrap2, p2 + d2 + wrap2
    p1, q1, r1, p2, q2, r2 = as_f32(p1, q1, r1, p2, q2, r2)
    exact = exact_build_test(p1, q1, r1, p2, q2, r2, length, periodic)

    home, other = (cells_of(p, q, lower, width, cells, periodic) for p, q in ((p1, q1), (p2, q2)))
    offset = np.where(periodic, (other - home + 1) % cells - 1, other - home)
    scanned = np.all(np.abs(offset) <= 1, axis=1)
    c1, c2 = ((f32(0.5) * (p + q).astype(f32)).astype(f32) for p, q in ((p1, q1), (p2, q2)))
    w1, w2 = ((half_length(p, q) + r).astype(f32) for p, q, r in ((p1, q1, r1), (p2, q2, r2)))

    def size(c):
        return ((np.abs(c[:, 0]) + np.abs(c[:, 1])).astype(f32) + np.abs(c[:, 2])).astype(f32)

    staged = (in_frame(c2, other, lower, width, length, inverse, periodic) +
              (offset.astype(f32) * width).astype(f32)).astype(f32)
    radius = ((w2 * f32(1.0002)).astype(f32) + (f32(4.0e-6) * size(c2)).astype(f32)).astype(f32)
    scale = f32(0.0)
    for axis in range(3):
        scale = f32(scale + f32(abs(lower[axis]) + f32(f32(2.0) * length[axis])))
    home_reach = (((w1 + SKIN).astype(f32) * f32(1.0002)).astype(f32) + f32(1.0e-6) * length.max()).astype(f32)
    home_limit = (home_reach + (f32(4.0e-6) * (size(c1) + f32(f32(2.0) * scale)).astype(f32)).astype(f32)).astype(f32)
    d = (staged - in_frame(c1, home, lower, width, length, inverse, periodic)).astype(f32)
    if np.any(periodic & (cells < 4)):
        nearest = (d - (np.rint((d * inverse).astype(f32)).astype(f32) * length).astype(f32)).astype(f32)
        d = np.where(periodic, nearest, d)
    limit = (home_limit + radius).astype(f32)
    squared = fma(d[:, 0], d[:, 0], fma(d[:, 1], d[:, 1], (d[:, 2] * d[:, 2]).astype(f32)))
    passes = squared <= (limit * limit).astype(f32)
    assert not np.any(exact & scanned & ~passes)
    assert (exact & scanned).sum() > 10_000
