"""minimum_image's image count, taken for three axes at once, is the division's.

minimum_image (tangle_b200/csrc/common.cuh) takes rintf(x * (1 / L)) box
lengths unless the product is within 1e-3 of a half-integer or beyond 4096;
otherwise it takes roundf(x / L). Restated in f32 on the samples of
test_image_round: the bits of roundf(x / L), signed zeros included, and the
division wherever x is not finite.
"""

import numpy as np
import pytest

from test_image_round import f32, roundf, samples


@pytest.mark.parametrize("length", [f32(v) for v in (2.0e-3, 3.0e-4, 1.0, 7.0, 1.234567e-5, 97.5)], ids=str)
def test_image_count_matches_division(length):
    x = np.concatenate([samples(np.random.default_rng(11), length, 50_000),
                        np.array([np.inf, -np.inf, np.nan], f32)])
    with np.errstate(invalid="ignore"):
        q = (x * (f32(1.0) / length).astype(f32)).astype(f32)
        count = np.rint(q).astype(f32)
        sure = (np.abs((q - count).astype(f32)) < f32(0.499)) & (np.abs(q) < f32(4096.0))
        want = roundf((x / length).astype(f32))
    assert not sure[-3:].any() and sure.mean() > 0.5
    assert np.array_equal(count[sure].view(np.uint32), want[sure].view(np.uint32))
