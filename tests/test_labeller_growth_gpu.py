"""sf_labeller_* over series whose frames and open pixels outgrow what the
labeller has made room for, again and again and across gaps in the numbering:
the carry has to come through every move. Against the oracle."""

import numpy as np
import pytest

from conftest import same_spots
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def signal(rng, h, w, n, fixed):
    """n pixels at random, and a set that stays signal on every frame (so it
    stays open)."""
    index = np.unique(np.concatenate([rng.choice(h * w, n, replace=False), fixed]))
    sig = np.zeros(len(index), O.SIGNAL_PIXEL)
    sig["index"] = index
    sig["value"] = rng.integers(1, 60000, len(index))
    return sig


@pytest.mark.parametrize("sizes", [
    [1, 10, 16383, 16384, 16385, 40000, 0, 3, 90000],
    [30000] * 7,
    [200, 0, 25000, 24000, 60000, 100, 59999],
])
def test_growing_series(gpu_lib, sizes):
    from dials_metal_spotfinder_b200.labeller import group
    h, w = 400, 500
    rng = np.random.default_rng(len(sizes))
    fixed = rng.choice(h * w, 3000, replace=False)
    signals = [signal(rng, h, w, n, fixed) for n in sizes]
    frames = [z + (2 if z > 4 else 0) for z in range(len(sizes))]  # a gap
    spots, pixels, counts = group(signals, h, w, frames, max_separation=0.0)
    want = O.group(signals, h, w, frames, max_separation=0.0)
    assert counts == want.counts
    assert pixels.tobytes() == want.pixels.tobytes()
    same_spots(spots, want.spots)
