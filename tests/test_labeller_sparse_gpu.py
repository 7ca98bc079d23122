"""The labeller on large frames with few signal pixels: the one-block launches
are for batches whose pixels and block tables (a word per 64 pixels of a
frame's area) are both small, so a 2162 x 2068 or 4362 x 4148 frame is left to
the launches of many blocks however sparse it is. Results against the oracle,
the route by the kernels that ran."""

import numpy as np
import pytest

from conftest import same_spots
from oracle import oracle as O

pytestmark = pytest.mark.gpu

EDGE, TABLE = 4096, 16  # pixels, and the table words that count as one


def table_pixels(h, w):
    return (h * w // 64 + 2) // TABLE


def blobs(h, w, n, seed):
    """n pixels of 2 x 2 blobs at random."""
    rng = np.random.default_rng(seed)
    at = np.zeros(0, np.int64)
    while len(at) < n:
        y, x = rng.integers(0, h - 1, n), rng.integers(0, w - 1, n)
        new = np.concatenate([(y + a) * w + x + b for a in (0, 1) for b in (0, 1)])
        at = np.unique(np.concatenate([at, new]))
    sig = np.zeros(n, O.SIGNAL_PIXEL)
    sig["index"] = np.sort(rng.choice(at, n, replace=False)) if n else []
    sig["value"] = rng.integers(1, 60000, n)
    return sig


def grouped(signals, h, w, **opt):
    """group() checked against the oracle, and the kernels that ran."""
    from torch.profiler import ProfilerActivity, profile
    from dials_metal_spotfinder_b200.labeller import group
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        spots, pixels, counts = group(signals, h, w, **opt)
    want = O.group(signals, h, w, **opt)
    assert counts == want.counts
    same_spots(spots, want.spots)
    assert pixels.tobytes() == want.pixels.tobytes()
    names = [e.name for e in prof.events()]
    assert any("lab_" in n for n in names), "no kernel was recorded"
    return sum("lab_small_open" in n for n in names), sum("lab_gather" in n for n in names)


@pytest.mark.parametrize("two_d", [False, True])
@pytest.mark.parametrize("h,w", [(2162, 2068), (4362, 4148)])
def test_large_sparse_frames(gpu_lib, h, w, two_d):
    signals = [blobs(h, w, n, 3 + k) for k, n in enumerate([0, 500, 3000, 0, 40, 900])]
    small, many = grouped(signals, h, w, two_d=two_d)
    # only what is left at the end, which has no frame, is one block's
    assert (small, many) == (1, len(signals))


@pytest.mark.parametrize("h,w", [(300, 400), (1021, 999), (1500, 1500)])
def test_both_sides_of_the_rule(gpu_lib, h, w):
    edge = EDGE - table_pixels(h, w)
    for by, small in ((-1, 2), (0, 2), (1, 1)):
        assert grouped([blobs(h, w, edge + by, 11 + by)], h, w)[0] == small
