"""The labeller at the edges of its one-block launches (4096 pixels held and
added) and of the results that come back with the counts (128 spots, 1536 pixels): batches
just below, at and above each, components of every size class in a small
batch, and series that cross the edge both ways, against the oracle."""

import numpy as np
import pytest

from conftest import same_spots
from oracle import oracle as O

pytestmark = pytest.mark.gpu

H, W = 300, 400
EDGE = 4096


def listed(mask, seed):
    rng = np.random.default_rng(seed)
    sig = np.zeros(int(mask.sum()), O.SIGNAL_PIXEL)
    sig["index"] = np.flatnonzero(mask)
    sig["value"] = rng.integers(1, 60000, len(sig))
    return sig


def check(signals, frames=None, **opt):
    from dials_metal_spotfinder_b200.labeller import group
    spots, pixels, counts = group(signals, H, W, frames, **opt)
    want = O.group(signals, H, W, frames, **opt)
    assert counts == want.counts
    same_spots(spots, want.spots)
    assert pixels.tobytes() == want.pixels.tobytes()
    return spots


def some(n, seed):
    """n pixels in blobs."""
    rng = np.random.default_rng(seed)
    mask = np.zeros((H, W), bool)
    while mask.sum() < n:
        y, x = rng.integers(0, H - 4), rng.integers(0, W - 4)
        mask[y:y + rng.integers(1, 5), x:x + rng.integers(1, 5)] = True
    on = np.flatnonzero(mask)
    mask.flat[rng.choice(on, len(on) - n, replace=False)] = False
    return mask


@pytest.mark.parametrize("held", [0, 1000])
@pytest.mark.parametrize("by", [-1, 0, 1])
@pytest.mark.parametrize("two_d", [False, True])
def test_pixels_around_the_edge(gpu_lib, held, by, two_d):
    # a whole frame stays held, so the second batch is `held` longer
    first, second = some(held, 1), some(EDGE + by - held, 2)
    check([listed(first, 3), listed(second, 4), listed(some(37, 5), 6)], two_d=two_d)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 700])
def test_spots_around_the_head(gpu_lib, n):
    # isolated pixels of one frame, all finished by the next
    mask = np.zeros((H, W), bool)
    at = 3 * np.arange(n)
    mask[at // W * 2, at % W] = True
    spots = check([listed(mask, 7), listed(np.zeros((H, W), bool), 8)], min_spot_size=1,
                  max_separation=0.0)
    assert len(spots) == n


@pytest.mark.parametrize("n", [511, 512, 513])
def test_finished_pixels_around_the_head(gpu_lib, n):
    # 3 n pixels in spots of three
    mask = np.zeros((H, W), bool)
    for k in range(n):
        mask[k // 50 * 2, k % 50 * 6:k % 50 * 6 + 3] = True
    check([listed(mask, 10), listed(np.zeros((H, W), bool), 11)], max_separation=0.0)
    # as few spots as there can be
    tall = np.zeros((H, W), bool)
    tall[:, 3:10] = True
    tall.flat[np.flatnonzero(tall)[3 * n:]] = False
    check([listed(tall, 12)], max_spot_size=5000, max_separation=0.0)


@pytest.mark.parametrize("sizes", [(256, 257), (512, 513), (1024, 1025), (1500, 1, 2, 3)])
def test_components_of_every_size_class(gpu_lib, sizes):
    mask = np.zeros((H, W), bool)
    for k, n in enumerate(sizes):
        block = np.zeros((60, 50), bool)
        block.flat[:n] = True
        mask[70 * k:70 * k + 60, 5:55] = block
    check([listed(mask, 9)], max_spot_size=1400, min_spot_size=1, max_separation=0.0)
    check([listed(mask, 9)], max_spot_size=2000, min_spot_size=1)
    check([listed(mask, 9)] * 2, max_spot_size=5000)


def test_a_series_that_crosses_the_edge_both_ways(gpu_lib):
    sizes = [10, 3000, 900, 3500, 5000, 0, 20, 4096, 0, 0, 300]
    signals = [listed(some(n, 20 + k) if n else np.zeros((H, W), bool), 40 + k)
               for k, n in enumerate(sizes)]
    check(signals)
    check(signals, frames=[2 * k + (k > 4) for k in range(len(sizes))])
    check(signals, two_d=True, min_spot_size=2, max_spot_size=9)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("nframes", [1, 3])
def test_an_engine_small_enough(gpu_lib, nframes, graph):
    """An engine whose lists and carry hold no more than the edge takes the
    one-block launches too, replayed from graphs as well."""
    from dials_metal_spotfinder_b200._lib import PIXEL, SPOT
    from dials_metal_spotfinder_b200.engine import Engine
    h, w, runs = 90, 110, 5
    rng = np.random.default_rng(61)
    frames = []
    for _ in range(nframes * runs):
        img = rng.poisson(1.0, (h, w)).astype(np.uint16)
        for y, x in zip(rng.integers(2, h - 3, 12), rng.integers(2, w - 3, 12)):
            img[y:y + 3, x:x + 3] += np.uint16(rng.integers(40, 900))
        frames.append(img)
    want = O.group([O.dext(f)[1] for f in frames], h, w)
    spots, pixels = [], []
    with Engine([(h, w)] * nframes, np.uint16) as eng:
        eng.enable_grouping(carry_capacity=300)
        eng.use_graph(graph)
        for r in range(runs):
            for f in range(nframes):
                eng.upload(0, f, frames[r * nframes + f])
            eng.run(0)
            spots.append(eng.spots())
            pixels.append(eng.pixels())
        eng.finish()
        spots.append(eng.spots())
        pixels.append(eng.pixels())
        counts, _ = eng.group_counts()
    assert counts == want.counts
    same_spots(np.concatenate(spots).astype(SPOT), want.spots)
    assert np.concatenate(pixels).astype(PIXEL).tobytes() == want.pixels.tobytes()
