"""The grouping at the edges of its tiles: 2048 and 8192 live positions, 64
finished components, 2048 bucket counts -- one fewer, as many and one more,
in 2D, in 3D with everything finished at once, and with open components
carried from frame to frame. Against the oracle."""

import numpy as np
import pytest

from conftest import same_spots
from oracle import oracle as O

pytestmark = pytest.mark.gpu

H, W = 600, 700


def runs(count, length, first=0):
    """`count` separate runs of `length` pixels, none touching another."""
    per_row = W // (length + 1)
    k = first + np.arange(count)
    start = 2 * (k // per_row) * W + (k % per_row) * (length + 1)
    return np.sort((start[:, None] + np.arange(length)).reshape(-1))


def as_signal(index, seed):
    sig = np.zeros(len(index), O.SIGNAL_PIXEL)
    sig["index"] = index
    sig["value"] = np.random.default_rng(seed).integers(1, 5000, len(index))
    return sig


def check(signals, **options):
    from dials_metal_spotfinder_b200.labeller import group
    spots, pixels, counts = group(signals, H, W, **options)
    want = O.group(signals, H, W, **options)
    assert counts == want.counts
    assert pixels.tobytes() == want.pixels.tobytes()
    same_spots(spots, want.spots)


@pytest.mark.parametrize("two_d", [False, True])
@pytest.mark.parametrize("components", [1, 31, 32, 33, 63, 64, 65, 511, 512, 513, 682, 683,
                                        2730, 2731, 8192, 8193])
def test_component_counts(gpu_lib, components, two_d):
    # three pixels each: 683 components pass 2048 positions, 2731 pass 8192
    check([as_signal(runs(components, 3), 1)], two_d=two_d, max_separation=0.0)


@pytest.mark.parametrize("pixels", [2047, 2048, 2049, 4096, 8191, 8192, 8193, 16384, 16385])
def test_position_counts(gpu_lib, pixels):
    # too small, accepted and too large ones among them
    sizes = np.resize([1, 3, 40, 2, 5], pixels)
    index, at, k = [], 0, 0
    while at < pixels:
        n = min(int(sizes[k]), pixels - at)
        index.append(runs(1, 40, k)[:n])
        at, k = at + n, k + 1
    check([as_signal(np.concatenate(index), 2)], max_spot_size=39, max_separation=0.0)


@pytest.mark.parametrize("frames", [2, 5, 33, 40])
def test_carried_components(gpu_lib, frames):
    # a component that ends on every frame, many that go on to the last
    lists = [np.sort(np.concatenate([runs(700, 3), runs(60 * (frames - z), 2, 5000)]))
             for z in range(frames)]
    check([as_signal(i, z) for z, i in enumerate(lists)], max_separation=0.0)


@pytest.mark.parametrize("frames", [1, 31, 32, 33, 64, 130])
def test_buckets_of_one_batch(gpu_lib, frames):
    """Components that close on every frame of one engine batch: more buckets
    than one scan tile, more frames than the segment lanes."""
    from dials_metal_spotfinder_b200.engine import Engine
    h, w = 96, 130
    rng = np.random.default_rng(frames)
    images = []
    for z in range(frames):
        img = rng.poisson(0.4, (h, w)).astype(np.uint16)
        y, x = rng.integers(3, h - 3, 30), rng.integers(3, w - 3, 30)
        for a, b in zip(y, x):
            img[a - 1:a + 2, b - 1:b + 2] += np.uint16(400)
        images.append(img)
    lab = O.Labeller(h, w)
    for z, img in enumerate(images):
        lab.add(z, O.dext(img)[1])
    lab.finish()
    want = lab.result()
    with Engine([(h, w)] * frames) as eng:
        eng.enable_grouping()
        for f, img in enumerate(images):
            eng.upload(0, f, img)
        eng.run(0)
        spots, pixels = [eng.spots()], [eng.pixels()]
        eng.finish()
        spots.append(eng.spots())
        pixels.append(eng.pixels())
        counts = eng.group_counts()[0]
    assert counts == want.counts
    assert np.concatenate(pixels).tobytes() == want.pixels.tobytes()
    same_spots(np.concatenate(spots), want.spots)
