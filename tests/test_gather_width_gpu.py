"""The grouping of batches at both sides of the frame area from which a warp of
the gather takes four chunks of positions at a time: few and many pixels, more
frames than fit the segments' shared copy, lists that end around a chunk and
around a warp's and a block's four. Against the oracle, the form by the
kernels that ran."""

import numpy as np
import pytest

from conftest import same_spots
from oracle import oracle as O

pytestmark = pytest.mark.gpu

AREA = 1 << 24


def lone(h, w, pixels, rng):
    """A frame with exactly `pixels` signal pixels, 8 apart."""
    img = np.zeros((h, w), np.uint16)
    k, per_row = np.arange(pixels), (w - 16) // 8
    img[8 + 8 * (k // per_row), 8 + 8 * (k % per_row)] = rng.integers(20000, 60000, pixels)
    return img


def grouped(images):
    from torch.profiler import ProfilerActivity, profile
    from dials_metal_spotfinder_b200.engine import Engine
    h, w = images[0].shape
    with Engine([(h, w)] * len(images)) as eng, \
            profile(activities=[ProfilerActivity.CUDA]) as prof:
        eng.enable_grouping()
        for f, img in enumerate(images):
            eng.upload(0, f, img)
        spots, pixels = [], []
        for step in (lambda: eng.run(0), lambda: eng.run(0), eng.finish):
            step()
            spots.append(eng.spots())
            pixels.append(eng.pixels())
        counts = eng.group_counts()[0]
    lists = [O.dext(img)[1] for img in images]
    want = O.group(lists + lists, h, w)
    assert counts == want.counts
    assert np.concatenate(pixels).tobytes() == want.pixels.tobytes()
    same_spots(np.concatenate(spots), want.spots)
    return [len(sig) for sig in lists], {e.name for e in prof.events() if "lab_gather" in e.name}


@pytest.mark.parametrize("frames,h,w", [
    (2, 2896, 2897), (2, 2896, 2896), (131, 360, 356), (131, 360, 355), (9, 1366, 1365)])
def test_both_widths(gpu_lib, frames, h, w):
    rng = np.random.default_rng(frames)
    sizes = np.resize([127, 1, 128, 0, 129, 31, 1023, 33, 1025], frames)
    lists, kernels = grouped([lone(h, w, int(n), rng) for n in sizes])
    assert lists == sizes.tolist()
    # the batches' form; finish(), which has no frames, takes one chunk
    four = [k for k in kernels if "<4>" in k or "ILi4E" in k]
    assert kernels and bool(four) == (frames * h * w >= AREA), kernels
