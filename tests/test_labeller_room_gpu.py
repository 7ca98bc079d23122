"""How much device memory a labeller takes for pixels it has not been given
yet: never more than a sixteenth of what is free, small buffers aside."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIDE = 8192
BYTES = 208  # a pixel's buffers, and something for rounding
LIST = 16    # ... and its record


def lone(n):
    """n pixels, none beside another, in a SIDE x SIDE frame."""
    at = 4 * np.arange(n, dtype=np.int64)
    sig = np.zeros(n, O.SIGNAL_PIXEL)
    sig["index"] = at + 2 * (at // SIDE % 2)
    sig["value"] = 7
    return sig


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_room_is_a_share_of_the_free_memory(gpu_lib):
    from dials_metal_spotfinder_b200.labeller import Labeller
    n = SIDE * SIDE // 4
    with_room = 7.5 * n * (BYTES - 20)  # half as much again, and four such batches
    free = free_bytes()
    if with_room < free / 16:
        pytest.skip("a device on which all the room fits its share")
    lab = Labeller(SIDE, SIDE)
    lab.add(0, lone(n))
    assert free - free_bytes() < free / 16
    lab.finish()
    counts = lab.counts()
    lab.close()
    assert counts["signal_pixels"] == counts["groups"] == counts["too_small"] == n


def test_room_is_not_asked_for_again(gpu_lib):
    """Where a batch leaves no room, the labeller grows to what it was asked
    for, not to that and the room it once had."""
    from dials_metal_spotfinder_b200.labeller import Labeller
    first, second = SIDE * SIDE // 16, SIDE * SIDE // 4
    free = free_bytes()
    if 7.5 * second * (BYTES - 20) < free / 16 or 7.5 * first * BYTES > free / 16:
        pytest.skip("a device on which both batches have room, or neither")
    lab = Labeller(SIDE, SIDE)
    lab.add(0, lone(first))
    lab.add(1, lone(second))
    used = free - free_bytes()
    assert lab.live() == first + second  # joined across the frames, or new
    assert used < (first + second) * BYTES + second * LIST + (64 << 20)
    lab.finish()
    assert lab.counts()["groups"] == second
    lab.close()
