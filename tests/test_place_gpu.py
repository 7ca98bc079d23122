"""The ordered placement at the edges of its groups of 1024 (row, strip)
tiles: frames of one tile fewer, exactly as many and one more, tiny frames
between large ones, groups with no records and with full rows, lists cut at
their capacity -- every frame's list against the oracle."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (height, width): width <= 232 is one strip, 233..464 two
BATCHES = [
    [(1023, 100), (1024, 100), (1025, 100), (1, 40), (2048, 60), (512, 300), (513, 300)],
    [(3, 3), (1100, 700), (5, 240), (64, 64)],
    [(2100, 500)] * 3,
]


def frame(rng, h, w, dtype, dense):
    img = rng.poisson(1.0, (h, w)).astype(dtype)
    n = max(1, h * w // (60 if dense else 900))
    y, x = rng.integers(0, h, n), rng.integers(0, w, n)
    for a, b in zip(y, x):
        img[max(0, a - 1):a + 2, max(0, b - 1):b + 2] += dtype(rng.integers(20, 900))
    img[h // 3:h // 3 + h // 4] = 0  # groups without a record
    return img


@pytest.mark.parametrize("dtype", [np.uint16, np.uint32])
@pytest.mark.parametrize("shapes", BATCHES)
def test_lists_at_group_edges(gpu_lib, shapes, dtype):
    from dials_metal_spotfinder_b200.engine import Engine
    rng = np.random.default_rng(5)
    with Engine(shapes, dtype, slots=2) as eng:
        for slot in range(2):
            frames = [frame(rng, h, w, dtype, k % 2 == slot) for k, (h, w) in enumerate(shapes)]
            for f, img in enumerate(frames):
                eng.upload(slot, f, img)
            eng.run(slot)
            eng.synchronize()
            counts = eng.counts(slot)
            for f, img in enumerate(frames):
                want_status, want, n = O.dext(img, capacity=img.size * img.itemsize // 16)
                status, got = eng.signal_status(slot, f)
                assert (counts[f], status) == (n, want_status), f
                if status == 0:
                    assert got.tobytes() == want.tobytes(), f
