"""The threshold where its warps share the rows of their tasks: heights just
below and above the shortest shared task, odd heights and claims' remainders,
frames whose rows cost very differently (so that rows are taken from others),
every block size, either pixel type. Every list against the oracle."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def lopsided(rng, h, w, dtype):
    """Masked columns and dense candidates on one side, nothing on the other."""
    img = rng.poisson(1.2, (h, w)).astype(dtype)
    img[:, w // 2:] = 0
    img[:, : w // 8] = np.iinfo(dtype).max
    n = h * w // 150
    y, x = rng.integers(0, h, n), rng.integers(0, max(1, w // 3), n)
    for a, b in zip(y, x):
        img[max(0, a - 1):a + 2, max(0, b - 1):b + 2] //= 2
        img[max(0, a - 1):a + 2, max(0, b - 1):b + 2] += dtype(rng.integers(20, 900))
    return img


@pytest.mark.parametrize("dtype,warps", [(np.uint16, 1), (np.uint16, 2), (np.uint16, 4),
                                         (np.uint32, 1), (np.uint32, 2)])
@pytest.mark.parametrize("seg", [95, 96, 97, 128, 333, 5000])
def test_shared_rows(gpu_lib, dtype, warps, seg):
    from dials_metal_spotfinder_b200.engine import Engine
    rng = np.random.default_rng(seg + warps)
    shapes = [(701, 700), (333, 470), (95, 233), (1, 300), (1003, 231)]
    frames = [lopsided(rng, h, w, dtype) for h, w in shapes]
    with Engine(shapes, dtype, seg_rows=seg, warps_per_block=warps) as eng:
        for f, img in enumerate(frames):
            eng.upload(0, f, img)
        for _ in range(3):  # the order in which rows are taken varies
            eng.run(0)
            eng.synchronize()
            for f, img in enumerate(frames):
                want_status, want, n = O.dext(img, capacity=img.size * img.itemsize // 16)
                status, got = eng.signal_status(0, f)
                assert status == want_status, f
                if status == 0:
                    assert got.tobytes() == want.tobytes(), f
