"""sf_find on frames at both sides of the size from which a frame crosses to
the device in one contiguous copy and is laid out there (plan.cu): row lengths
that divide into words of every width, either pixel type, page-locked and
ordinary memory, one shape after another in one thread, against the oracle."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(512, 511), (512, 512), (513, 512), (1031, 263), (700, 1030), (64, 4099), (4103, 66)]


@pytest.mark.parametrize("dtype", [np.uint16, np.uint32])
@pytest.mark.parametrize("pinned", [False, True])
def test_both_uploads(gpu_lib, dtype, pinned):
    import dials_metal_spotfinder_b200 as sf
    rng = np.random.default_rng(11)
    for h, w in SHAPES + SHAPES[:2]:
        img = rng.poisson(1.5, (h, w)).astype(dtype)
        y, x = rng.integers(0, h, 60), rng.integers(0, w, 60)
        img[y, x] += dtype(500)
        img[rng.random((h, w)) < 0.002] = np.iinfo(dtype).max
        frame = img
        if pinned:
            buf = sf.HostBuffer((h, w), dtype)
            buf.array[:] = img
            frame = buf.array
        status, want, _ = O.dext(img)
        got_status, got = sf.find_status(frame)
        assert (got_status, got.tobytes()) == (status, want.tobytes()), (h, w)
