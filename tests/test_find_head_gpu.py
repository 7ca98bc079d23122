"""sf_find with lists about as long as the head that comes back with the count
(1024 records): one fewer, as many, one more, none, and the caller's capacity
at, below and above the count, against the oracle."""

import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 1023, 1024, 1025, 1500, 2049])
@pytest.mark.parametrize("dtype", [np.uint16, np.uint32])
def test_lengths_around_the_head(gpu_lib, n, dtype):
    from dials_metal_spotfinder_b200._lib import SIGNAL_PIXEL, lib
    h, w = 700, 900
    img = np.zeros((h, w), dtype)
    # one pixel alone is signal
    at = 12 * np.arange(n)
    img[(at // 880) * 12 + 8, at % 880 + 8] = 1000
    status, want, found = O.dext(img)
    assert status == 0 and found == n
    fn = lib.sf_find_u16 if dtype == np.uint16 else lib.sf_find_u32
    for capacity in sorted({0, n - 1, n, n + 1, 1024, 4096} - {-1}):
        out = np.full(max(capacity, 1) + 1, 7, SIGNAL_PIXEL)
        before = out.copy()
        got = ctypes.c_size_t(99)
        status = fn(img.ctypes.data, h, w, out.ctypes.data, capacity, ctypes.byref(got))
        assert got.value == n
        if n > capacity:
            assert status == -2 and out.tobytes() == before.tobytes()
            continue
        assert status == 0
        assert out[:n].tobytes() == want.tobytes()
        assert out[n:].tobytes() == before[n:].tobytes()  # nothing past the count
