"""The threshold at the edges of its strips (232 output columns for 16-bit
pixels, 108 for 32-bit ones) and of a lane's columns (8 and 4): widths just
below, at and above multiples of either, with signal, masked pixels and the
largest values along every boundary, against the oracle."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def edges(dtype, w, h, large):
    rng = np.random.default_rng(w * 7 + h)
    img = rng.poisson(2.0, (h, w)).astype(dtype)
    top = np.iinfo(dtype).max
    out = 232 if dtype == np.uint16 else 108
    for at in list(range(0, w + out, out)) + [w]:
        for x in range(at - 12, at + 12):
            if 0 <= x < w:
                kind = rng.integers(0, 8)
                y = rng.integers(0, h)
                if kind < 4:  # a spot
                    img[max(0, y - 1):y + 2, max(0, x - 1):x + 2] += dtype(rng.integers(30, 3000))
                elif kind < 6:  # masked: either sentinel
                    img[y, x] = top - rng.integers(0, 2)
                elif large:  # sums of squares that wrap
                    img[y, x] = top - 2 - rng.integers(0, 5)
    return img


@pytest.mark.parametrize("large", [False, True])
@pytest.mark.parametrize("dtype,widths", [
    (np.uint16, [1, 7, 8, 9, 231, 232, 233, 255, 256, 257, 463, 464, 465, 697]),
    (np.uint32, [1, 3, 4, 5, 107, 108, 109, 127, 128, 129, 215, 216, 217, 324, 325, 1081])])
def test_widths_around_strips(gpu_lib, dtype, widths, large):
    from dials_metal_spotfinder_b200.engine import Engine
    shapes = [(h, w) for w in widths for h in (1, 11, 64)]
    frames = [edges(dtype, w, h, large) for h, w in shapes]
    for warps in (1, 2, 4):
        with Engine(shapes, dtype, warps_per_block=warps) as eng:
            for f, img in enumerate(frames):
                eng.upload(0, f, img)
            eng.run(0)
            eng.synchronize()
            for f, img in enumerate(frames):
                _, want, found = O.dext(img)
                got_status, got = eng.signal_status(0, f)
                # a list holds a record per 16 bytes of its frame
                assert got_status == (0 if found <= img.nbytes // 16 else -2)
                if got_status == 0:
                    assert got.tobytes() == want.tobytes(), (shapes[f], warps)


@pytest.mark.parametrize("large", [False, True])
@pytest.mark.parametrize("w", [1, 3, 4, 5, 103, 104, 105, 127, 128, 129, 207, 208, 209, 384, 521])
def test_narrow_strips_of_small_frames(gpu_lib, w, large):
    """One small 16-bit frame: strips of 104 output columns, 4 a lane, where
    the task height is not given; and the same frame with it given, in strips
    of 232. Through sf_find too, which leaves it open."""
    import dials_metal_spotfinder_b200 as sf
    from dials_metal_spotfinder_b200.engine import Engine
    for h in (1, 10, 67, 256):
        img = edges(np.uint16, w, h, large)
        _, want, found = O.dext(img)
        fits = found <= img.nbytes // 16
        for seg in (0, 4):
            with Engine([(h, w)], np.uint16, seg_rows=seg) as eng:
                info = eng.info()
                strips = -(-w // (232 if seg else 104))
                assert info["tasks"] == strips * -(-h // info["seg_rows"])
                eng.upload(0, 0, img)
                eng.run(0)
                eng.synchronize()
                status, got = eng.signal_status(0, 0)
                assert status == (0 if fits else -2)
                assert not fits or got.tobytes() == want.tobytes()
        if fits:
            assert sf.find(img).tobytes() == want.tobytes()
