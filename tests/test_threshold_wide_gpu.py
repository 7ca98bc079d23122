"""The edges of the 232-column strips, eight columns a lane, of 16-bit frames:
what sf_find and an engine without a task height leave to strips of 104 at
these sizes. Widths around the strips and the lanes, ragged and uniform frames,
sums of squares that wrap, tiles around the placement's groups; and strips of
104 whose warps share rows. Against the oracle, the strips by the tasks."""

import numpy as np
import pytest

from oracle import oracle as O
from test_place_gpu import BATCHES, frame
from test_threshold_columns_gpu import strip_columns
from test_threshold_sharing_gpu import lopsided
from test_threshold_strips_gpu import edges

pytestmark = pytest.mark.gpu


def check(shapes, frames, columns, runs=1, **config):
    from dials_metal_spotfinder_b200.engine import Engine
    with Engine(shapes, np.uint16, **config) as eng:
        assert strip_columns(eng, shapes) == columns
        for f, img in enumerate(frames):
            eng.upload(0, f, img)
        wanted = {}
        for _ in range(runs):
            eng.run(0)
            eng.synchronize()
            for f, img in enumerate(frames):
                if id(img) not in wanted:
                    wanted[id(img)] = O.dext(img, capacity=max(1, img.nbytes // 16))
                want_status, want, n = wanted[id(img)]
                status, got = eng.signal_status(0, f)
                assert (status, eng.counts(0)[f]) == (want_status, n), shapes[f]
                if status == 0:
                    assert got.tobytes() == want.tobytes(), shapes[f]
        return eng.info()


@pytest.mark.parametrize("large", [False, True])
@pytest.mark.parametrize("warps", [1, 2, 4])
@pytest.mark.parametrize("seg", [4, 23])
def test_widths_around_strips(gpu_lib, seg, warps, large):
    widths = [1, 7, 8, 9, 231, 232, 233, 255, 256, 257, 463, 464, 465, 697]
    shapes = [(h, w) for w in widths for h in (1, 11, 64)]
    frames = [edges(np.uint16, w, h, large) for h, w in shapes]
    check(shapes, frames, 232, seg_rows=seg, warps_per_block=warps)


def ragged(h, w):
    rng = np.random.default_rng(h * 10007 + w)
    img = rng.poisson(3.0, (h, w)).astype(np.uint16)
    for y, x in zip(rng.integers(0, h, h * w // 400 + 1), rng.integers(0, w, h * w // 400 + 1)):
        img[max(0, y - 1):y + 2, max(0, x - 1):x + 2] += np.uint16(rng.integers(30, 3000))
    img[rng.random((h, w)) < 0.01] = 0xFFFF
    img[rng.random((h, w)) < 0.01] = 0xFFFE
    return img


def wrapping():
    rng = np.random.default_rng(3)
    img = rng.poisson(2.0, (120, 350)).astype(np.uint16)
    for x in (40, 228, 330):  # within a strip and across its end
        img[40:47, x:x + 7] = rng.integers(20000, 65533, (7, 7))
        img[70, x] = img[95:98, x + 2] = 65533
        img[85:87, x - 9:x + 4] = rng.integers(3000, 65000, (2, 13))
        img[20:23, x + 8:x + 10] = rng.integers(300, 60000, (3, 2))
    return img


def test_ragged_uniform_and_wrapping_frames(gpu_lib):
    frames = [ragged(h, w) for h, w in [(2, 2), (5, 300), (300, 5), (21, 231), (22, 232),
                                        (23, 233), (40, 464), (41, 465), (257, 511),
                                        (600, 700)]]
    frames += [np.full((70, 300), v, np.uint16) for v in (0, 1, 0xFFFE, 0xFFFF, 0xFFFD)]
    frames.append(wrapping())
    check([f.shape for f in frames], frames, 232, seg_rows=9)


@pytest.mark.parametrize("shapes", BATCHES[:2])
def test_tiles_around_the_placement_groups(gpu_lib, shapes):
    rng = np.random.default_rng(6)
    frames = [frame(rng, h, w, np.uint16, k % 2 == 0) for k, (h, w) in enumerate(shapes)]
    check(shapes, frames, 232, seg_rows=37)


@pytest.mark.parametrize("warps", [1, 2, 4])
def test_shared_rows_of_narrow_strips(gpu_lib, tmp_path, monkeypatch, warps):
    """Tall frames of one strip of 104: their tasks are high enough to share."""
    monkeypatch.setenv("SPOTFINDER_TUNE_CACHE", str(tmp_path / "none.txt"))
    rng = np.random.default_rng(warps)
    made = [lopsided(rng, 4362, 104, np.uint16) for _ in range(4)]
    info = check([(4362, 104)] * 64, made * 16, 104, runs=2, warps_per_block=warps)
    assert info["seg_rows"] >= 96
