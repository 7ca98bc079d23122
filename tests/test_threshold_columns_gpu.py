"""Which strips a batch of 16-bit frames is taken in: 104 output columns, four a
lane, where the cost model's figure for them is below 1.07 times that of 232,
eight a lane."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def strip_columns(eng, shapes):
    """The strips an engine's tasks are counted in."""
    info = eng.info()
    for out in (104, 232):
        tasks = sum(-(-w // out) * -(-h // min(info["seg_rows"], h)) for h, w in shapes)
        if tasks == info["tasks"]:
            return out
    raise AssertionError(info)


# the faster by measurement on a B200, at the heights the model gives either
@pytest.mark.parametrize("frames,h,w,columns", [
    (1, 256, 384, 104), (1, 700, 900, 104), (1, 800, 800, 104), (1, 1062, 1028, 104),
    (1, 1200, 1200, 104), (1, 300, 4000, 104), (8, 256, 384, 104), (4, 512, 512, 104),
    (16, 512, 512, 104), (1, 1500, 1500, 232), (1, 2162, 2068, 232), (16, 256, 384, 232),
    (32, 256, 384, 232), (64, 128, 128, 232), (4, 700, 900, 232), (16, 2162, 2068, 232)])
def test_the_faster_strips_are_taken(gpu_lib, tmp_path, monkeypatch, frames, h, w, columns):
    import torch
    from dials_metal_spotfinder_b200.engine import Engine
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("measured on 148 SMs")
    monkeypatch.setenv("SPOTFINDER_TUNE_CACHE", str(tmp_path / "none.txt"))
    shapes = [(h, w)] * frames
    with Engine(shapes, np.uint16) as eng:
        assert strip_columns(eng, shapes) == columns
