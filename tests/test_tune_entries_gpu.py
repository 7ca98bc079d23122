"""What an engine makes of the tuner file's entries."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_entries_of_another_kernel_are_not_read(gpu_lib, tmp_path, monkeypatch):
    """An entry with no kernel version holds blocks per SM and a height that
    were measured with another kernel and model."""
    import torch
    from dials_metal_spotfinder_b200.engine import Engine
    from dials_metal_spotfinder_b200.tune import tune
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("SPOTFINDER_TUNE_CACHE", str(cache))
    p = torch.cuda.get_device_properties(0)
    key = f"u32:300x400:sm{p.multi_processor_count}:{p.name.replace(' ', '_')}"
    with Engine([(300, 400)] * 2, np.uint32) as eng:
        untuned = eng.tuning(), eng.info()["grid_blocks"]
    cache.write_text(f"{key} 8 1 2 20.5 1\n")
    with Engine([(300, 400)] * 2, np.uint32) as eng:
        assert (eng.tuning(), eng.info()["grid_blocks"]) == untuned
        assert not eng.tuning()["from_cache"]
    # the key is that of an entry written now, but for the version
    tune([np.zeros((300, 400), np.uint32)] * 2, min_frames=2, max_frames=2, steps=1)
    written = cache.read_text().splitlines()[-1].split()[0]
    assert written.endswith(key) and written != key
    with Engine([(300, 400)] * 2, np.uint32) as eng:
        assert eng.tuning()["from_cache"]


@pytest.mark.parametrize("frames,h,w", [(8, 256, 384), (8, 512, 512), (2, 1062, 1028)])
def test_an_entry_is_relative_to_the_model(gpu_lib, tmp_path, monkeypatch, frames, h, w):
    """Small batches, for which the model picks heights below 16 rows and
    strips of 104 columns: an entry multiplies that height, and leaves the
    strips as they are."""
    from dials_metal_spotfinder_b200.engine import Engine
    from dials_metal_spotfinder_b200.tune import tune
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("SPOTFINDER_TUNE_CACHE", str(cache))
    rng = np.random.default_rng(3)
    tuned = tune([rng.poisson(1.0, (h, w)).astype(np.uint16) for _ in range(frames)],
                 min_frames=frames, max_frames=frames, steps=1)
    key = cache.read_text().split()[0]
    shapes = [(h, w)] * frames
    for warps in (1, 2, 4):
        with Engine(shapes, np.uint16, warps_per_block=warps) as eng:  # the model's
            model = eng.info()
        for ratio in (0.5, 1, 1.5, 2):
            cache.write_text(f"{key} {frames} {warps} {ratio} 20.5 0\n")
            with Engine(shapes, np.uint16) as eng:
                assert eng.tuning()["from_cache"]
                info = eng.info()
            rows = max(min(16, model["seg_rows"]), min(int(model["seg_rows"] * ratio + 0.5), h))
            strips = model["tasks"] // (frames * -(-h // model["seg_rows"]))
            assert info["seg_rows"] == rows
            assert info["tasks"] == frames * strips * -(-h // rows)
    if tuned["blocks_per_sm"] == 0:
        with Engine(shapes, np.uint16, warps_per_block=tuned["warps_per_block"]) as eng:
            base = eng.info()["seg_rows"]
        assert tuned["seg_rows"] == max(min(16, base),
                                        min(int(base * tuned["seg_ratio"] + 0.5), h))
