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
