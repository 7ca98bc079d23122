"""A grouping launch's wait for tiles that are never published ends by its
limit and is reported as that, not as a capacity: tests/cpp/wait_check.cu,
built beside the library."""

import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_wait_gives_up_and_says_so(gpu_lib):
    exe = os.path.join(ROOT, "dials_metal_spotfinder_b200", "_build", "wait_check")
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stderr
    published, late, timeout, overflow = p.stdout.splitlines()
    assert published == "prefix 23 status 0 own 36 done 1"
    assert late == "prefix 0 status 3 own 13 done 1"
    assert timeout == "grouping: a wait on the device gave up (status 3)"
    assert overflow == "grouping capacity exceeded (status 1)"
