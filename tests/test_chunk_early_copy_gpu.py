"""Chunks whose bytes are on their way before their framing is checked: a
refused one (each place of a batch, so before, at and after the last staging
set) leaves the decoder fit for the next, and chunks longer than a frame of
incompressible blocks take the other order in the same batch."""

import struct

import numpy as np
import pytest

import dials_metal_spotfinder_b200.chunk as C
from dials_metal_spotfinder_b200._lib import BadArgument
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPE = (130, 261)


def frames(n):
    rng = np.random.default_rng(77)
    out = []
    for _ in range(n):
        img = rng.poisson(1.3, SHAPE).astype(np.uint16)
        img[rng.random(SHAPE) < 0.004] = 900
        out.append(img)
    return out


def tiny_blocks(img):
    """Plain LZ4 of one literal run per 8 bytes: longer than the frame."""
    raw = img.tobytes()
    out = struct.pack(">QI", len(raw), 8)
    for at in range(0, len(raw), 8):
        part = raw[at:at + 8]
        out += struct.pack(">I", len(part) + 1) + bytes([len(part) << 4]) + part
    return np.frombuffer(out, np.uint8)


@pytest.mark.parametrize("n", [1, 3, 5])
def test_a_refused_batch_and_the_next(gpu_lib, n):
    from dials_metal_spotfinder_b200.engine import Engine
    imgs = frames(n)
    good = [C.encode(img, "bslz4") for img in imgs]
    with Engine([SHAPE] * n, np.uint16, slots=2) as eng:
        for at in range(n):
            for bad in (good[at][:-1], good[at][:11], good[at][:12]):
                with pytest.raises(BadArgument):
                    eng.upload_chunks(at % 2, good[:at] + [bad] + good[at + 1:])
            eng.upload_chunks(at % 2, good)
            eng.run(at % 2)
            eng.synchronize()
            for f, img in enumerate(imgs):
                assert eng.signal(at % 2, f).tobytes() == O.dext(img)[1].tobytes()


def test_chunks_longer_than_their_frames(gpu_lib):
    from dials_metal_spotfinder_b200.engine import Engine
    imgs = frames(6)
    short = [C.encode(img, "lz4") for img in imgs]
    long = [tiny_blocks(img) for img in imgs]
    assert all(len(c) > imgs[0].nbytes * 9 / 8 for c in long)
    with Engine([SHAPE] * 6, np.uint16) as eng:
        for first in range(4):  # the batch's first long chunk
            eng.upload_chunks(0, short[:first] + long[first:5] + short[5:], algorithm="lz4")
            eng.run(0)
            eng.synchronize()
            for f, img in enumerate(imgs):
                assert eng.signal(0, f).tobytes() == O.dext(img)[1].tobytes()


def test_device_decode_after_a_refusal(gpu_lib):
    import torch
    img = frames(1)[0]
    dev = torch.empty(SHAPE, dtype=torch.uint16, device="cuda")
    for algorithm in ("lz4", "bslz4"):
        good = C.encode(img, algorithm)
        for bad in (good[:-1], good[:12], good[:5]):
            with pytest.raises(BadArgument):
                C.decode_device(bad, SHAPE, np.uint16, dev.data_ptr(), algorithm=algorithm)
        dev.zero_()
        torch.cuda.synchronize()
        C.decode_device(good, SHAPE, np.uint16, dev.data_ptr(), algorithm=algorithm)
        assert np.array_equal(dev.cpu().numpy(), img)
    long = tiny_blocks(img)
    C.decode_device(long, SHAPE, np.uint16, dev.data_ptr(), algorithm="lz4")
    assert np.array_equal(dev.cpu().numpy(), img)
