"""The device's LZ4 block decode over the forms its copying tells apart:
match offsets below and above the 32 bytes a warp writes at a time, periods
that are copied in words and that are not, long and short matches, literals
of every length, sequence counts at the edges of the 128 a warp holds, block
sizes and rows of every alignment. Blocks are put together sequence by
sequence here, so the expected bytes are known without a decoder."""

import struct

import numpy as np
import pytest

from dials_metal_spotfinder_b200 import chunk as C

pytestmark = pytest.mark.gpu


def length_bytes(n):
    out = bytearray()
    while n >= 255:
        out.append(255)
        n -= 255
    out.append(n)
    return bytes(out)


class Block:
    """An LZ4 block and the bytes it decodes to."""

    def __init__(self, n):
        self.n, self.out, self.lz = n, bytearray(), bytearray()

    def sequence(self, literals, off=0, ml=0):
        lit = len(literals)
        self.lz.append((min(lit, 15) << 4) | (min(ml - 4, 15) if off else 0))
        if lit >= 15:
            self.lz += length_bytes(lit - 15)
        self.lz += literals
        self.out += literals
        if off:
            self.lz += struct.pack("<H", off)
            if ml - 4 >= 15:
                self.lz += length_bytes(ml - 19)
            for _ in range(ml):
                self.out.append(self.out[-off])

    def finish(self, rng):
        """The last sequence: literals up to n (none where n is reached)."""
        self.sequence(rng.integers(0, 256, self.n - len(self.out), dtype=np.uint8).tobytes())
        assert len(self.out) == self.n
        return bytes(self.lz), bytes(self.out)


def random_block(rng, n, kind):
    b = Block(n)
    while True:
        room = n - len(b.out)
        lit, ml = {
            "short": (int(rng.integers(0, 3)), int(rng.integers(4, 12))),
            "long": (int(rng.integers(0, 40)), int(rng.integers(4, 900))),
            "mixed": (int(rng.integers(0, 20)), int(rng.choice([4, 5, 31, 32, 33, 64, 70, 300]))),
        }[kind]
        if not b.out:
            lit = max(lit, 1)
        if lit + ml > room:
            return b.finish(rng)
        have = len(b.out) + lit
        off = int(rng.choice([1, 2, 3, 4, 5, 7, 8, 15, 16, 17, 24, 31, 32, 33, 40, 63, 64, 65,
                              100, 1000, 5000, have]))
        b.sequence(rng.integers(0, 256, lit, dtype=np.uint8).tobytes(), min(off, have), ml)


def counted_block(rng, n, sequences):
    """Exactly `sequences` sequences, the last without literals."""
    b = Block(n)
    b.sequence(b"\x01\x02\x03\x04", 3, 4)
    for k in range(sequences - 3):
        b.sequence(bytes([k & 255]), 1 + k % 37 if k % 37 < len(b.out) else 1, 4)
    off = 6
    b.sequence(b"", off, n - len(b.out))
    b.sequence(b"")
    return bytes(b.lz), bytes(b.out)


def decode_on_device(ch, shape, dtype, pitch):
    import torch
    h, w = shape
    dev = torch.full((h * pitch,), 0xA5, dtype=torch.uint8, device="cuda")
    C.decode_device(ch, shape, dtype, dev.data_ptr(), pitch, "lz4")
    got = dev.cpu().numpy().reshape(h, pitch)
    row = w * np.dtype(dtype).itemsize
    assert (got[:, row:] == 0xA5).all()
    return got[:, :row].tobytes()


def check(blocks, block_bytes, width, dtype=np.uint16):
    raw = b"".join(out for _, out in blocks)
    eb = np.dtype(dtype).itemsize
    assert len(raw) % (width * eb) == 0
    h = len(raw) // (width * eb)
    ch = bytearray(struct.pack(">QI", len(raw), block_bytes))
    for lz, _ in blocks:
        ch += struct.pack(">I", len(lz)) + lz
    ch = np.frombuffer(bytes(ch), np.uint8)
    assert C.decode(ch, (h, width), dtype, "lz4").tobytes() == raw
    for pitch in (width * eb, width * eb + 18, -(-width * eb // 128) * 128 + 20):
        assert decode_on_device(ch, (h, width), dtype, pitch) == raw, (width, pitch)


@pytest.mark.parametrize("kind", ["short", "long", "mixed"])
@pytest.mark.parametrize("block_bytes,width", [(8192, 64), (8192, 1), (8192, 4096), (16384, 2048),
                                               (1000, 25), (8190, 4095), (64, 8)])
def test_random_sequences(gpu_lib, kind, block_bytes, width):
    rng = np.random.default_rng(block_bytes * 7 + width + len(kind))
    check([random_block(rng, block_bytes, kind) for _ in range(24)], block_bytes, width)


@pytest.mark.parametrize("sequences", [3, 4, 5, 8, 127, 128, 129, 130, 255, 256, 257, 513, 1000])
def test_sequence_counts(gpu_lib, sequences):
    rng = np.random.default_rng(sequences)
    check([counted_block(rng, 8192, sequences) for _ in range(3)], 8192, 64)


@pytest.mark.parametrize("off", [1, 2, 3, 4, 6, 8, 12, 16, 20, 31, 32, 33, 47, 64, 96, 200])
def test_one_long_match(gpu_lib, off):
    """From every phase within the 32 bytes a warp writes at a time."""
    rng = np.random.default_rng(off)
    blocks = []
    for lead in range(off, off + 33):
        b = Block(2048)
        b.sequence(rng.integers(0, 256, lead, dtype=np.uint8).tobytes(), off, 1500 + lead)
        blocks.append(b.finish(rng))
    check(blocks, 2048, 32 * 11)
