"""Long sequences of the device's LZ4 decoder: matches of thousands of bytes from every kind
of offset after zero to hundreds of literals, in a checkpoint whose colour plane is replaced
by a block written here. The plane must come back as the format defines the block.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 512, 256
HEAD = 9000  # literals first, so that the farthest offset lies inside
OFFSETS = [1, 2, 3, 4, 5, 7, 12, 31, 63, 64, 100, 127, 128, 129, 300, 2047, 2048, 2049, 4095, 4096, 4097, 8063, 8064,
           8065, 8191, 8192, 9000]
LITERALS = [0, 0, 1, 2, 4, 5, 15, 96, 124, 126, 127, 128, 129, 130, 271]
TOTALS = [33, 128, 129, 130, 255, 256, 257, 1000, 4096, 4225, 8192, 9000, 20000]


def _ext(v):
    return b"\xff" * (v // 255) + bytes([v % 255])


def _block(rng, size):
    """A block of `size` bytes and what it decodes to."""
    out, plain = bytearray(), bytearray()

    def emit(lit, off, ml):
        m = ml - 4
        out.append((min(len(lit), 15) << 4) | (min(m, 15) if ml else 0))
        if len(lit) >= 15:
            out.extend(_ext(len(lit) - 15))
        out.extend(lit)
        plain.extend(lit)
        if ml:
            out.extend(off.to_bytes(2, "little"))
            if m >= 15:
                out.extend(_ext(m - 15))
            pat = bytes(plain[len(plain) - off:])
            plain.extend((pat * (ml // off + 1))[:ml])

    emit(rng.bytes(HEAD), 1, 4)
    while True:
        lit, off, tot = (int(rng.choice(a)) for a in (LITERALS, OFFSETS, TOTALS))
        if len(plain) + max(tot, lit + 4) + 5 > size:
            break
        emit(rng.bytes(lit), off, max(tot - lit, 4))
    emit(rng.bytes(size - len(plain)), 0, 0)
    assert len(plain) == size
    return bytes(out), np.frombuffer(bytes(plain), np.uint8)


@pytest.mark.parametrize("seed", range(6))
def test_long_sequences_decode(fse, seed):
    rng = np.random.default_rng(seed)
    world = fse.World(W, H, seed=1)
    blob = world.checkpoint().tobytes()
    block, plain = _block(rng, 4 * W * H)
    assert len(block) <= 65536, "decoded whole from shared memory"
    # the file: 8 + 9 * 4 bytes, then per section u32 tag, i64 bytes, i32 blocks, per block i32 raw, i32 packed
    at, packed = 44, 0
    while True:
        tag = int.from_bytes(blob[at:at + 4], "little")
        packed = int.from_bytes(blob[at + 20:at + 24], "little")
        if tag == 2:
            break
        assert int.from_bytes(blob[at + 12:at + 16], "little") == 1
        at += 24 + packed
    assert int.from_bytes(blob[at + 4:at + 12], "little") == 4 * W * H
    new = blob[:at + 20] + len(block).to_bytes(4, "little") + block + blob[at + 24 + packed:]
    world.restore(np.frombuffer(new, np.uint8))
    got = world.state()["colour"].view(np.uint8).reshape(-1)
    bad = np.nonzero(got != plain)[0]
    assert len(bad) == 0, "first wrong byte %d of %d" % (bad[0], len(bad))
    world.close()
