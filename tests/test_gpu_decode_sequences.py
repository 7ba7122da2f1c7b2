"""The device's LZ4 decoder on blocks whose sequences take every form: zero to hundreds of
literals, matches from 4 bytes to past the one-step copy's 128, offsets from 1 to past its
ring, matches that overlap themselves and that read the sequence's own literals, and the
same blocks with bytes changed. Both decode to, or are refused at, what the oracle does.
"""
import numpy as np
import pytest

from pack_cases import HEADER, SRC1, sample_world, split_blocks

pytestmark = pytest.mark.gpu

W, H = 384, 256


def _records(rng):
    """One tile's 12-byte records: runs of one record, copies from near and far, noise."""
    n = SRC1 // 12
    out = np.zeros((n, 12), np.uint8)
    i = 0
    while i < n:
        k = int(rng.integers(1, 60))
        k = min(k, n - i)
        kind = rng.integers(0, 5)
        if kind == 0:  # bytes of zero: any offset matches
            pass
        elif kind == 1 and i:  # an earlier stretch again, also one past the ring
            d = int(rng.integers(1, min(i, 1500) + 1))
            for j in range(k):
                out[i + j] = out[i + j - d]
        else:  # one record repeated, or new ones
            r = np.zeros(12, np.uint8)
            r[0] = rng.integers(0, 6)
            r[4:10] = rng.integers(0, 256, 6)
            out[i:i + k] = r
            if kind == 2:
                k = min(k, 3)
                out[i:i + k, 4:10] = rng.integers(0, 256, (k, 6))
        i += k
    return out.tobytes()


def _ext(v):
    b = bytearray()
    while v >= 255:
        b.append(255)
        v -= 255
    b.append(v)
    return bytes(b)


def _encode(rng, data):
    """An LZ4 block of `data` with matches cut and chosen at random."""
    n, out, p, anchor = len(data), bytearray(), 0, 0

    def emit(a, b, off, ml):
        ll, m = b - a, ml - 4
        out.append((min(ll, 15) << 4) | (min(m, 15) if ml else 0))
        if ll >= 15:
            out.extend(_ext(ll - 15))
        out.extend(data[a:b])
        if ml:
            out.extend(off.to_bytes(2, "little"))
            if m >= 15:
                out.extend(_ext(m - 15))

    caps = [4, 5, 18, 19, 31, 32, 33, 64, 96, 124, 127, 128, 129, 160, 272, 273, 274, 275, 600, 1500]
    while p < n - 12:
        best = None
        for d in rng.permutation([1, 2, 3, 5, 7, 12, 24, 36, 127, 128, 129, 8064, 8065, 8076, 8192, 8208,
                                  12 * int(rng.integers(1, 1500)), int(rng.integers(1, 400))]):
            d = int(d)
            if d > p or data[p:p + 4] != data[p - d:p - d + 4]:
                continue
            cap = min(int(rng.choice(caps)), n - 5 - p)
            ml = 4
            while ml < cap and data[p + ml] == data[p + ml - d]:
                ml += 1
            best = (d, ml)
            break
        if best is None or rng.random() < 0.02:
            p += 1
            continue
        emit(anchor, p, best[0], best[1])
        p += best[1]
        anchor = p
        if rng.random() < 0.2:  # literals although a match would do
            p += int(rng.choice([1, 2, 3, 4, 5, 14, 15, 16]))
    emit(anchor, n, 0, 0)
    return bytes(out)


@pytest.mark.parametrize("seed", [0, 1])
def test_sequences_decode_as_the_oracle(fse, oracle_mod, seed):
    oracle_mod.Oracle().reset_materials()
    rng = np.random.default_rng(seed)
    data, offs = sample_world(oracle_mod, W, H, 4).pack(0)
    files = []
    for k in range(len(offs) - 1):
        hd, _, c2 = split_blocks(data, offs, k)
        block = _encode(rng, _records(rng))
        assert len(block) < 64 * 1024, "decoded whole from shared memory"
        head = bytearray(data[offs[k]:offs[k] + HEADER].tobytes())
        head[5:9] = len(block).to_bytes(4, "little")
        files.append((bytes(head), block, bytes(c2)))

    def load(parts):
        raw = [b"".join(p) for p in parts]
        at = np.cumsum([0] + [len(r) for r in raw]).astype(np.int64)
        buf = np.frombuffer(b"".join(raw), np.uint8).copy()
        ow = oracle_mod.OracleWorld(W, H, 128, 3, 1)
        rc, _ = ow.unpack(buf, at)
        world = fse.World(W, H, seed=1, temperature=True)
        if rc == 0:
            world.unpack(buf, at)
        else:
            with pytest.raises(fse.FseError):
                world.unpack(buf, at)
        got, want = world.state(), ow.state()
        for key in ("id", "colour", "scalar"):
            assert np.array_equal(got[key], want[key]), (key, rc)
        world.close()
        return rc

    assert load(files) == 0
    refused = 0
    for _ in range(24):
        k = int(rng.integers(0, len(files)))
        block = bytearray(files[k][1])
        for at in rng.integers(0, len(block), 2):
            block[at] = rng.choice([0, 1, 0x0F, 0xF0, 0xFF, int(rng.integers(0, 256))])
        refused += load(files[:k] + [(files[k][0], bytes(block), files[k][2])] + files[k + 1:]) != 0
    assert refused > 0
