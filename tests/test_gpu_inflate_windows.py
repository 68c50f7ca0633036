"""GPU: the device inflater's windowed symbol decoding against zlib, where a
window can go wrong: blocks that end inside a window, runs that stand for more
bytes than a window holds, sources on either side of the window and of the
shared-memory ring, codes longer than the lookup tables, streams back to
back.  The bytes are exact; so is the refusal of a cut stream."""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dna(rng, n):
    return rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), size=n).tobytes()


def _blocks(data, level, size):
    """A gzip stream of many small blocks (a full flush every `size` bytes)."""
    c = zlib.compressobj(level, zlib.DEFLATED, 31)
    out = b"".join(c.compress(data[i:i + size]) + c.flush(zlib.Z_FULL_FLUSH) for i in range(0, len(data), size))
    return out + c.flush()


def _data(kind, rng):
    if kind == "dna":
        return _dna(rng, 150_001)
    if kind == "runs":  # runs from a few bytes to several windows' worth between stretches of sequence
        return b"".join(_dna(rng, int(rng.integers(1, 700))) + b"N" * int(n)
                        for n in np.exp(rng.uniform(0, np.log(40_000), 40)))
    if kind == "near":  # distances 1..40, overlapping copies
        s = bytearray(_dna(rng, 64))
        while len(s) < 60_000:
            d, n = int(rng.integers(1, 41)), int(rng.integers(3, 90))
            for _ in range(n):
                s.append(s[-d])
            s += _dna(rng, int(rng.integers(0, 6)))
        return bytes(s)
    if kind == "far":  # distances on both sides of the ring and up to 32 KiB
        base = _dna(rng, 33_000)
        return base + b"".join(base[o:o + 200] for o in rng.integers(0, 32_000, 300).tolist())
    p = 0.5 ** (np.arange(256) / 9.0)  # codes of up to 15 bits
    return rng.choice(256, size=120_000, p=p / p.sum()).astype(np.uint8).tobytes()


@pytest.mark.parametrize("kind", ["dna", "runs", "near", "far", "skew"])
def test_windows_match_zlib(engine, kind):
    rng = np.random.default_rng(sum(kind.encode()))
    data = _data(kind, rng)
    streams, want = [], []
    for level in (1, 4, 6, 9):
        for cut in (len(data), 4096, 4097, 1):
            d = data[:cut]
            c = zlib.compressobj(level, zlib.DEFLATED, 31)
            streams.append(c.compress(d) + c.flush())
            want.append(d)
        for size in (37, 1000, 5000):
            d = data[:30_000]
            streams.append(_blocks(d, level, size))
            want.append(d)
    got = engine.gunzip(streams, [len(w) for w in want])
    for i, ((st, out), w) in enumerate(zip(got, want)):
        assert st == 0, i
        assert out == w, i


def test_cut_streams_are_refused(engine):
    rng = np.random.default_rng(3)
    data = _dna(rng, 40_000) + b"N" * 30_000 + _dna(rng, 5000)
    c = zlib.compressobj(6, zlib.DEFLATED, 31)
    good = c.compress(data) + c.flush()
    cuts = sorted(set(rng.integers(20, len(good), 60).tolist())) + [len(good) - 1]
    got = engine.gunzip([good[:n] for n in cuts] + [good], [len(data)] * (len(cuts) + 1))
    assert all(st in (1, 2) for st, _ in got[:-1])
    assert got[-1] == (0, data)
