"""GPU: builds at the sizes where a kernel's tiling can go wrong, against the
CPU oracle: k-mer occurrences on the edges of the occurrence blocks (256) and
tiles (2048), records spanning many tiles (homopolymers, short tandem repeats),
tables processed in bucket groups.  Fragments and color sets are exact."""
import os

import numpy as np
import pytest

from cdbg_gpu import native

pytestmark = pytest.mark.gpu


def _dna(rng, n):
    return rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), size=n).tobytes()


def _check(oracle, engine, tmp_path, genomes, k, B):
    """genomes: one list of sequences per color."""
    files = []
    for g, seqs in enumerate(genomes):
        p = os.path.join(str(tmp_path), "g%d.fa" % g)
        with open(p, "wb") as f:
            f.write(b"".join(b">s%d\n%s\n" % (i, s) for i, s in enumerate(seqs)))
        files.append(p)
    lst = os.path.join(str(tmp_path), "files.txt")
    with open(lst, "w") as f:
        f.write("".join(p + "\n" for p in files))
    bd, od = os.path.join(str(tmp_path), "b"), os.path.join(str(tmp_path), "o")
    os.makedirs(bd)
    oracle.phase1(lst, k, B, bucket_dir=bd)
    oracle.phase2(bd, B, k, len(genomes), od)
    flat = [(s, g) for g, seqs in enumerate(genomes) for s in seqs]
    r = engine.build(native.host_batch([s for s, _ in flat], [g for _, g in flat]), k, B, len(genomes))
    frag, cs = os.path.join(str(tmp_path), "f.bin"), os.path.join(str(tmp_path), "c.sets")
    want = open(os.path.join(od, "frag_unitigs.bin"), "rb").read()
    assert native.result_frag_bytes(r) == want
    engine.build_files(files, k, B, frag, cs)
    assert open(frag, "rb").read() == want
    assert open(cs, "rb").read() == open(os.path.join(od, "out.color_sets"), "rb").read()


@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 2047, 2048, 2049, 6143])
def test_occurrence_tile_edges(oracle, engine, tmp_path, k, n):
    rng = np.random.default_rng(n + k)
    s = _dna(rng, n + k - 1)
    t = bytearray(s)
    t[len(t) // 2] = ord("A") if t[len(t) // 2] != ord("A") else ord("C")
    _check(oracle, engine, tmp_path, [[s], [bytes(t), s[: k + 3]]], k, 1)


@pytest.mark.parametrize("group_mb", [0, 1])
@pytest.mark.parametrize("k", [31, 63])
def test_long_records_and_groups(oracle, tmp_path, k, group_mb):
    rng = np.random.default_rng(7 + k)
    a, b = _dna(rng, 30_000), _dna(rng, 20_011)
    g0 = [a, b"A" * 5000, b[:300] + b"AC" * 2600 + b[300:]]
    g1 = [a[:9000] + b"T" * 4097 + a[9000:], b]
    g2 = [b"G" * (k + 255), a[100:131 + k], (b[:211] * 30)[:5200]]
    with native.Engine(0) as e:
        e.set_tuning(table_group_mb=group_mb)
        _check(oracle, e, tmp_path, [g0, g1, g2], k, 37)


@pytest.mark.parametrize("k", [21, 31, 63])
@pytest.mark.parametrize("buckets,n", [(1, 300_000), (1, 250_000), (3, 900_000), (64, 200_000)])
def test_neighbour_lookups_by_bucket_size(oracle, engine, tmp_path, k, buckets, n):
    """Extension masks with the presence filter (buckets of up to 2^18
    occurrences), split buckets among them, and without; branches, repeats and
    self-neighbours."""
    rng = np.random.default_rng(n + k + buckets)
    a = _dna(rng, n)
    b = bytearray(a[: n // 3])
    for i in rng.integers(0, len(b), len(b) // 60).tolist():
        b[i] = b"ACGT"[int(rng.integers(0, 4))]
    _check(oracle, engine, tmp_path, [[a, b"A" * (2 * k), b"ACGT" * k], [bytes(b), a[-2 * k:] + a[:2 * k]]], k, buckets)


@pytest.mark.parametrize("shift", [0, 1, 7, 16])
@pytest.mark.parametrize("tail", [0, 1, 15, 31, 47])
def test_device_input_alignment(oracle, engine, tmp_path, shift, tail):
    """Sequences in HBM at any byte offset, ending at any distance from an
    aligned address, in either case, with runs of other characters."""
    import torch
    k, B = 31, 16
    rng = np.random.default_rng(shift * 50 + tail)
    s = [_dna(rng, 4000 + tail), _dna(rng, 31).lower(), b"ACGTN" + _dna(rng, 333) + b"-" * 40 + _dna(rng, 64), b"NN",
         _dna(rng, 97)]
    data = np.frombuffer(b"".join(s), dtype=np.uint8)
    off = np.zeros(len(s) + 1, dtype=np.int64)
    off[1:] = np.cumsum([len(x) for x in s])
    buf = torch.empty(shift + len(data), dtype=torch.uint8, device="cuda")
    buf[shift:] = torch.from_numpy(data.copy())
    d_off, d_col = torch.from_numpy(off).cuda(), torch.tensor([0, 0, 1, 1, 1], dtype=torch.int32).cuda()
    torch.cuda.synchronize()
    b = native.SeqBatch(buf.data_ptr() + shift, len(data), d_off.data_ptr(), d_col.data_ptr(), len(s), 1)
    want = engine.build(native.host_batch(s, [0, 0, 1, 1, 1]), k, B, 2)
    want = native.result_frag_bytes(want)
    assert native.result_frag_bytes(engine.build(b, k, B, 2)) == want
    _check(oracle, engine, tmp_path, [s[:2], s[2:]], k, B)


@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("unit", [33, 64, 65, 131, 700])
def test_cycles_and_broken_chains(oracle, engine, tmp_path, k, unit):
    """Chains that are cycles, of up to 64 k-mers and more, chains broken by
    contig ends inside a bucket, and chains that are one fragment."""
    rng = np.random.default_rng(unit + k)
    u, a, b = _dna(rng, unit), _dna(rng, 500), _dna(rng, 900)
    g0 = [u * (3 + 2 * k // unit), a, b[:400]]
    g1 = [a[100:300], b[300:], b[200:260 + k]]
    g2 = [a[:k], a[-k:], a[200:200 + k + 1], u + u[: k + 2]]
    for B in (1, 5):
        d = tmp_path / str(B)
        d.mkdir()
        _check(oracle, engine, d, [g0, g1, g2], k, B)


@pytest.mark.parametrize("colors", [1, 2, 3, 31, 255, 256, 257, 512, 513, 1100])
def test_color_set_encoding(oracle, engine, tmp_path, colors):
    """Color sets of every form (sparse, plain bitmap, complement, all) at the
    widths where the encoder's lane groups change, some classes new in a later
    batch."""
    k, B = 31, 8
    rng = np.random.default_rng(colors)
    blocks = [_dna(rng, 90 + 7 * i) for i in range(9)]
    share = [1.0, 0.95, 0.8, 0.74, 0.5, 0.26, 0.2, 0.05, 0.0]
    genomes = [[b for b, p in zip(blocks, share) if rng.random() < p] + [_dna(rng, 40)] for _ in range(colors)]
    genomes[-1].append(blocks[-1])
    _check(oracle, engine, tmp_path, genomes, k, B)
    flat = [(s, g) for g, seqs in enumerate(genomes) for s in seqs]
    hb = native.host_batch([s for s, _ in flat], [g for _, g in flat])

    def out(**kw):
        r = engine.build(hb, k, B, colors, **kw)
        return native.result_frag_bytes(r), native.result_class_words(r).tobytes(), native.result_class_offsets(r).tobytes()

    assert out(batch_occ=64) == out()


@pytest.mark.parametrize("colors", [2, 31, 255, 256, 257, 512, 513])
def test_unions_of_many_records(oracle, engine, tmp_path, colors):
    """K-mers in 2 to 150 records each (one block between different flanks), of
    few and many colors, at the widths where the unions' lane groups change and
    around the counts where the whole warp takes a union's rest."""
    k, B = 31, 2
    rng = np.random.default_rng(1000 + colors)
    genomes = [[] for _ in range(colors)]
    for n in (2, 8, 9, 31, 32, 33, 64, 65, 150):
        block = _dna(rng, k + 2)
        for i in range(n):
            seq = _dna(rng, 6) + block + _dna(rng, 6)
            few = int(rng.integers(1, 4)) if i % 3 else int(rng.integers(1, colors + 1))
            for g in rng.choice(colors, size=min(few, colors), replace=False):
                genomes[g].append(seq)
    for g in genomes:
        g.append(_dna(rng, 40))
    _check(oracle, engine, tmp_path, genomes, k, B)
    flat = [(s, g) for g, seqs in enumerate(genomes) for s in seqs]
    hb = native.host_batch([s for s, _ in flat], [g for _, g in flat])

    def out():
        r = engine.build(hb, k, B, colors)
        return native.result_frag_bytes(r), native.result_class_words(r).tobytes(), native.result_class_offsets(r).tobytes()

    want = out()
    try:
        for heavy in (1, 20, 100000):
            engine.set_tuning(heavy_colors=heavy)
            assert out() == want
    finally:
        engine.set_tuning()


@pytest.mark.parametrize("n", [440_000, 470_000, 600_000])
def test_neighbour_lookups_of_large_buckets_of_long_kmers(oracle, engine, tmp_path, n):
    """128-bit k-mers on both sides of the largest bucket that gets the wide
    presence filter (7 * 2^16 occurrences)."""
    k = 63
    rng = np.random.default_rng(n)
    a = _dna(rng, n)
    b = bytearray(a[:6000])
    for i in rng.integers(0, len(b), 90).tolist():
        b[i] = b"ACGT"[int(rng.integers(0, 4))]
    _check(oracle, engine, tmp_path, [[a, b"A" * (2 * k), b"ACGT" * k], [bytes(b), a[-2 * k:] + a[:2 * k]]], k, 1)
