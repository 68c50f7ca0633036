"""The choice between the forms of the extension-mask pass (csrc/ext_plan.hpp).
CPU: the rule itself, compiled into a small driver -- full groups go through the
filter, groups of few buckets and buckets too large for a filter go flat, and
every bucket has blocks.  GPU: builds whose buckets take the filter, the wide
filter and no filter give the same fragments and color sets."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG

DRIVER = r'''
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "ext_plan.hpp"
using namespace cdbg;
// wide keys, then "count size" pairs; prints buckets per form, blocks of the filters
// and occurrences of a flat block
int main(int argc, char** v) {
    std::vector<uint64_t> off{12345};
    for (int i = 2; i + 1 < argc; i += 2)
        for (long j = atol(v[i]); j; --j) off.push_back(off.back() + strtoull(v[i + 1], 0, 10));
    const uint64_t tn = off.back() - off[0];
    const ext_plan p(v[1][0] == '1', tn);
    const uint64_t cut = p.cut(off.data(), off.size() - 1);
    uint64_t nb[3] = {}, bl[2] = {};
    for (size_t b = 0; b + 1 < off.size(); ++b) {
        const uint64_t n = off[b + 1] - off[b];
        if (!n) continue;
        const int f = p.form(n, cut);
        nb[f]++;
        if (f != EXT_FLAT) bl[f] += p.parts(n);
        if (!p.parts(n)) return 1;
        if (f != EXT_FLAT && n > p.wide_occ) return 2;
        if (f == EXT_WIDE && v[1][0] == '0') return 3;
    }
    std::printf("%llu %llu %llu %llu %llu %llu\n", (unsigned long long)nb[0], (unsigned long long)nb[1],
                (unsigned long long)nb[2], (unsigned long long)bl[0], (unsigned long long)bl[1], (unsigned long long)p.flat_occ(tn));
    return 0;
}
'''


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("ext")
    (d / "d.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(PKG, "csrc"), "-o", str(d / "d"), str(d / "d.cpp")],
                   check=True)

    def run(wide, *sizes):
        r = subprocess.run([str(d / "d"), "1" if wide else "0", *map(str, sizes)], capture_output=True, text=True)
        assert r.returncode == 0, r.returncode
        return [int(x) for x in r.stdout.split()]

    return run


@pytest.mark.parametrize("wide", [False, True])
def test_forms_by_group(plan, wide):
    assert plan(wide) == [0] * 5 + [256]
    assert plan(wide, 5, 0) == [0] * 5 + [256]
    assert plan(wide, 64, 600)[:3] == [64, 0, 0]           # a toy build: one launch, no probes to spare
    assert plan(wide, 1024, 49_000)[:3] == [1024, 0, 0]    # full groups
    assert plan(wide, 4096, 200_000)[:3] == [4096, 0, 0]
    assert plan(wide, 4096, 262_144)[:3] == [4096, 0, 0]   # the largest with a filter
    assert plan(wide, 4096, 262_145)[:3] == ([0, 4096, 0] if wide else [0, 0, 4096])
    assert plan(wide, 4096, 7 << 16)[:3] == ([0, 4096, 0] if wide else [0, 0, 4096])
    assert plan(wide, 4096, (7 << 16) + 1)[:3] == [0, 0, 4096]
    for n in (20_000, 100_000, 250_000, 400_000):          # one bucket, a few: the whole chip probes
        assert plan(wide, 1, max(n, 50_000))[2] == 1
        assert plan(wide, 4, max(n, 50_000))[2] == 4
    assert plan(wide, 4096, 100_000, 3, 5_000_000)[:3] == [4096, 0, 3]
    for n in (1, 30, 120):                                 # blocks cost more than what small buckets hold
        assert plan(wide, 16_384, n)[2] == 16_384
    assert plan(wide, 60_000, 40, 900, 60_000)[:3] in ([900, 0, 60_000], [60_900, 0, 0])
    # flat blocks of one round of 256 where the chip is idle, never more than the kernel's lists hold
    assert plan(wide, 1, 60_000)[5] == 256
    assert plan(wide, 4096, 1_000_000)[5] == (512 if wide else 1024)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("bases,buckets", [(900, 7), (40_000, 1), (40_000, 1500), (60_000, 20_000), (1_500_000, 30_000),
                                           (1_500_000, 400)])
def test_small_buckets(oracle, engine, tmp_path, k, bases, buckets):
    """Flat blocks over many small buckets, empty ones among them, and large ones
    beside them, against the CPU oracle."""
    from test_gpu_edges import _check
    rng = np.random.default_rng(bases + buckets + k)
    dna = lambda n: rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), size=n).tobytes()  # noqa: E731
    a = dna(bases)
    b = bytearray(a[: bases // 2])
    for i in rng.integers(0, len(b), len(b) // 70).tolist():
        b[i] = b"ACGT"[int(rng.integers(0, 4))]
    low = b"A" * (bases // 8) + b"AC" * (bases // 16) + dna(50)  # a few buckets hold an eighth of all
    _check(oracle, engine, tmp_path, [[a, low], [bytes(b), a[-2 * k:] + a[: 2 * k]]], k, buckets)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [31, 45, 63])
@pytest.mark.parametrize("size", [12_000, 120_000, 255_000, 300_000])
def test_forms_give_the_same(oracle, engine, k, size):
    """Enough buckets that those of `size` occurrences take a filter (the wide one
    past 2^18 at k > 31), against the same buckets in groups of their own, which
    go flat."""
    from cdbg_gpu import native
    B = 12_000_000 // size if size < 100_000 else 90
    rng = np.random.default_rng(size + k)
    a = rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), size=B * size)
    b = a[: len(a) // 20].copy()
    at = rng.integers(0, len(b), len(b) // 40)
    b[at] = rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), size=len(at))
    seqs = [a.tobytes(), b.tobytes(), b"A" * (2 * k) + b"N" + b"ACGT" * k, a[-2 * k:].tobytes() + a[: 2 * k].tobytes()]
    hb = native.host_batch(seqs, [0, 1, 1, 2])

    def out():
        r = engine.build(hb, k, B, 3)
        return native.result_frag_bytes(r), native.result_class_words(r).tobytes(), native.result_class_offsets(r).tobytes()

    want = out()
    try:
        engine.set_tuning(table_group_mb=1)
        assert out() == want
    finally:
        engine.set_tuning()
