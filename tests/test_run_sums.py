"""CPU: the sums the run table carries by look-back (csrc/run_sums.hpp) keep
their width: at the largest number of runs an input may have, each sum -- runs,
stream words, minimizer tiles -- stays below the status word's flag bits, so the
index of a run is its own whatever the input."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

DRIVER = r'''
#include <cstdio>
#include <initializer_list>
#include "run_sums.hpp"
using namespace cdbg;
int main() {
    const unsigned __int128 cap = (((unsigned __int128)1) << LOOKBACK_SUM_BITS) - 1;
    unsigned bad = 0, n = 0;
    for (uint32_t k : {2u, 3u, 21u, 31u, 32u, 33u, 63u})
        for (uint32_t tt : {1024u, 2048u, 4096u})
            for (uint64_t l : {(uint64_t)0, (uint64_t)k - 1, (uint64_t)k, (uint64_t)k + 1, (uint64_t)100,
                               (uint64_t)4096 + k, (uint64_t)1 << 31, MAX_RUN_BASES}) {
                const run_sums a = run_adds(l, k, tt);
                const bool keep = l >= k;
                bad += a.runs != (keep ? 1u : 0u);
                bad += a.words != (keep ? (l + 31) / 32 : 0);
                bad += a.tiles != (keep ? (l - k + 1) / tt + 1 : 0);  // (k-1)-mers: l - k + 2
                for (uint64_t runs : {(uint64_t)1, ((uint64_t)1 << 30) - 1, (uint64_t)1 << 30, (uint64_t)1 << 31,
                                      MAX_RAW_RUNS}) {
                    for (uint64_t v : {a.runs, a.words, a.tiles}) bad += (unsigned __int128)v * runs > cap;
                    n += 3;
                }
            }
    std::printf("%u checked, %u bad\n", n, bad);
    return bad != 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_sums_of_the_most_runs(tmp_path):
    src, exe = tmp_path / "d.cpp", tmp_path / "d"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(PKG, "csrc"), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.strip().endswith(" 0 bad")


@pytest.mark.gpu
@pytest.mark.parametrize("k", [21, 31])
@pytest.mark.parametrize("runs", [1, 2047, 2048, 2049, 4100, 70_000])
def test_run_table_tiles(oracle, engine, tmp_path, k, runs):
    """Runs shorter and longer than k around the tiles (2048 runs) of the run
    table's pass, the last one kept and not, against the oracle."""
    import numpy as np
    from cdbg_gpu import native
    rng = np.random.default_rng(runs + k)
    for last in (k - 1, k, 3 * k):
        lens = rng.integers(1, 2 * k + 2, runs)
        lens[rng.integers(0, runs, 3)] = 5000
        lens[-1] = last
        lens[0] = max(int(lens[0]), k) if runs > 1 else last
        dna = rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), size=int(lens.sum())).tobytes()
        cut = np.concatenate([[0], np.cumsum(lens)])
        seq = b"N".join(dna[a:b] for a, b in zip(cut[:-1].tolist(), cut[1:].tolist()))
        d = tmp_path / ("l%d" % last)
        d.mkdir()
        fa, lst = d / "a.fa", d / "files.txt"
        fa.write_bytes(b">s\n" + seq + b"\n")
        lst.write_text(str(fa) + "\n")
        bd, od = d / "b", d / "o"
        bd.mkdir()
        oracle.phase1(str(lst), k, 16, bucket_dir=str(bd))
        oracle.phase2(str(bd), 16, k, 1, str(od))
        r = engine.build(native.host_batch([seq], [0]), k, 16, 1)
        assert native.result_frag_bytes(r) == (od / "frag_unitigs.bin").read_bytes(), (last, runs)
