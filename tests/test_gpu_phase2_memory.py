"""GPU: drop-in phase 2 hands its fragments over batch by batch: it holds the
same device memory, at its peak and afterwards, with and without a (generous)
memory cap, and writes the same files."""
import os

import pytest

from cdbg_gpu import native, synth

pytestmark = pytest.mark.gpu


def test_phase2_holds_one_batch(tmp_path):
    k, B, n = 31, 256, 12
    p = synth.make_params(seed=11, len_min=3_000_000, len_max=3_000_000, div_min=0.02, div_max=0.03)
    lst = synth.write_fasta(p, n, str(tmp_path / "in"))
    files = [x.strip() for x in open(lst) if x.strip()]
    bd = tmp_path / "b"
    bd.mkdir()
    with native.Engine(0) as e:
        _, unc = e.phase1(files, k, B, str(bd))
    used, out = {}, {}
    for cap in (0, 64 << 30):
        with native.Engine(0) as e:
            e.set_memory_limit(cap)
            frag, sets = tmp_path / ("f%d" % (cap > 0)), tmp_path / ("s%d" % (cap > 0))
            e.phase2(str(bd), B, k, n, str(frag), str(sets), batch_occ=1 << 20, pass_bytes=int(sum(unc)) + 1)
            used[cap] = e.memory()
            out[cap] = (frag.read_bytes(), sets.read_bytes())
    a, b = out.values()
    assert a == b
    assert used[0] == used[64 << 30]
    assert os.path.getsize(tmp_path / "f0") > 100 << 20
