"""The fragment file may be anything that can be written: a new or an existing
file, a FIFO, a device.  CPU: the ranged output file (host/io.hpp, range_file)
through a small driver.  GPU: cdbg_gpu_phase2 to a FIFO and to /dev/null."""
import os
import shutil
import stat
import subprocess
import threading

import numpy as np
import pytest

from conftest import PKG

DRIVER = r'''
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <vector>
#include "io.hpp"
// path, total bytes, bytes per range, descending
int main(int, char** v) {
    const uint64_t n = strtoull(v[2], 0, 10), step = strtoull(v[3], 0, 10);
    std::vector<uint8_t> d(n);
    for (uint64_t i = 0; i < n; ++i) d[i] = (uint8_t)(i * 131 + (i >> 8));
    try {
        cdbg::io::range_file f(v[1]);
        const uint64_t m = (n + step - 1) / step;
        for (uint64_t j = 0; j < m; ++j) {
            const uint64_t x = (v[4][0] == '1' ? m - 1 - j : j) * step;
            f.write(d.data() + x, x, std::min(step, n - x), 4);
        }
        f.finish(n);
    } catch (std::exception const& e) {
        std::puts(e.what());
        return 1;
    }
    return 0;
}
'''


def _bytes(n):
    i = np.arange(n, dtype=np.uint64)
    return ((i * np.uint64(131) + (i >> np.uint64(8))) & np.uint64(255)).astype(np.uint8).tobytes()


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("rf")
    src, exe = d / "d.cpp", d / "d"
    src.write_text("#include <algorithm>\n" + DRIVER)
    host = os.path.join(PKG, "host")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", host, "-o", str(exe), str(src), os.path.join(host, "io.cpp"), "-lz",
                    "-l:liblz4.so.1", "-lpthread"], check=True)
    return str(exe)


def _fifo_reader(path):
    got = []

    def read():
        with open(path, "rb") as f:
            got.append(f.read())

    t = threading.Thread(target=read)
    t.start()
    return t, got


def _run(driver, path, n, step, descending=False):
    return subprocess.run([driver, str(path), str(n), str(step), "1" if descending else "0"], capture_output=True,
                          text=True, timeout=60)


@pytest.mark.parametrize("base", ["tmp", "shm"])
@pytest.mark.parametrize("descending", [False, True])
@pytest.mark.parametrize("n,step", [(1, 7), (100_000, 4096), (20 << 20, 9 << 20)])
def test_regular_files(driver, tmp_path, base, descending, n, step):
    if base == "shm" and not os.path.isdir("/dev/shm"):
        pytest.skip("no /dev/shm")
    path = tmp_path / "f" if base == "tmp" else "/dev/shm/cdbg_range_%d" % os.getpid()
    try:
        with open(path, "wb") as f:  # an older, longer file
            f.write(b"x" * (n + 1000))
        r = _run(driver, path, n, step, descending)
        assert r.returncode == 0, r.stdout
        assert open(path, "rb").read() == _bytes(n)
    finally:
        os.unlink(path)


def test_a_new_file_has_the_usual_mode(driver, tmp_path):
    old = os.umask(0o027)
    try:
        assert _run(driver, tmp_path / "f", 10, 10).returncode == 0
    finally:
        os.umask(old)
    assert stat.S_IMODE(os.stat(tmp_path / "f").st_mode) == 0o640


@pytest.mark.parametrize("n,step", [(10, 3), (300_000, 70_001), (9 << 20, 9 << 20)])
def test_fifo(driver, tmp_path, n, step):
    path = str(tmp_path / "p")
    os.mkfifo(path)
    t, got = _fifo_reader(path)
    r = _run(driver, path, n, step)
    t.join(60)
    assert r.returncode == 0, r.stdout
    assert got == [_bytes(n)]


def test_fifo_refuses_to_go_back(driver, tmp_path):
    path = str(tmp_path / "p")
    os.mkfifo(path)
    t, _ = _fifo_reader(path)
    r = _run(driver, path, 100, 30, descending=True)
    t.join(60)
    assert r.returncode == 1 and "in order" in r.stdout


def test_device(driver):
    r = _run(driver, "/dev/null", 1 << 20, 70_001)
    assert r.returncode == 0, r.stdout
    r = _run(driver, "/dev/full", 1 << 20, 70_001)
    assert r.returncode == 1 and "short write" in r.stdout


def test_unwritable_path(driver, tmp_path):
    r = _run(driver, tmp_path / "none" / "f", 10, 10)
    assert r.returncode == 1 and "cannot open" in r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("target", ["fifo", "null"])
@pytest.mark.parametrize("passes", [1, 3])
def test_phase2_to_anything_writable(engine, tmp_path, target, passes):
    from cdbg_gpu import synth
    k, B, n = 31, 24, 3
    p = synth.make_params(seed=5, len_min=20000, len_max=20000, div_min=0.005, div_max=0.01)
    lst = synth.write_fasta(p, n, str(tmp_path / "in"))
    files = [x.strip() for x in open(lst) if x.strip()]
    bd = tmp_path / "b"
    bd.mkdir()
    _, unc = engine.phase1(files, k, B, str(bd))
    pass_bytes = int(sum(unc)) // passes
    ref, sets = tmp_path / "ref.bin", tmp_path / "ref.sets"
    s = engine.phase2(str(bd), B, k, n, str(ref), str(sets), pass_bytes=pass_bytes)
    assert s.n_passes >= passes
    path, out = ("/dev/null", None) if target == "null" else (str(tmp_path / "p"), None)
    if target == "fifo":
        os.mkfifo(path)
        t, out = _fifo_reader(path)
    s2 = engine.phase2(str(bd), B, k, n, path, str(tmp_path / "s2"), pass_bytes=pass_bytes, delete_consumed=True)
    if target == "fifo":
        t.join(60)
        assert out == [ref.read_bytes()]
    assert s2.n_fragments == s.n_fragments
    assert (tmp_path / "s2").read_bytes() == sets.read_bytes()
