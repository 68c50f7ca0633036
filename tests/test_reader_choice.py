"""CPU: which reader a set of files takes (host/io.hpp, device_reader_pays), from
sizes alone, compiled into a small driver."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

DRIVER = r'''
#include <cstdio>
#include <cstdlib>
#include "io.hpp"
int main(int, char** v) {
    std::puts(cdbg::io::device_reader_pays(strtoull(v[1], 0, 10), strtoull(v[2], 0, 10), strtoull(v[3], 0, 10),
                                           (uint32_t)atoi(v[4])) ? "device" : "host");
}
'''


@pytest.fixture(scope="module")
def choice(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("rc")
    (d / "d.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(PKG, "host"), "-o", str(d / "d"), str(d / "d.cpp")],
                   check=True)

    def run(files, size, ratio, threads):
        a = [size, files * size, int(files * size * ratio), threads]
        return subprocess.run([str(d / "d"), *map(str, a)], capture_output=True, text=True, check=True).stdout.strip()

    return run


def test_choice_by_sizes(choice):
    m = 2_400_000
    # sequence: a file may hold about 1/T of the input
    assert choice(64, m, 0.31, 16) == choice(21, m, 0.32, 16) == choice(6, m, 0.32, 4) == "device"
    assert choice(12, m, 0.31, 16) == choice(4, m, 0.31, 4) == choice(1, 100 * m, 0.31, 16) == "host"
    # runs deflate further, and the host inflates them faster
    assert choice(21, m, 0.155, 16) == choice(8, m, 0.155, 4) == choice(100, m, 0.01, 16) == "host"
    assert choice(48, m, 0.155, 16) == choice(12, m, 0.155, 4) == "device"
    # what deflates less counts its bytes
    assert choice(19, m, 0.9, 16) == "host" and choice(21, m, 0.9, 16) == "device"
