"""Kernel attributes are set once on every device (croma_once.cuh), compiled on
the host with made-up devices: each has its own first call, a failed one is made
again, threads agree; and no launch keeps one result for the whole process."""
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "croma-fp_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "croma_once.cuh"
static int calls[80];
int main()
{
    static croma::OncePerDevice once;
    auto set = [](int dev, int result) { return once(dev, [=] { calls[dev]++; return result; }); };
    if (set(0, 0) || set(0, 5) || calls[0] != 1) return 1;          // kept on device 0
    if (set(1, 7) != 7 || set(1, 0) || set(1, 9) || calls[1] != 2) return 2;   // its own on device 1, tried again
    if (set(79, 0) || set(79, 3) != 3 || calls[79] != 2) return 3;  // beyond the table: always
    std::vector<std::thread> pool;
    std::atomic<int> bad{0}, ran{0};
    for (int t = 0; t < 16; t++)
        pool.emplace_back([&, t] {
            for (int d = 2; d < 60; d++)
                if (once(d, [&] { ran++; return 0; })) bad++;
        });
    for (auto &t : pool) t.join();
    if (bad || ran < 58 || ran > 58 * 16) return 4;
    const int before = ran;
    for (int d = 2; d < 60; d++) once(d, [&] { ran++; return 0; });
    return ran == before ? 0 : 5;
}
"""


def test_once_on_each_device(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0


def test_no_launch_keeps_an_attribute_for_the_process():
    """A function-local static initialised by cudaFuncSetAttribute holds the first device's result for all."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                assert not re.search(r"static\s+const\s+cudaError_t\s+\w+\s*=\s*cudaFuncSetAttribute", f.read()), name
