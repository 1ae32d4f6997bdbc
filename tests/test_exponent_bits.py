"""The singularity test of the pivots (croma_bits.cuh) on the host, compiled so
that signed overflow ends the program: over the whole range of both operands it
is the comparison of the exponents that its comment states, and nothing in it
overflows."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include "croma_bits.cuh"
int main()
{
    // n = 2^e (1 + f), th = 2^k (1 + f'): the test is n 2^996 < th on the high words
    const double frac[3] = {1.0, 1.25, 1.9999990463256836};   // exact in the high word
    for (int e = -1022; e <= 1023; e++)
        for (int k = -1022; k <= 1023; k += 7)
            for (int s = 0; s < 4; s++)
                for (double fn : frac) {
                    const double n = std::ldexp(s & 1 ? -fn : fn, e), th = std::ldexp(s & 2 ? -1.5 : 1.5, k);
                    const bool want = e + 996 < k || (e + 996 == k && fn < 1.5);
                    if (croma::continuant_singular(n, th) != want) {
                        std::printf("e %d k %d fraction %g\n", e, k, fn);
                        return 1;
                    }
                }
    const double inf = INFINITY, nan = NAN;
    if (!croma::continuant_singular(0.0, 1.0) || croma::continuant_singular(inf, inf) || croma::continuant_singular(nan, 1.0))
        return 2;
    return 0;
}
"""


def test_singularity_test_does_not_overflow(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "bits.cpp", tmp_path / "bits"
    src.write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover=all",
                    "-I" + os.path.join(ROOT, "croma-fp_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
