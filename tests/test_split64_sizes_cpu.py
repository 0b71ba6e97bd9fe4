"""The digit splits' workspace (lywell_gb300/csrc/mlf_split64.h): after any two
products of 2 to 64 columns on one context, both buffers hold what the second
writes.  No GPU: the header is compiled with the host C++ compiler.

What a product of n columns writes: parts [split][column][unknown], the split
worked out here, and exponents, some per unknown and some per column (of a box)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SRC = r"""
#include <cstdio>
#include "mlf_split64.h"
using namespace mlf;
int main() {
    const int nsm = 152;
    long pairs = 0, bad = 0;
    for (int dense = 0; dense < 2; ++dense)
        for (int tiles = 1; tiles <= 2000; ++tiles) {
            const int N = 57 * tiles, boxes = (tiles + 3) / 4;   // any; both sides scale with them
            const size_t fixed = 2 * (size_t)N + (dense ? (N + 31) / 32 : 0), per_col = dense ? 1 : boxes;
            OzSizes need[65];
            for (int n = 2; n <= 64; ++n) need[n] = oz_sizes(tiles, nsm, N, dense, fixed, per_col, n);
            for (int a = 2; a <= 64; ++a)
                for (int b = 2; b <= 64; ++b, ++pairs) {
                    OzSizes cap = need[a];
                    if (oz_short(cap, need[b])) {
                        cap.sums = std::max(cap.sums, need[b].sums);
                        cap.exps = std::max(cap.exps, need[b].exps);
                    }
                    const int ctas = tiles * ((b + 11) / 12);
                    const int split = std::max(1, std::min(dense ? 8 : 4, (4 * nsm + ctas - 1) / ctas));
                    bad += cap.sums < (size_t)split * b * N || cap.exps < fixed + per_col * b;
                }
        }
    std::printf("%ld %ld\n", pairs, bad);
    return 0;
}
"""


def test_both_buffers_cover_the_second_product(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src = tmp_path / "t.cpp"
    src.write_text(SRC)
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "lywell_gb300", "csrc"), str(src), "-o",
                    str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split()
    assert out == [str(2 * 2000 * 63 * 63), "0"]
