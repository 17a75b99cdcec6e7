"""The bound on the cells a placed disk meets (it sizes the cover lists) holds
for boxes a rounding error short of a whole number of cells."""
import os
import subprocess

import pytest

from godar_b200 import build

MAIN = r"""
#include <cstdio>
#include <random>
#include "cover.h"
using namespace godar;
int main() {
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    long long bad = 0, n = 0, wide = 0;
    for (int nc : {1, 2, 3, 7, 100, 1023, 8192})
        for (int k = 0; k < 4000; k++) {
            const double L = 100.0 + 1e5 * U(g), cw = L / nc;
            // a box of m cells, up to two rounding errors narrower or wider
            const int m = 1 + (int)(U(g) * 4.0);
            double r = 0.5 * m * cw;
            for (int s = (int)(U(g) * 5.0) - 2; s != 0; s += s < 0 ? 1 : -1) r = std::nextafter(r, s < 0 ? 0.0 : 1e9);
            for (int q = 0; q < 8; q++) {
                // centres that put an edge of the box on or beside a cell's edge
                double x = r + cw * (int)(U(g) * nc);
                if (q & 1) x = L - r;
                for (int s = q / 2; s > 0; s--) x = std::nextafter(x, (q & 2) ? 0.0 : 1e9);
                for (int per = 0; per < 2; per++) {
                    int a, b;
                    cell_span(x - r, x + r, cw, nc, per, a, b);
                    n++;
                    wide += b - a + 1 > std::floor(2.0 * r / cw) + 2.0;
                    bad += b - a + 1 > cells_met(r, cw, nc);
                }
            }
        }
    std::printf("%lld %lld %lld\n", n, wide, bad);
    return 0;
}
"""


def test_no_disk_meets_more_cells_than_the_bound(tmp_path):
    src, exe = tmp_path / "cover.cpp", tmp_path / "cover"
    src.write_text(MAIN)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.NVCC)), "include")
    subprocess.check_call(["g++", "-O1", "-ffp-contract=off", "-std=c++17", "-I", build.CSRC, "-I", cuda, str(src),
                           "-o", str(exe)])
    n, wide, bad = map(int, subprocess.check_output([str(exe)], text=True).split())
    assert n > 0
    assert wide > 0          # boxes beyond the width's own count do occur
    assert bad == 0
