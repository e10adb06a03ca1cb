"""Interpolation weights and cells of feet (csrc/af_exact.cuh) against native
binary64 arithmetic on the CPU, for every axis extent an engine accepts: 3 to
2^20 - 1 cells and their ghosts, and powers of two and their neighbours, where
the shifts change."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aeroflux_gb300", "csrc")

MAIN = r"""
#include "af_exact.cuh"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace af::exact;

int main(int argc, char** argv) {
    std::mt19937_64 rng(11);
    const long n = atol(argv[1]);
    long bad = 0, feet = 0, cells = 0, wide = 0;
    for (long i = 0; i < n; ++i) {
        long na;
        switch (rng() % 4) {  // padded extents: any, around a power of two, the largest
        case 0: na = 3 + (long)(rng() % ((1u << 20) + 1300)); break;
        case 1: na = (1l << (2 + rng() % 19)) + (long)(rng() % 7) - 3; break;
        case 2: na = (1l << 20) + (long)(rng() % 1300); break;
        default: na = (1l << 21) - (long)(rng() % 3); break;  // what the shifts hold for
        }
        if (na < 3) na = 3;
        double p;
        switch (rng() % 6) {
        case 0: p = (double)(rng() % na) + ldexp((double)(rng() >> 11), -53); break;
        case 1: p = (double)(rng() % na) + ldexp(1.0, -(int)(rng() % 60)); break;
        case 2: p = (double)(rng() % na) - ldexp(1.0, -(int)(rng() % 60)); break;
        case 3: p = (double)(1l << (rng() % 21)) - ldexp((double)(rng() % 5), -32); break;
        case 4: p = (double)(na - 1) + ldexp((double)(long)(rng() % 9) - 4.0, -31); break;
        default: p = (double)(na - 2) + ldexp((double)(rng() >> 11), -53);
        }
        const unsigned lim = (unsigned)(bits_of((double)(na - 1)) >> 32);
        int a0 = -1, c0 = -1;
        Weights w;
        if (foot_cell(p, lim, &c0)) {
            ++cells;
            bad += !(p >= 0.0 && p < na - 1 && c0 == (int)p);
        } else {
            bad += p >= 0.0 && !std::signbit(p) && p < na - 1;
        }
        if (!foot_split(p, lim, &a0, &w)) continue;
        ++feet;
        wide += p >= 1048576.0;
        const double t = p - (double)(int)p, o = 1.0 - t;
        const double d = (rng() & 1 ? 1.0 : -1.0) * ldexp(1.0 + ldexp((double)(rng() >> 12), -52), (int)(rng() % 200) - 100);
        bad += a0 != (int)p || a0 > na - 2 || !(p > 0.0) || (w.t == 0) != (t == 0.0);
        if (t != 0.0) bad += bits_of(weight_mul(w.t, w.te, d)) != bits_of(d * t);
        bad += bits_of(weight_mul(w.o, w.oe, d)) != bits_of(d * o);
    }
    printf("%ld %ld %ld %ld\n", bad, feet, cells, wide);
}
"""


def test_feet_of_every_extent(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "feet.cpp", tmp_path / "feet"
    src.write_text(MAIN)
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    n = 3_000_000
    bad, feet, cells, wide = (int(v) for v in subprocess.run([str(exe), str(n)], check=True, capture_output=True,
                                                             text=True).stdout.split())
    assert bad == 0
    assert feet > n // 4 and cells > n // 4 and wide > n // 20
