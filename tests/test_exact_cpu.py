"""The integer forms of binary64 products, sums and interpolation weights
(csrc/af_exact.cuh) against the native operations, bit for bit, on the CPU:
the header compiles as plain C++ there."""
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

static std::mt19937_64 rng(7);

// A binary64 with the exponent field in [lo, hi] and a significand at an
// edge (zero, all ones, short, ragged at word boundaries) or random.
static double draw(int lo, int hi) {
    u64 m = rng() & kFracBits;
    switch (rng() % 8) {
    case 0: m = 0; break;
    case 1: m = kFracBits; break;
    case 2: m &= ~((1ull << 26) - 1); break;
    case 3: m &= 0xFFFFF00000000ull; break;
    case 4: m &= 0xFFFFFFFFull; break;
    }
    const u64 e = (u64)lo + rng() % (u64)(hi - lo + 1);
    return from_bits(m | (e << 52) | ((rng() & 1) << 63));
}

int main(int argc, char** argv) {
    const long n = atol(argv[1]);
    long bad = 0, products = 0, feet = 0, cells = 0, sums = 0;
    for (long i = 0; i < n; ++i) {  // constant times anything, extremes, zero and NaN included
        const double c = fabs(draw(1, 2046)), x = i % 64 ? draw(0, 2047) : (i % 128 ? 0.0 : -0.0);
        const double got = mulc(mul_const(c), x), want = c * x;
        bad += !(bits_of(got) == bits_of(want) || (std::isnan(got) && std::isnan(want)));
        // in range: two constants and an exact power of two, as the sweep chains them
        const double y = draw(kExpLo, kExpLo + kExpSpan - 1);
        const MulC a = mul_const(fabs(draw(1023 - kConstExp, 1023 + kConstExp))),
                   b = mul_const(fabs(draw(1023 - kConstExp, 1023 + kConstExp)));
        if (!a.ok || !b.ok || !mul_range(bits_of(y))) { ++bad; continue; }
        ++products;
        bad += from_bits(mulc_bits(b, mulc_bits(a, bits_of(y), -2))) != (a.v * (0.25 * y)) * b.v;
    }
    for (long i = 0; i < n; ++i) {  // feet: inside, on faces, near 0, 1 and n - 1, outside, NaN
        const int na = 3 + (int)(rng() % 1000);
        double p;
        switch (rng() % 6) {
        case 0: p = (double)(rng() % na) + ldexp((double)(rng() >> 11), -53); break;
        case 1: p = (double)(rng() % na) + ldexp(1.0, -(int)(rng() % 60)); break;
        case 2: p = (double)(rng() % na) - ldexp(1.0, -(int)(rng() % 60)); break;
        case 3: p = draw(1000, 1034); break;
        case 4: p = draw(0, 2047); break;
        default: p = (double)(na - 1) - ldexp((double)(rng() % 3), -40);
        }
        const unsigned lim = (unsigned)(bits_of((double)(na - 1)) >> 32);
        int a0 = -1, c0 = -1;
        Weights w;
        if (foot_cell(p, lim, &c0)) {
            ++cells;
            bad += !(p >= 0.0 && p < na - 1 && c0 == (int)p);
        }
        if (!foot_split(p, lim, &a0, &w)) continue;
        ++feet;
        const double t = p - (double)(int)p, o = 1.0 - t;
        const double d = rng() % 16 ? draw(kExpLo, kExpLo + kExpSpan - 1) : (rng() % 2 ? 0.0 : -0.0);
        bad += a0 != (int)p || a0 > na - 2 || !(p > 0.0) || !weight_range(d) || (w.t == 0) != (t == 0.0);
        if (t != 0.0) bad += bits_of(weight_mul(w.t, w.te, d)) != bits_of(d * t);
        bad += bits_of(weight_mul(w.o, w.oe, d)) != bits_of(d * o);
    }
    for (long i = 0; i < n; ++i) {  // sums: any exponents, near ones, near cancellation, ties, zero, extremes
        const double a = draw(i % 4 ? 40 : 0, i % 4 ? 2046 : 2047);
        const u64 ab = bits_of(a), ea = exp_field(ab);
        double b;
        switch (rng() % 6) {
        case 0: b = draw(0, 2047); break;
        case 1: b = draw(ea > 40 ? (int)ea - 40 : 0, ea < 2007 ? (int)ea + 40 : 2047); break;
        case 2: b = from_bits((ab ^ ((rng() & 1) << 63)) + (rng() & 0xFFF) - 0x800); break;
        case 3: b = from_bits((ab ^ ((rng() & 1) << 63)) + ((rng() & 0xFFF) << 30) - (0x800ull << 30)); break;
        case 4: b = from_bits(((rng() & 1) << 63) | ((ea > 60 ? ea - 50 - rng() % 6 : ea) << 52) | (rng() & 0xF)); break;
        default: b = rng() % 2 ? -a : (rng() % 2 ? 0.0 : -0.0);
        }
        Sum s;
        if (add_sum(ab, bits_of(b), &s)) {
            ++sums;
            bad += pack_sum(s) != bits_of(a + b);
        }
        if (add_sum(ab, bits_of(b) ^ kSignBit, &s)) {
            bad += pack_sum(s) != bits_of(a - b);
            if (s.c == 0) bad += div6_sum(s) != bits_of((a - b) / 6.0);
        }
    }
    printf("%ld %ld %ld %ld %ld\n", bad, products, feet, cells, sums);
}
"""


def test_integer_forms_equal_the_native_operations(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "exact.cpp", tmp_path / "exact"
    src.write_text(MAIN)
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    n = 3_000_000
    bad, products, feet, cells, sums = (int(v) for v in subprocess.run([str(exe), str(n)], check=True, capture_output=True,
                                                                 text=True).stdout.split())
    assert bad == 0
    assert products == n and feet > n // 4 and cells > n // 4 and sums > n // 3  # the integer forms took them
