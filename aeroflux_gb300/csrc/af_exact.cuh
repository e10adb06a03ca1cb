// af_exact.cuh -- binary64 products and interpolation weights with integer
// instructions, rounded exactly as the binary64 operations they stand for.
// Internal to libaeroflux_cuda; also compiles as plain C++, so the CPU tests
// compare every function with the native operation.
//
// Why: GB300 issues one warp-wide binary64 operation per SM quarter every 81
// cycles (add, multiply, FMA and compare alike), a 32-bit logic, shift or
// multiply-add every 2.2, an integer add every 1.0 and a 32x32->64 multiply
// about every 5, all of them while the binary64 pipe is busy (measured with
// independent chains).  A product costs about 20 logic and shift
// instructions and four wide multiplies here, about 50 cycles of pipes the
// binary64 kernels leave idle.
#pragma once

#if defined(__CUDACC__)
#define AF_HD __host__ __device__ __forceinline__
#else
#define AF_HD inline
#endif

#include <stdint.h>
#include <string.h>

namespace af {
namespace exact {

typedef unsigned long long u64;

// The words go through an opaque move: knowing they are a binary64's, the
// compiler turns integer tests on them (zero, finite, sign) back into
// binary64 compares (measured: 11.3 instead of 7.0 binary64 instructions a
// face in the sweeps).
AF_HD u64 bits_of(double x) {
#if defined(__CUDA_ARCH__)
    unsigned lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
    return ((u64)hi << 32) | lo;
#else
    u64 b;
    memcpy(&b, &x, sizeof b);
    return b;
#endif
}
AF_HD double from_bits(u64 b) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double x;
    memcpy(&x, &b, sizeof x);
    return x;
#endif
}
AF_HD int clz64(u64 v) {  // v != 0
#if defined(__CUDA_ARCH__)
    return __clzll((long long)v);
#else
    return __builtin_clzll(v);
#endif
}

// The native product for operands outside the integer forms' range: a call,
// so that it neither runs ahead of the branch that needs it nor turns into a
// predicated instruction, either of which would take the binary64 pipe.
#if defined(__CUDACC__)
static __host__ __device__ __noinline__ double mul_native(double a, double b) { return a * b; }
#else
static double mul_native(double a, double b) { return a * b; }
#endif

constexpr u64 kFracBits = 0xFFFFFFFFFFFFFull;
constexpr u64 kImplicit = 0x10000000000000ull;
constexpr u64 kSignBit = 0x8000000000000000ull;

// Exponent fields the integer products take: far enough from both ends that
// two products with constants of field 1023 +- kConstExp, or one with a
// weight of at least 2^-52, stay normal.
constexpr unsigned kExpLo = 400u, kExpSpan = 1247u;
constexpr int kConstExp = 190;
AF_HD unsigned exp_field(u64 b) { return (unsigned)(b >> 52) & 0x7FFu; }
AF_HD bool mul_range(u64 b) { return exp_field(b) - kExpLo < kExpSpan; }

// RN of the product of two positive significands, as the bits of a binary64:
// a = ah:al is a 53-bit significand shifted to the top of 64 bits, b a
// 53-bit significand, e the exponent field of the product when it lies in
// [1, 2) (the sum of the fields minus 1023).  The 128-bit product's high
// half holds the 53 (or 52) leading bits, the low half the fraction that
// decides the rounding; its lowest word only matters as a sticky bit.
AF_HD u64 sig_mul(unsigned ah, unsigned al, u64 b, int e) {
    const unsigned bh = (unsigned)(b >> 32), bl = (unsigned)b;
    const u64 p = (u64)al * bl;
    const u64 t1 = (u64)al * bh + (p >> 32);
    const u64 t2 = (u64)ah * bl + (unsigned)t1;
    u64 m = (u64)ah * bh + (t2 >> 32) + (t1 >> 32);
    unsigned f = (unsigned)t2;
    const unsigned low = (unsigned)p;  // its low 11 bits are zero, so doubling it loses nothing but its top bit
    if (!(m & kImplicit)) {
        m = (m << 1) | (f >> 31);
        f = (f << 1) | (low >> 31);
    } else {
        e += 1;
    }
    f |= low != 0u ? 1u : 0u;
    // Round to nearest even: carry when f > 1/2, or f = 1/2 and m is odd.
    m += ((u64)f + 0x7FFFFFFFu + ((unsigned)m & 1u)) >> 32;
    return m + ((u64)(unsigned)(e - 1) << 52);
}

AF_HD u64 significand(u64 b) { return (b & kFracBits) | kImplicit; }

// A positive constant factor, split once.
struct MulC {
    double v;
    unsigned h, l;  // significand at the top of 64 bits
    int e;          // exponent (field - 1023)
    int ok;         // normal, positive and |e| <= kConstExp
};
inline MulC mul_const(double v) {
    MulC m;
    const u64 b = bits_of(v), s = significand(b) << 11;
    m.v = v;
    m.h = (unsigned)(s >> 32);
    m.l = (unsigned)s;
    m.e = (int)exp_field(b) - 1023;
    m.ok = (b & kSignBit) == 0 && m.e >= -kConstExp && m.e <= kConstExp;
    return m;
}

// RN(m.v * x) for the bits of an x that mul_range accepts; shift multiplies
// by a further 2^shift (exact).
AF_HD u64 mulc_bits(const MulC& m, u64 x, int shift = 0) {
    return sig_mul(m.h, m.l, significand(x), (int)exp_field(x) + m.e + shift) | (x & kSignBit);
}
AF_HD double mulc(const MulC& m, double x) {
    const u64 b = bits_of(x);
    if (m.ok && mul_range(b)) return from_bits(mulc_bits(m, b));
    return mul_native(m.v, x);
}

// Linear interpolation weights at a foot: t and RN(1 - t) as significands at
// the top of 64 bits with their exponent fields.
struct Weights {
    u64 t, o;
    int te, oe;
};

// Splits the foot p, already inside the axis, into its cell a0 = trunc(p)
// and the weights of the taps a0 (o) and a0 + 1 (t); t = 0 for a foot on a
// face.  lim is the high word of binary64(n - 1), n the axis's padded extent:
// n - 1 < 2^21, so that the word holds it whole and p's cell has at most 21 bits.
// False -- nothing decided -- for NaN, p >= n - 1 and p < 2^-11.
AF_HD bool foot_split(double p, unsigned lim, int* a0, Weights* w) {
    const u64 b = bits_of(p);
    const unsigned hi = (unsigned)(b >> 32);
    if (hi - 0x3FF00000u < lim - 0x3FF00000u) {  // 1 <= p < n - 1
        const int e = (int)(hi >> 20) - 1023;    // 0 .. 20
        const u64 m = significand(b);
        *a0 = (int)((unsigned)(m >> 32) >> (20 - e));
        // t in units of 2^-52 (p >= 1 has no finer bits), so 1 - t is exact.
        const u64 t = (m << e) & kFracBits;
        const u64 o = kImplicit - t;
        const int st = clz64(t | 1ull), so = clz64(o);
        w->t = t << st;  // stays 0 for t = 0
        w->te = 1023 + 11 - st;
        w->o = o << so;
        w->oe = 1023 + 11 - so;
        return true;
    }
    if (hi - 0x3F400000u < 0x3FF00000u - 0x3F400000u && lim > 0x3FF00000u) {  // 2^-11 <= p < 1: cell 0, t = p
        const int f = (int)(hi >> 20);
        w->t = significand(b) << 11;
        w->te = f;
        *a0 = 0;
        // 1 - p in units of 2^-64, then RN to 53 bits.
        const u64 o = 0ull - (w->t >> (1022 - f));
        const int so = clz64(o);
        u64 v = o << so;
        int oe = 1022 - so;
        const u64 r = v + 0x3FFull + ((v >> 11) & 1ull);
        if (r < v) {  // rounded up to the next power of two
            v = kSignBit;
            oe += 1;
        } else {
            v = r & ~0x7FFull;
        }
        w->o = v;
        w->oe = oe;
        return true;
    }
    return false;
}

// trunc(p) for a foot 0 <= p < n - 1 (lim as in foot_split); false otherwise.
AF_HD bool foot_cell(double p, unsigned lim, int* a0) {
    const u64 b = bits_of(p);
    const unsigned hi = (unsigned)(b >> 32);
    if (hi >= lim) return false;  // past the last cell, negative or NaN
    const int e = (int)(hi >> 20) - 1023;
    *a0 = e < 0 ? 0 : (int)((unsigned)(significand(b) >> 32) >> (20 - e));
    return true;
}

// RN(d * weight), weight > 0, for a zero d or one that mul_range accepts
// (weight_range).
AF_HD bool is_zero(u64 b) { return (b << 1) == 0; }
AF_HD bool weight_range(double d) { return mul_range(bits_of(d)) || is_zero(bits_of(d)); }
AF_HD double weight_mul(u64 w, int we, double d) {
    const u64 b = bits_of(d);
    if (is_zero(b)) return d;
    return from_bits(sig_mul((unsigned)(w >> 32), (unsigned)w, significand(b), (int)exp_field(b) + we - 1023) |
                     (b & kSignBit));
}

// ---------------------------------------------------------------------------
// RN(a + b) and RN(RN(a - b) / 6) with 32-bit instructions
// ---------------------------------------------------------------------------
// 32 bits of hi:lo starting s bits up (fsr) or s bits down from the top (fsl); 0 <= s < 32.
AF_HD unsigned fsr(unsigned lo, unsigned hi, int s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, s);
#else
    return (unsigned)((((u64)hi << 32) | lo) >> s);
#endif
}
AF_HD unsigned fsl(unsigned lo, unsigned hi, int s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, s);
#else
    return (unsigned)(((((u64)hi << 32) | lo) << s) >> 32);
#endif
}
AF_HD int clz32(unsigned v) {
#if defined(__CUDA_ARCH__)
    return __clz((int)v);
#else
    return v ? __builtin_clz(v) : 32;
#endif
}
// h:l:r += carry-in and b:bl:0, 96 bits.
AF_HD void add96(unsigned& h, unsigned& l, unsigned& r, unsigned bh, unsigned bl, unsigned cin) {
#if defined(__CUDA_ARCH__)
    asm("add.cc.u32 %0, %0, %5;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %3;"
        : "+r"(r), "+r"(l), "+r"(h)
        : "r"(bh), "r"(bl), "r"(cin));
#else
    const unsigned __int128 t = (((unsigned __int128)h << 64) | ((unsigned __int128)l << 32) | r) +
                                (((unsigned __int128)bh << 64) | ((unsigned __int128)bl << 32)) + cin;
    h = (unsigned)(t >> 64), l = (unsigned)(t >> 32), r = (unsigned)t;
#endif
}
// h:l += v; the carry out.
AF_HD unsigned add64_carry(unsigned& h, unsigned& l, unsigned v) {
#if defined(__CUDA_ARCH__)
    unsigned c;
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %2, 0, 0;" : "+r"(l), "+r"(h), "=r"(c) : "r"(v));
    return c;
#else
    const unsigned __int128 t = (((unsigned __int128)h << 32) | l) + v;
    h = (unsigned)(t >> 32), l = (unsigned)t;
    return (unsigned)(t >> 64);
#endif
}

// A rounded sum before packing: its 53-bit significand at the top of c:h:l
// (c = 1, h = 0 when it rounded up to the next power of two), the low 11
// bits of l unspecified; e the exponent field for c = 0; sign in bit 31.
struct Sum {
    unsigned c, h, l, sign;
    int e;
};

// RN(a + b) for normal operands (fields 64 .. 2044) at most 31 binades
// apart whose sum keeps at least one of the larger one's upper 21 bits;
// false otherwise (*s is then unspecified).  The smaller significand is
// aligned to the larger over 96 bits, which hold every bit of both, so the
// sum is exact before it is rounded once.  The logic and shift pipe bounds
// this form: the complement of a subtraction is a multiply-add.
AF_HD bool add_sum(u64 a, u64 b, Sum* s) {
    const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
    const unsigned ma = ah & 0x7FFFFFFFu, mb = bh & 0x7FFFFFFFu;
    const bool sw = ma < mb;
    const unsigned big = ma > mb ? ma : mb, small = ma < mb ? ma : mb;
    const unsigned bigl = sw ? bl : al, smalll = sw ? al : bl;
    const int eb = (int)(big >> 20), d = eb - (int)(small >> 20);
    const unsigned B = (big & 0xFFFFFu) | 0x100000u, S = (small & 0xFFFFFu) | 0x100000u;
    const unsigned m = (unsigned)((int)(ah ^ bh) >> 31), f = m | 1u;  // -1 - v = v * -1 + -1 to subtract
    const int dd = d & 31;
    unsigned r = fsr(0u, smalll, dd) * f + m, l = fsr(smalll, S, dd) * f + m, h = (S >> dd) * f + m;
    add96(h, l, r, B, bigl, m & 1u);
    // h = 0: deep cancellation; h negative: equal high words.
    const bool ok = small >= (64u << 20) && big < (2045u << 20) && d <= 31 && h - 1u < 0x3FFFFFu;
    const int z = clz32(h) & 31;  // 10 .. 31
    s->h = fsl(l, h, z);
    s->l = fsl(r, l, z);
    // Round to nearest even at bit 11 of l; what lies below l is sticky.
    const unsigned q = ((s->l >> 11) & 1u) | ((r << z) != 0u ? 1u : 0u);
    s->c = add64_carry(s->h, s->l, 0x3FFu + q);
    s->e = eb + 11 - z;
    s->sign = (sw ? bh : ah) & 0x80000000u;
    return ok;
}
AF_HD u64 pack_sum(const Sum& s) {
    const unsigned hi = (((unsigned)(s.e - 1) << 20) + fsr(s.h, s.c, 11)) | s.sign;
    return ((u64)hi << 32) | fsr(s.l, s.h, 11);
}

// RN(x / 6) of a rounded sum with c = 0, as div6_int divides: x / 6 =
// 2^-1 x / 3, the significand division by 3 exact integer work (a
// multiply-high by ceil(2^64 / 3) is the exact quotient below 2^63).
AF_HD u64 div6_sum(const Sum& s) {
    const unsigned t = s.h >= 0xC0000000u ? 1u : 2u;
    const int up = 11 - (int)t;
    const u64 n = ((u64)(s.h >> up) << 32) | fsr(s.l & ~0x7FFu, s.h, up);
#if defined(__CUDA_ARCH__)
    u64 q = __umul64hi(n, 0x5555555555555556ull);
#else
    u64 q = n / 3;
#endif
    if ((unsigned)n - 3u * (unsigned)q == 2u) q += 1ull;  // remainder 2/3: up; 1/3: down; never a tie
    return (q + ((u64)(unsigned)(s.e - 2 - (int)t) << 52)) | ((u64)s.sign << 32);
}

}  // namespace exact
}  // namespace af
