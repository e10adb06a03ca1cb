// af_fp64.cu -- FP64 plain form of AeroFlux's fractional-step stages for
// sm_103a.  Every kernel reproduces the reference's binary64 arithmetic bit
// for bit: explicit round-to-nearest intrinsics (never contracted into FMA,
// as Go on amd64 never contracts), the reference's left-to-right evaluation
// order, and sign flips done on the sign bit as Go's unary minus does.
//
// The reference runs each stage as a loop nest over Z-slabs with a join
// between phases; here each stage is one grid-wide kernel and the join is the
// kernel boundary.  Every stage is per-cell independent, so results do not
// depend on the launch shape.
#include "../../include/aeroflux_cuda.h"
#include "af_cells.cuh"
#include "af_internal.h"

#include <math.h>
#include <stdio.h>

#include <algorithm>
#include <cmath>
#include <mutex>

namespace af {
namespace {

using namespace cells;

inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// applyVelocityBC, stencil.go:246-315: 3 components x 3 write sets, each cell
// written once (see bc_cell).
__global__ void k_velocity_bc(Geom g, double* u, double* v, double* w, Status* st, int gate) {
    pdl_wait();
    if (gated(st, gate)) return;
    const int comp = blockIdx.y / 3, set = blockIdx.y % 3;
    const BcComp c = bc_comp(g, comp, view(u, g.u.count, DK_F64_BC, 0), view(v, g.v.count, DK_F64_BC, 0),
                             view(w, g.w.count, DK_F64_BC, 0));
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= bc_set_count(c, set)) return;
    bc_cell(c, g.G, set, i);
}

// ---------------------------------------------------------------------------
// advectDiffuseAxis / advectComponent / faceVelocity / sampleTrilinear,
// stencil.go:21-225.
// ---------------------------------------------------------------------------
struct SweepArgs {
    AF_PTR(const double) u;
    AF_PTR(const double) v;
    AF_PTR(const double) w;
    AF_PTR(double) tu;
    AF_PTR(double) tv;
    AF_PTR(double) tw;
    Dims du, dv, dw;
    int NX, NY, NZ, G;
    exact::MulC dt, invH, lam;
    int has_lam;
    unsigned lim[3];  // per component: high word of binary64(its extent along the sweep axis - 1)
    Status* st;
    int phase;
    void set_scheme(int axis, double dt_, double invH_, double lam_) {
        dt = exact::mul_const(dt_);
        invH = exact::mul_const(invH_);
        lam = exact::mul_const(lam_);
        has_lam = lam_ != 0;
        const Dims* d[3] = {&du, &dv, &dw};
        for (int c = 0; c < 3; ++c) {
            const int n = axis == 0 ? d[c]->nx : (axis == 1 ? d[c]->ny : d[c]->nz);
            lim[c] = (unsigned)(exact::bits_of((double)(n - 1)) >> 32);
        }
    }
};

// faceVelocity (stencil.go:128-155) along the sweep axis at a face of
// component C, only the component on the active axis: the other two feed
// nothing and have no side effects.  Where four faces are averaged, the sum
// is returned and *shift = -2: the caller folds the exact factor 1/4 in.
template <int AX, int C>
__device__ __forceinline__ double face_vel_sum(const SweepArgs& a, int x, int y, int z, int* shift) {
    *shift = C == AX ? 0 : -2;
    const Dims& d = AX == 0 ? a.du : (AX == 1 ? a.dv : a.dw);
    AF_PTR(const double) f = AX == 0 ? a.u : (AX == 1 ? a.v : a.w);
    const int sy = (int)d.sy, sz = (int)d.sz;
    const int i = x + y * sy + z * sz;  // a field holds < 2^31 elements
    if (C == AX) return f[i];
    // The reference's tap order: before the sweep axis's own component
    // (-e_C, 0, e_AX - e_C, e_AX), after it (-e_C, e_AX - e_C, 0, e_AX).
    const int ec = C == 0 ? 1 : (C == 1 ? sy : sz), ea = AX == 0 ? 1 : (AX == 1 ? sy : sz);
    if (AX > C) return dadd(dadd(dadd(f[i - ec], f[i]), f[i + ea - ec]), f[i + ea]);
    return dadd(dadd(dadd(f[i - ec], f[i + ea - ec]), f[i]), f[i + ea]);
}

__device__ __forceinline__ double lerp(double a, double b, double t, double omt) {
    // a*(1-t) + b*t as the reference writes it; omt = 1-t, the same bits the
    // reference recomputes for every lerp
    return dadd(dmul(a, omt), dmul(b, t));
}

// a*(1-t) + b*t for t = +0, with integer instructions: 1-t = 1 exactly, a*1
// is a (NaN stays NaN), b*0 is a zero carrying b's sign when b is finite and
// NaN otherwise, and a + (+-0) is a except that -0 + +0 = +0.
__device__ __forceinline__ double lerp_t0(double a, double b) {
    const unsigned long long ua = (unsigned long long)__double_as_longlong(a);
    const unsigned long long ub = (unsigned long long)__double_as_longlong(b);
    const bool b_nonfinite = (ub & 0x7FF0000000000000ull) == 0x7FF0000000000000ull;
    const bool a_nan = (ua & ~kSign) > 0x7FF0000000000000ull;
    if (b_nonfinite || a_nan) return __longlong_as_double(0x7FFFFFFFFFFFFFFFll);
    if ((ua & ~kSign) == 0ull) return __longlong_as_double((long long)(ua & ub & kSign));
    return a;
}

// |v| < 2^1023 on the high word: a lerp of two such values with weights in
// [0, 1] is finite (the result is bounded by the larger magnitude times
// (1-t) + t <= 1 + 2^-53), so it adds as an exact zero when its weight is +0.
__device__ __forceinline__ bool below_2p1023(double v) {
    return ((unsigned)(dbits(v) >> 32) & 0x7FF00000u) < 0x7FE00000u;
}

// v * dt * invH as the reference evaluates it, (dt*v)*invH; shift: v's exact
// power-of-two factor (face_vel_sum).
__device__ __forceinline__ double face_shift(const SweepArgs& a, double v, int shift) {
    const unsigned long long b = dbits(v);
    if (a.dt.ok && a.invH.ok) {
        if (exact::mul_range(b)) return dfrom(exact::mulc_bits(a.invH, exact::mulc_bits(a.dt, b, shift)));
        if (exact::is_zero(b)) return v;
    }
    return exact::mul_native(exact::mul_native(a.dt.v, shift ? quarter(v) : v), a.invH.v);
}

// sampleTrilinear (stencil.go:166-225) for any backtrace coordinate pa along
// the sweep axis: the clamp, the amd64 truncation, the bounds check of a NaN
// coordinate and the whole interpolation.  Taken by the faces the integer
// form leaves out (zero or extreme taps, clamped or non-finite coordinates);
// a call, so none of its binary64 operations run ahead of the branch.
// False: a contained fault, recorded; the face is not written.
template <int AX>
__device__ __noinline__ bool sample_general(const SweepArgs& a, int c, int x, int y, int z, double pa, double* out) {
    const Dims& d = c == 0 ? a.du : (c == 1 ? a.dv : a.dw);
    AF_PTR(const double) sd = c == 0 ? a.u : (c == 1 ? a.v : a.w);
    const int na = AX == 0 ? d.nx : (AX == 1 ? d.ny : d.nz);
    // Clamp to [0, na-1] (pa < 0 and pa > maxA on the bit patterns: -0 and
    // NaN pass through unchanged, as the comparisons leave them).
    const unsigned long long pab = dbits(pa);
    const bool pnan = (pab & ~kSign) > 0x7FF0000000000000ull;
    if (!pnan) {
        if ((pab & kSign) && (pab & ~kSign)) pa = 0.0;
        else if (!(pab & kSign) && pab > dbits(i2d_small(na - 1))) pa = i2d_small(na - 1);
    }
    // Truncation toward zero as amd64 CVTTSD2SQ does (NaN -> INT64_MIN).  The
    // two other coordinates are integer faces strictly inside the padded
    // field, so their floor is the face itself and their weight is +0.
    long long a0 = pnan ? (long long)0x8000000000000000ull : d2i_trunc_small(pa);
    if (a0 >= na - 1) a0 = na - 2;
    const double t = pnan ? dsub(pa, (double)a0) : frac_sub(pa, a0);
    long long x0 = x, y0 = y, z0 = z;
    if (AX == 0) x0 = a0;
    if (AX == 1) y0 = a0;
    if (AX == 2) z0 = a0;
    // Index arithmetic wraps modulo 2^64, as Go's int does.
    const unsigned long long i000 =
        (unsigned long long)x0 + (unsigned long long)y0 * (unsigned long long)d.sy +
        (unsigned long long)z0 * (unsigned long long)d.sz;
    if (pnan) {
        // Only a NaN coordinate can leave the field; Go bounds-checks the taps
        // in source order and panics at the first out-of-range one.
        const unsigned long long sy = d.sy, sz = d.sz, n = d.count;
        const unsigned long long taps[8] = {i000, i000 + 1, i000 + sy, i000 + sy + 1,
                                            i000 + sz, i000 + sz + 1, i000 + sz + sy, i000 + sz + sy + 1};
        bool oob = false;
#pragma unroll
        for (int k = 0; k < 8; ++k) oob |= (long long)taps[k] < 0 || taps[k] >= n;
        if (oob) {
            atomicMin(&a.st->fault_gate, a.st->step * 8u + (unsigned)a.phase);
            atomicMin(&a.st->fault_key, fault_key(c, x, y, z));
            return false;  // the faulting face is not written, as the panic leaves it
        }
    }
    const long long sy = d.sy, sz = d.sz, b = (long long)i000;
    // Only the active axis has a nonzero weight; the lerps along the other
    // two (weight exactly +0) run on the integer pipe with identical bits.
    const double t0 = sd[b], t1 = sd[b + 1], t2 = sd[b + sy], t3 = sd[b + sy + 1];
    const double t4 = sd[b + sz], t5 = sd[b + sz + 1], t6 = sd[b + sz + sy], t7 = sd[b + sz + sy + 1];
    const double omt = dsub(1.0, t);
    if (AX == 0)
        *out = lerp_t0(lerp_t0(lerp(t0, t1, t, omt), lerp(t2, t3, t, omt)),
                       lerp_t0(lerp(t4, t5, t, omt), lerp(t6, t7, t, omt)));
    else if (AX == 1)
        *out = lerp_t0(lerp(lerp_t0(t0, t1), lerp_t0(t2, t3), t, omt), lerp(lerp_t0(t4, t5), lerp_t0(t6, t7), t, omt));
    else
        *out = lerp(lerp_t0(lerp_t0(t0, t1), lerp_t0(t2, t3)), lerp_t0(lerp_t0(t4, t5), lerp_t0(t6, t7)), t, omt);
    return true;
}

// lam * ((m - 2*c) + p), the directional diffusion (stencil.go:73-119).
__device__ __forceinline__ double diffusion(const SweepArgs& a, double m, double c, double p) {
    return exact::mulc(a.lam, dadd(dsub(m, twice(c)), p));
}

// One face of component C.  The common face -- backtrace inside the field,
// both interpolated taps zero or normal, none of the other six huge --
// computes its six products (dt, 1/h, the two weights, the diffusion) and its
// weights with integer instructions (af_exact.cuh), so only the additions
// (eight, or five where the face's own component is the velocity) are left
// to the binary64 pipe, which bounds the kernel.  The lerps along the two
// other axes, whose weight is zero, then return their first operand (their
// second ones are finite) unless it is -0.
// Measured at 256^3 per launch: 2.28 / 2.45 / 2.71 ms (x, y, z) with the
// products, weights and compares on the binary64 pipe (25-29 of its
// instructions a face), 0.78 ms each so (7); block shapes from 32 x 4 to
// 256 x 1 measure the same.
template <int AX, int C>
__device__ __forceinline__ void sweep_face(const SweepArgs& a, int x, int y, int z) {
    const Dims& d = C == 0 ? a.du : (C == 1 ? a.dv : a.dw);
    AF_PTR(const double) sd = C == 0 ? a.u : (C == 1 ? a.v : a.w);
    AF_PTR(double) dd = C == 0 ? a.tu : (C == 1 ? a.tv : a.tw);
    const int sy = (int)d.sy, sz = (int)d.sz;
    const int i = x + y * sy + z * sz, st = AX == 0 ? 1 : (AX == 1 ? sy : sz);
    int shift;
    const double vel = face_vel_sum<AX, C>(a, x, y, z, &shift);
    const int ca = AX == 0 ? x : (AX == 1 ? y : z);
    // Backtrace along the active axis only: p -= dt*v*invH.
    const double pa = dsub(i2d_small(ca), face_shift(a, vel, shift));
    int a0;
    exact::Weights w;
    double adv;
    bool done = false;
    if (exact::foot_split(pa, a.lim[C], &a0, &w)) {
        const int b = i + (a0 - ca) * st;
        // The cell's taps: b and b + st interpolate along the axis, the
        // other six carry a zero weight.
        const int s1 = AX == 0 ? sy : 1, s2 = AX == 2 ? sy : sz;
        const double d0 = sd[b], d1 = sd[b + st];
        const double q[6] = {sd[b + s1], sd[b + s1 + st], sd[b + s2], sd[b + s2 + st], sd[b + s1 + s2],
                             sd[b + s1 + s2 + st]};
        unsigned any = 0;
#pragma unroll
        for (int k = 0; k < 6; ++k) any |= (unsigned)(dbits(q[k]) >> 32);
        bool ok = exact::weight_range(d0) && exact::weight_range(d1);
        if (any & 0x40000000u) {  // some |tap| >= 2: look at each
#pragma unroll
            for (int k = 0; k < 6; ++k) ok = ok && below_2p1023(q[k]);
        }
        if (ok) {
            // On a face: d0 * 1 + d1 * 0.
            adv = w.t == 0 ? d0 : dadd(exact::weight_mul(w.o, w.oe, d0), exact::weight_mul(w.t, w.te, d1));
            done = dbits(adv) != kSign;
        }
    }
    if (!done && !sample_general<AX>(a, C, x, y, z, pa, &adv)) return;
    double lap = 0.0;
    if (a.has_lam) lap = diffusion(a, sd[i - st], sd[i], sd[i + st]);
    dd[i] = dadd(adv, lap);
}

// The face of a thread: z layers of blocks per component, a warp to 32
// consecutive x.  A U row holds NX + 1 faces; with NX a multiple of 32 its
// last face would cost a whole warp, so those faces come in further z layers,
// 32 rows to a warp.  False: no face.
__device__ __forceinline__ bool block_face(const SweepArgs& a, int* c, int* x, int* y, int* z) {
    const int zr = a.NZ + 1, layer = (int)blockIdx.z;
    if (layer < 3 * zr) {
        *c = layer < zr ? 0 : (layer < 2 * zr ? 1 : 2);
        *z = a.G + layer - *c * zr;
        *x = a.G + (int)(blockIdx.x * blockDim.x + threadIdx.x);
        *y = a.G + (int)(blockIdx.y * blockDim.y + threadIdx.y);
        // Face-count extents of the component (stencil.go:53-68).
        return *x < a.G + a.NX + (*c == 0) && *y < a.G + a.NY + (*c == 1) && *z < a.G + a.NZ + (*c == 2);
    }
    const unsigned blk = ((unsigned)(layer - 3 * zr) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    const unsigned k = (blk * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
    if (k >= (unsigned)a.NY * (unsigned)a.NZ) return false;
    *c = 0;
    *x = a.G + a.NX;
    *z = a.G + (int)(k / (unsigned)a.NY);
    *y = a.G + (int)(k % (unsigned)a.NY);
    return true;
}
dim3 face_grid(const Geom& g, dim3 block) {
    const unsigned gx = cdiv(g.NX, block.x), gy = cdiv(g.NY + 1, block.y), gz = 3u * (unsigned)(g.NZ + 1);
    if (g.NX % block.x) return dim3(gx, gy, gz);  // the last face shares its row's last warp
    const unsigned last = cdiv((long long)g.NY * g.NZ, (long long)gx * gy * block.x * block.y);
    if (gz + last > 65535u) return dim3(gx + 1, gy, gz);  // the z extent of a launch
    return dim3(gx, gy, gz + last);
}

template <int AX>
__global__ void k_sweep_fp64(const __grid_constant__ SweepArgs a) {
    pdl_wait();
    if (gated(a.st, a.phase)) return;
    int c, x, y, z;
    if (!block_face(a, &c, &x, &y, &z)) return;
    if (c == 0) sweep_face<AX, 0>(a, x, y, z);
    else if (c == 1) sweep_face<AX, 1>(a, x, y, z);
    else sweep_face<AX, 2>(a, x, y, z);
}

// ---------------------------------------------------------------------------
// MacCormack correction of one axis sweep (Selle, Fedkiw, Kim, Liu, Rossignac,
// "An Unconditionally Stable MacCormack Method", J. Sci. Comput. 2008), the
// higher-order advection the reference lists as its missing remedy for
// semi-Lagrangian dissipation (README "Known limitations").  The forward
// step is the reference sweep itself run with lam = 0 into `fwd` (phi^ =
// semi-Lagrangian advection of the component, faults and all); this kernel
// traces the same face velocity forward (x + dt*v*invH) through phi^ to get
// phi~, forms phi^ + (phi - phi~)/2, falls back to phi^ where that leaves the
// range of the two source values the forward step interpolated (the limiter
// that keeps the scheme unconditionally stable), and adds the reference's
// directional diffusion of phi.  Along the sweep axis only: the tangential
// weights are zero, as in the forward step.  Taps of phi^ outside the faces
// the sweep writes read phi (the boundary-conditioned field) instead.
// The correction of one face for any operands (clamped or NaN feet, zero,
// huge or non-finite taps); a call, as sample_general is.
template <int AX>
__device__ __noinline__ double maccormack_general(const SweepArgs& a, AF_PTR(const double) fd, int c, int i, int ca,
                                                  int lo, int hi, double pf, double pb, double fwd) {
    const Dims& d = c == 0 ? a.du : (c == 1 ? a.dv : a.dw);
    AF_PTR(const double) sd = c == 0 ? a.u : (c == 1 ? a.v : a.w);
    const int na = AX == 0 ? d.nx : (AX == 1 ? d.ny : d.nz);
    const long long step = AX == 0 ? 1 : (AX == 1 ? d.sy : d.sz);
    if (isnan(pf) || isnan(pb)) return fwd;  // the forward step has dealt with it
    const double maxA = (double)(na - 1);
    pf = fmin(fmax(pf, 0.0), maxA);
    pb = fmin(fmax(pb, 0.0), maxA);
    long long f0 = (long long)pf, b0 = (long long)pb;
    if (f0 >= na - 1) f0 = na - 2;
    if (b0 >= na - 1) b0 = na - 2;
    const long long base = i - (long long)ca * step;  // the face's row at axis coordinate 0
    const double s0 = sd[base + f0 * step], s1 = sd[base + (f0 + 1) * step];
    const double mn = fmin(s0, s1), mx = fmax(s0, s1);
    auto phi_hat = [&](long long k) { return (k >= lo && k <= hi) ? fd[base + k * step] : sd[base + k * step]; };
    const double tb = dsub(pb, (double)b0);
    const double back = dadd(dmul(phi_hat(b0), dsub(1.0, tb)), dmul(phi_hat(b0 + 1), tb));
    const double out = dadd(fwd, dmul(0.5, dsub(sd[i], back)));
    return out >= mn && out <= mx ? out : fwd;
}

// Finite doubles in their numeric order as integers, -0 equal to +0.
__device__ __forceinline__ long long order_key(double v) {
    const long long k = (long long)dbits(v);
    return (k << 1) == 0 ? 0 : k ^ ((k >> 63) & 0x7FFFFFFFFFFFFFFFll);
}
__device__ __forceinline__ bool finite(double v) {
    return ((unsigned)(dbits(v) >> 32) & 0x7FF00000u) != 0x7FF00000u;
}

// As sweep_face: the common face's products, weights, halving and limiter
// comparisons are integer instructions, its additions (eleven, or eight where
// the component is the velocity) the only work of the binary64 pipe.  With
// the forward step, a sweep at 128^3 went from about 1.0 to 0.22 ms.
template <int AX, int C>
__device__ __forceinline__ void maccormack_face(const SweepArgs& a, const double* fwd_field, int x, int y, int z) {
    const Dims& d = C == 0 ? a.du : (C == 1 ? a.dv : a.dw);
    AF_PTR(const double) sd = C == 0 ? a.u : (C == 1 ? a.v : a.w);
    AF_PTR(const double) fd = view(fwd_field, d.count, DK_F64_MACCORMACK, 0);
    AF_PTR(double) dd = C == 0 ? a.tu : (C == 1 ? a.tv : a.tw);
    const int sy = (int)d.sy, sz = (int)d.sz;
    const int i = x + y * sy + z * sz, st = AX == 0 ? 1 : (AX == 1 ? sy : sz);
    const int ca = AX == 0 ? x : (AX == 1 ? y : z);
    // Written faces on the axis.
    const int lo = a.G, hi = a.G + (AX == 0 ? a.NX : (AX == 1 ? a.NY : a.NZ)) - (C == AX ? 0 : 1);
    const double fwd = fd[i], here = sd[i];
    int shift;
    const double vel = face_vel_sum<AX, C>(a, x, y, z, &shift);
    const double cad = i2d_small(ca), s = face_shift(a, vel, shift);
    // Forward foot (the one the forward step sampled) and backward foot.
    const double pf = dsub(cad, s), pb = dadd(cad, s);
    int f0, b0;
    exact::Weights w;
    double out;
    bool done = false;
    if (exact::foot_cell(pf, a.lim[C], &f0) && exact::foot_split(pb, a.lim[C], &b0, &w)) {
        const int base = i - ca * st;
        const double s0 = sd[base + f0 * st], s1 = sd[base + (f0 + 1) * st];
        auto phi_hat = [&](int k) { return (k >= lo && k <= hi) ? fd[base + k * st] : sd[base + k * st]; };
        const double e0 = phi_hat(b0), e1 = phi_hat(b0 + 1);
        if (exact::weight_range(e0) && exact::weight_range(e1)) {
            const double back = w.t == 0 ? e0 : dadd(exact::weight_mul(w.o, w.oe, e0), exact::weight_mul(w.t, w.te, e1));
            out = dadd(fwd, half(dsub(here, back)));
            if (dbits(back) != kSign && finite(s0) && finite(s1) && finite(out)) {
                const long long k0 = order_key(s0), k1 = order_key(s1), k = order_key(out);
                if (k < (k0 < k1 ? k0 : k1) || k > (k0 < k1 ? k1 : k0)) out = fwd;
                done = true;
            }
        }
    }
    if (!done) out = maccormack_general<AX>(a, fd, C, i, ca, lo, hi, pf, pb, fwd);
    double lap = 0.0;
    if (a.has_lam) lap = diffusion(a, sd[i - st], here, sd[i + st]);
    dd[i] = dadd(out, lap);
}

template <int AX>
__global__ void k_maccormack_fp64(const __grid_constant__ SweepArgs a, const double* fu, const double* fv,
                                  const double* fw) {
    pdl_wait();
    if (gated(a.st, a.phase)) return;
    int c, x, y, z;
    if (!block_face(a, &c, &x, &y, &z)) return;
    if (c == 0) maccormack_face<AX, 0>(a, fu, x, y, z);
    else if (c == 1) maccormack_face<AX, 1>(a, fv, x, y, z);
    else maccormack_face<AX, 2>(a, fw, x, y, z);
}

// ---------------------------------------------------------------------------
// computeDivergence (project.go:42-62).  For the red-black sweeps it also
// stores B = h2*Div, the product every update recomputes (project.go:126),
// split by colour -- same bits, one multiply fewer per update -- and zeroes
// their P (project.go:81-83).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void split_store(const Split& S, const exact::MulC& h2, int xi, int yi, int zi, double d) {
    AF_PTR(double) b = view(S.b, 2 * S.bn, DK_F64_DIV, 0);
    const int c = (xi + yi + zi + S.G) & 1;
    b[c * S.bn + ((xi >> 1) + S.hx * (yi + S.NY * zi))] = exact::mulc(h2, d);
}
__device__ __forceinline__ void split_zero(const Split& S) {
    AF_PTR(double) p = view(S.p, 2 * S.pn, DK_F64_DIV, 0);
    const long long block = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    const int n = blockDim.x * blockDim.y, t = threadIdx.y * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * gridDim.y * gridDim.z * n;
    for (long long k = block * n + t; k < 2 * S.pn; k += stride) p[k] = 0.0;
}

__global__ void k_divergence_fp64(const __grid_constant__ Geom g, const double* __restrict__ u,
                                  const double* __restrict__ v, const double* __restrict__ w, double* __restrict__ dv,
                                  const __grid_constant__ Split S, int with_b,
                                  const __grid_constant__ exact::MulC scale, const __grid_constant__ exact::MulC h2,
                                  Status* st, int gate) {
    pdl_wait();
    if (gated(st, gate)) return;
    if (with_b) split_zero(S);
    const int xi = blockIdx.x * blockDim.x + threadIdx.x;
    const int yi = blockIdx.y * blockDim.y + threadIdx.y;
    const int zi = blockIdx.z;
    if (xi >= g.NX || yi >= g.NY) return;
    const int x = g.G + xi, y = g.G + yi, z = g.G + zi;
    const double d = div_value(g, view(u, g.u.count, DK_F64_DIV, 0), view(v, g.v.count, DK_F64_DIV, 0),
                               view(w, g.w.count, DK_F64_DIV, 0), scale, x, y, z);
    view(dv, g.p.count, DK_F64_DIV, 0)[x + y * g.p.sy + z * g.p.sz] = d;
    if (with_b) split_store(S, h2, xi, yi, zi, d);
}

// The same split arrays for the red-black phase hook, when Div was supplied
// directly instead of by the divergence kernel.
__global__ void k_split_from_div(const __grid_constant__ Geom g, const double* __restrict__ dv,
                                 const __grid_constant__ Split S, const __grid_constant__ exact::MulC h2) {
    split_zero(S);
    const int xi = blockIdx.x * blockDim.x + threadIdx.x;
    const int yi = blockIdx.y * blockDim.y + threadIdx.y;
    const int zi = blockIdx.z;
    if (xi >= g.NX || yi >= g.NY) return;
    const int i = (g.G + xi) + (g.G + yi) * (int)g.p.sy + (g.G + zi) * (int)g.p.sz;
    split_store(S, h2, xi, yi, zi, view(dv, g.p.count, DK_F64_B, 0)[i]);
}

// ---------------------------------------------------------------------------
// gaussSeidelSweep, project.go:103-130, with applyPressureBC folded in: the
// split arrays' ghosts (see Split) always hold what the reference's mirror
// before each colour would put there.
// ---------------------------------------------------------------------------
// EMU selects which of the update's six binary64 additions (five, and the
// subtraction last) run on the integer pipe (bit k: operation k of the
// chain); the others issue on the binary64 pipe.  Every choice computes the
// same bits.
static __device__ __noinline__ double sub_div6_call(double a, double b) { return div6_int(dsub(a, b)); }

template <int EMU>
__device__ __forceinline__ double rb_update(double xm, double xp, double ym, double yp, double zm, double zp,
                                            double b) {
    const double v[5] = {xp, ym, yp, zm, zp};
    double sum = xm;
#pragma unroll
    for (int k = 0; k < 5; ++k) sum = ((EMU >> k) & 1) ? dadd_int(sum, v[k]) : dadd(sum, v[k]);
    if ((EMU >> 5) & 1) {
        // The subtraction feeds the division unpacked.
        exact::Sum s;
        if (exact::add_sum(dbits(sum), dbits(b) ^ kSign, &s) && s.c == 0) return dfrom(exact::div6_sum(s));
        return sub_div6_call(sum, b);
    }
    return div6_int(dsub(sum, b));
}

// A thread per cell of the colour, a plane's cells dealt out in order, which
// keeps the warps of short and ragged rows full (a block per row measured the
// same on long rows, blocks of 256 slower; several cells a thread along z,
// unrolled or marching, are slower on every grid or on the small ones).  An
// odd row's last slot of the colour it has one cell less of computes its
// in-bounds neighbours too and drops the result, so warps do not diverge.
// The sweeps touch scratch only, so they do not look at the fault gate: the
// join does, before P is written.
template <int EMU>
__global__ void __launch_bounds__(128) k_rbgs_fp64(const __grid_constant__ Split S, int color) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= S.hx * S.NY) return;
    const int y = (int)S.fhx.div((unsigned)t), j = t - y * S.hx, z = (int)blockIdx.y;
    const int q = (color + S.G + y + z) & 1, x = 2 * j + q;
    AF_PTR(double) own = view(S.p, 2 * S.pn, DK_F64_RBGS, 0) + (color ? S.pn : 0);
    AF_PTR(double) opp = view(S.p, 2 * S.pn, DK_F64_RBGS, 0) + (color ? 0 : S.pn);
    AF_PTR(const double) b = view((const double*)S.b, 2 * S.bn, DK_F64_RBGS, 0) + (color ? S.bn : 0);
    const int i = (j + 1) + S.px * (y + 1) + S.plane * (z + 1);
    pdl_wait();
    // Of the two x neighbours one has the cell's own half index, the other
    // the next (odd x) or the previous one; their sum does not depend on
    // which is which.
    const double r = rb_update<EMU>(opp[i], opp[q ? i + 1 : i - 1], opp[i - S.px], opp[i + S.px], opp[i - S.plane],
                                    opp[i + S.plane], b[t + S.hx * S.NY * z]);
    pdl_trigger();  // the next sweep's blocks get ready while this one's last ones finish
    if (x >= S.NX) return;
    own[i] = r;
    if ((unsigned)(x - 1) >= (unsigned)(S.NX - 2) || (unsigned)(y - 1) >= (unsigned)(S.NY - 2) ||
        (unsigned)(z - 1) >= (unsigned)(S.NZ - 2)) {  // a wall cell: its ghosts
        if (x == 0) opp[i - 1] = r;
        if (x == S.NX - 1) opp[q ? i + 1 : i] = r;
        if (y == 0) opp[i - S.px] = r;
        if (y == S.NY - 1) opp[i + S.px] = r;
        if (z == 0) opp[i - S.plane] = r;
        if (z == S.NZ - 1) opp[i + S.plane] = r;
    }
}

// ---------------------------------------------------------------------------
// All the sweeps of one solve on a small grid, in one launch: a cluster of
// kRbCluster blocks holds P in its shared memory.  Block k owns the rows
// (y, z) from k * rows on, both colours; a thread owns up to NC cells of each
// colour, whose B, own value and the shared-memory addresses of their six
// neighbours -- in whichever block they lie; its own cell's across a wall --
// it keeps in registers over all sweeps.  A colour costs the neighbour loads,
// the update (the subtraction on the integer pipe: a thread waits for its own
// chain here, and the first addition there would be a longer link than on the
// binary64 pipe), one store and a cluster barrier.
// us per colour, a launch each / so: 12^3 1.75 / 0.77, 16^3 1.75 / 0.68, 24^3
// 1.88 / 1.33, 40x12x33 1.9 / 1.37, 28^3 1.88 / 1.84, 32^3 1.92 / 2.26: past
// kRbMaxCells the binary64 pipe bounds it, of which a cluster has only its
// SMs' share.
// ---------------------------------------------------------------------------
constexpr int kRbCluster = 16, kRbThreads = 512;
constexpr int kRbMaxCells = 20480;
// A block's two colours of at most 2 * kRbThreads slots fit the shared memory
// a launch gets without asking for more.  The limit is not set per solve: it
// belongs to the function, not to an engine, and a smaller engine on another
// thread would lower it between a larger one's check and its launch.
static_assert(2 * 2 * kRbThreads * sizeof(double) <= 48 * 1024, "no larger shared-memory limit is asked for");

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The address, in the cluster's shared window, of a block's copy of a
// shared-memory address.
__device__ __forceinline__ unsigned cluster_addr(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ double cluster_ld(unsigned addr) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int NC>
__global__ void __launch_bounds__(kRbThreads) k_rbgs_cluster(const __grid_constant__ Split S, long long pairs) {
    extern __shared__ __align__(16) double rb_smem[];  // [colour][row of the block][half index]
    pdl_wait();
    const int rows = (S.NY * S.NZ + kRbCluster - 1) / kRbCluster;  // per block
    const int mine = (int)cluster_rank(), row0 = mine * rows;
    const int n = max(0, min(rows, S.NY * S.NZ - row0)) * S.hx;    // slots of a colour here
    const unsigned base = (unsigned)__cvta_generic_to_shared(rb_smem);
    AF_PTR(double) sm = view(rb_smem, 2ll * rows * S.hx, DK_F64_RBGS, 0);
    AF_PTR(const double) b = view((const double*)S.b, 2 * S.bn, DK_F64_RBGS, 0);
    AF_PTR(double) p = view(S.p, 2 * S.pn, DK_F64_RBGS, 0);
    unsigned nb[2][NC][6];
    int at[2][NC];
    double bv[2][NC], own[2][NC];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            const int t = (int)threadIdx.x + k * kRbThreads;
            const int r = (int)S.fhx.div((unsigned)t), j = t - r * S.hx, row = row0 + r;
            const int z = row / S.NY, y = row - z * S.NY;
            const int q = (c + S.G + y + z) & 1, x = 2 * j + q;
            at[c][k] = -1;
            own[c][k] = bv[c][k] = 0.0;
            if (t < n && x < S.NX) {
                at[c][k] = c * rows * S.hx + t;
                bv[c][k] = b[(c ? S.bn : 0) + j + S.hx * row];
                // The other colour's cell at half index jj of a row.
                auto other = [&](int rr, int jj) {
                    const int k2 = rr / rows;
                    return cluster_addr(base + 8u * (unsigned)(((c ^ 1) * rows + rr - k2 * rows) * S.hx + jj),
                                        (unsigned)k2);
                };
                const unsigned self = cluster_addr(base + 8u * (unsigned)at[c][k], (unsigned)mine);
                nb[c][k][0] = x > 0 ? other(row, (x - 1) >> 1) : self;
                nb[c][k][1] = x < S.NX - 1 ? other(row, (x + 1) >> 1) : self;
                nb[c][k][2] = y > 0 ? other(row - 1, j) : self;
                nb[c][k][3] = y < S.NY - 1 ? other(row + 1, j) : self;
                nb[c][k][4] = z > 0 ? other(row - S.NY, j) : self;
                nb[c][k][5] = z < S.NZ - 1 ? other(row + S.NY, j) : self;
            }
        }
    for (int i = (int)threadIdx.x; i < 2 * rows * S.hx; i += kRbThreads) sm[i] = 0.0;  // project.go:81-83
    cluster_sync();
    for (long long it = 0; it < pairs; ++it)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            double v[NC];
#pragma unroll
            for (int k = 0; k < NC; ++k)
                if (at[c][k] >= 0)
                    v[k] = rb_update<0x20>(cluster_ld(nb[c][k][0]), cluster_ld(nb[c][k][1]), cluster_ld(nb[c][k][2]),
                                        cluster_ld(nb[c][k][3]), cluster_ld(nb[c][k][4]), cluster_ld(nb[c][k][5]),
                                        bv[c][k]);
#pragma unroll
            for (int k = 0; k < NC; ++k)
                if (at[c][k] >= 0) sm[at[c][k]] = own[c][k] = v[k];
            cluster_sync();
        }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int k = 0; k < NC; ++k)
            if (at[c][k] >= 0) {
                const int t = (int)threadIdx.x + k * kRbThreads;
                const int r = (int)S.fhx.div((unsigned)t), row = row0 + r, z = row / S.NY, y = row - z * S.NY;
                p[(c ? S.pn : 0) + (t - r * S.hx + 1 + S.px * (y + 1) + S.plane * (z + 1))] = own[c][k];
            }
}

// The split P into P: a ghost of the first layer holds the interior cell at
// the clamped coordinates (applyPressureBC, project.go:139-163, composed),
// the layers past it stay zero (project.go:81-83).
__global__ void k_join_fp64(const __grid_constant__ Geom g, const __grid_constant__ Split S, double* p_, Status* st,
                            int gate) {
    pdl_wait();
    if (gated(st, gate)) return;
    const int x = blockIdx.x * blockDim.x + threadIdx.x - g.G;
    const int y = blockIdx.y * blockDim.y + threadIdx.y - g.G;
    const int z = (int)blockIdx.z - g.G;
    if (x >= g.NX + g.G || y >= g.NY + g.G) return;
    AF_PTR(double) p = view(p_, g.p.count, DK_F64_PBC, 0);
    AF_PTR(const double) s = view((const double*)S.p, 2 * S.pn, DK_F64_PBC, 0);
    double v = 0.0;
    if (x >= -1 && x <= g.NX && y >= -1 && y <= g.NY && z >= -1 && z <= g.NZ) {
        const int cx = min(max(x, 0), g.NX - 1), cy = min(max(y, 0), g.NY - 1), cz = min(max(z, 0), g.NZ - 1);
        v = s[((cx + cy + cz + g.G) & 1 ? S.pn : 0) + ((cx >> 1) + 1 + S.px * (cy + 1) + S.plane * (cz + 1))];
    }
    p[(x + g.G) + (y + g.G) * (int)g.p.sy + (z + g.G) * (int)g.p.sz] = v;
}

// applyPressureBC, project.go:139-163 (see pbc_cell).
__global__ void k_pressure_bc(Geom g, double* __restrict__ p, Status* st, int gate) {
    if (gated(st, gate)) return;
    const int set = blockIdx.y;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pbc_set_count(g, set)) return;
    pbc_cell(g, view(p, g.p.count, DK_F64_PBC, 0), set, i);
}

// subtractGradient, project.go:172-205 (see grad_cell), a plane's cells dealt
// out in order.  256^3: 282 us with a thread a face, 207 so.
__global__ void __launch_bounds__(256) k_gradient_fp64(const __grid_constant__ Geom g, const FastDiv fx,
                                                       const double* __restrict__ p, double* u_, double* v_, double* w_,
                                                       const __grid_constant__ exact::MulC scale, Status* st,
                                                       int gate) {
    pdl_wait();
    if (gated(st, gate)) return;
    const unsigned e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (unsigned)(g.NX + 1) * (unsigned)(g.NY + 1)) return;
    const unsigned y = fx.div(e);
    AF_PTR(double) u = view(u_, g.u.count, DK_F64_GRAD, 0);
    AF_PTR(double) v = view(v_, g.v.count, DK_F64_GRAD, 0);
    AF_PTR(double) w = view(w_, g.w.count, DK_F64_GRAD, 0);
    grad_cell(g, view(p, g.p.count, DK_F64_GRAD, 0), u, v, w, u, v, w, scale, g.G + (int)(e - y * fx.d), g.G + (int)y,
              g.G + (int)blockIdx.y);
}

__global__ void k_step_tick(Status* st) {
    pdl_wait();
    st->step += 1;
}

// ---------------------------------------------------------------------------
// Diagnostics.  A max is exact in any order; NaN is skipped as the
// reference's `if a > mx` skips it.  Non-negative doubles order like their
// bit patterns, so one atomicMax per block combines the blocks, and every
// test on a value is an integer one (a binary64 compare costs the binary64
// pipe as much as an addition).  A warp walks a row, eight rows to a block (32
// left the last wave half empty).  us a call at 256^3 before/now: max
// divergence 279/188, max |velocity| 224/78 (HBM), kinetic energy 498/226;
// the binary64 pipe bounds the first and the last, and further additions on
// the integer pipe made neither faster.
// ---------------------------------------------------------------------------
constexpr int kDiagThreads = 256, kDiagRows = 8;

__device__ __forceinline__ unsigned long long abs_bits(double d) {
    const unsigned long long b = dbits(d) & ~kSign;
    return b > 0x7FF0000000000000ull ? 0ull : b;
}

__device__ __forceinline__ void block_max_commit(unsigned long long m, unsigned long long* out) {
    __shared__ unsigned long long sm[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, o);
        m = t > m ? t : m;
    }
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < blockDim.x / 32 ? sm[threadIdx.x] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, o);
            m = t > m ? t : m;
        }
        if (threadIdx.x == 0 && m) atomicMax(out, m);
    }
}

// max |du + dv + dw| for MaxDivergence (project.go:210-232), which is
// RN(1/h * that): rounding is monotone, so the product commutes with the
// maximum and is taken once, by the host.  Of the five additions one runs on
// the integer pipe beside the others.
__global__ void __launch_bounds__(kDiagThreads) k_max_divergence(const __grid_constant__ Geom g,
                                                                 const double* __restrict__ u_,
                                                                 const double* __restrict__ v_,
                                                                 const double* __restrict__ w_,
                                                                 unsigned long long* out) {
    const int G = g.G;
    AF_PTR(const double) AF_RESTRICT u = view(u_, g.u.count, DK_F64_MAXDIV, 0);
    AF_PTR(const double) AF_RESTRICT v = view(v_, g.v.count, DK_F64_MAXDIV, 0);
    AF_PTR(const double) AF_RESTRICT w = view(w_, g.w.count, DK_F64_MAXDIV, 0);
    const int z = G + (int)blockIdx.y, y0 = (int)blockIdx.x * kDiagRows;
    unsigned long long m = 0;
    for (int r = (int)threadIdx.x >> 5; r < kDiagRows && y0 + r < g.NY; r += kDiagThreads / 32) {
        const int y = G + y0 + r;
        const int iu = y * (int)g.u.sy + z * (int)g.u.sz, iv = y * (int)g.v.sy + z * (int)g.v.sz;
        const int iw = y * (int)g.w.sy + z * (int)g.w.sz;
        for (int x = G + ((int)threadIdx.x & 31); x < G + g.NX; x += 32) {
            const double du = dsub(u[iu + x + 1], u[iu + x]);
            const double dv = dsub_int(v[iv + x + (int)g.v.sy], v[iv + x]);
            const double d = dadd(dadd(du, dv), dsub(w[iw + x + (int)g.w.sz], w[iw + x]));
            const unsigned long long t = abs_bits(d);
            m = t > m ? t : m;
        }
    }
    block_max_commit(m, out);
}

// MaxVelocity, stencil.go:319-331: every element of U, V, W, ghosts included.
__global__ void __launch_bounds__(kDiagThreads) k_max_abs3(const double* __restrict__ u_, long long nu,
                                                           const double* __restrict__ v_, long long nv,
                                                           const double* __restrict__ w_, long long nw,
                                                           unsigned long long* out) {
    AF_PTR(const double) AF_RESTRICT f[3] = {view(u_, nu, DK_F64_MAXABS, 0), view(v_, nv, DK_F64_MAXABS, 0),
                                             view(w_, nw, DK_F64_MAXABS, 0)};
    const long long n[3] = {nu, nv, nw};
    unsigned long long m = 0;
    const long long stride = (long long)gridDim.x * kDiagThreads;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        long long i = (long long)blockIdx.x * kDiagThreads + threadIdx.x;
        for (; i + 3 * stride < n[k]; i += 4 * stride) {  // four loads in flight
            const double a = f[k][i], b = f[k][i + stride], c = f[k][i + 2 * stride], d = f[k][i + 3 * stride];
            const unsigned long long p = max(abs_bits(a), abs_bits(b)), q = max(abs_bits(c), abs_bits(d));
            m = max(m, max(p, q));
        }
        for (; i < n[k]; i += stride) m = max(m, abs_bits(f[k][i]));
    }
    block_max_commit(m, out);
}

// KineticEnergy, project.go:238-258.  The reference sums serially; this sums
// each block of rows in a fixed per-thread order and a fixed shuffle tree,
// then the blocks in a fixed tree, so the result depends on the grid only and
// is bit-identical run to run (it differs from the serial sum by rounding).
constexpr int kKeThreads = 256;
// Partial sums at most, and the rows of a block: enough blocks to fill the
// GPU, as the grid alone decides.  Short rows, and planes of fewer rows than
// half of a block's warps, are dealt out cell by cell instead of a row a warp,
// 1024 cells or more to a block.  us a call, a row a warp / so: 1x1000x1000
// 414 / 40, 8x512x512 163 / 52, 16x512x512 188 / 81, 1000x1x1000 77 / 40.
constexpr int kKeMaxPartials = 16384;
inline bool ke_dense(const Geom& g) { return g.NX < 32 || g.NY < kKeThreads / 64; }
inline int ke_rows(const Geom& g) {
    int per = ke_dense(g) ? (1024 + g.NX - 1) / g.NX : kKeThreads / 32;  // a row a warp
    while ((long long)g.NZ * ((g.NY + per - 1) / per) > kKeMaxPartials && per < g.NY) per *= 2;
    return per;
}

__device__ __forceinline__ double block_sum_fixed(double s) {
    __shared__ double sm[kKeThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = dadd(s, __shfl_xor_sync(0xffffffffu, s, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    s = threadIdx.x < kKeThreads / 32 ? sm[threadIdx.x] : 0.0;
    if (threadIdx.x < 32) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = dadd(s, __shfl_xor_sync(0xffffffffu, s, o));
    }
    return s;
}

// Per cell three additions of face pairs (one of them on the integer pipe),
// three exact halvings (exponent) and three fused multiply-adds.
template <bool DENSE>
__global__ void __launch_bounds__(kKeThreads) k_ke_planes(const __grid_constant__ Geom g, const FastDiv fx,
                                                          const double* __restrict__ u_,
                                                          const double* __restrict__ v_,
                                                          const double* __restrict__ w_, int rows,
                                                          double* partials_) {
    const int G = g.G;
    AF_PTR(const double) AF_RESTRICT u = view(u_, g.u.count, DK_F64_KE, 0);
    AF_PTR(const double) AF_RESTRICT v = view(v_, g.v.count, DK_F64_KE, 0);
    AF_PTR(const double) AF_RESTRICT w = view(w_, g.w.count, DK_F64_KE, 0);
    AF_PTR(double) partials = view(partials_, (long long)gridDim.x * gridDim.y, DK_F64_KE, 0);
    const int z = G + (int)blockIdx.x, y0 = (int)blockIdx.y * rows;
    double s = 0.0;
    auto cell = [&](long long iu, long long iv, long long iw) {
        const double uc = half(dadd_int(u[iu], u[iu + 1]));
        const double vc = half(dadd(v[iv], v[iv + g.v.sy]));
        const double wc = half(dadd(w[iw], w[iw + g.w.sz]));
        s = __fma_rn(uc, uc, s);
        s = __fma_rn(vc, vc, s);
        s = __fma_rn(wc, wc, s);
    };
    if (DENSE) {
        const unsigned n = (unsigned)min(rows, g.NY - y0) * (unsigned)g.NX;
        for (unsigned k = threadIdx.x; k < n; k += kKeThreads) {
            const unsigned r = fx.div(k);
            const int x = G + (int)(k - r * fx.d), y = G + y0 + (int)r;
            cell(x + y * g.u.sy + z * g.u.sz, x + y * g.v.sy + z * g.v.sz, x + y * g.w.sy + z * g.w.sz);
        }
    } else {
        for (int r = (int)threadIdx.x >> 5; r < rows && y0 + r < g.NY; r += kKeThreads / 32) {
            const int y = G + y0 + r;
            const long long iu = y * g.u.sy + z * g.u.sz, iv = y * g.v.sy + z * g.v.sz, iw = y * g.w.sy + z * g.w.sz;
            for (int x = G + ((int)threadIdx.x & 31); x < G + g.NX; x += 32) cell(iu + x, iv + x, iw + x);
        }
    }
    s = block_sum_fixed(s);
    if (threadIdx.x == 0) partials[(long long)blockIdx.x * gridDim.y + blockIdx.y] = s;
}

__global__ void __launch_bounds__(kKeThreads) k_ke_final(const double* partials_, int n, double* out) {
    AF_PTR(const double) partials = view(partials_, (long long)n, DK_F64_KE, 0);
    double s = 0.0;
    for (int k = threadIdx.x; k < n; k += kKeThreads) s = dadd(s, partials[k]);
    s = block_sum_fixed(s);
    if (threadIdx.x == 0) *out = s;
}

// Self-test of the exact /6 forms against IEEE division over PCG32-random
// doubles: uniform significands, exponents spread over the whole range
// (including subnormals, zero, Inf and NaN patterns).  Counts mismatching
// bit patterns (NaNs compare by NaN-ness).
__global__ void k_selftest_div6(unsigned long long n, unsigned long long seed, unsigned long long* bad) {
    unsigned long long local = 0;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        // splitmix64 of (seed, i): every input independent of the launch shape
        unsigned long long z = seed + (i + 1) * 0x9E3779B97F4A7C15ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        const double x = __longlong_as_double((long long)z);
        const double ref = x / 6.0;
        const double a = div6_int(x), c = div6(x);
        const bool ok_a = __double_as_longlong(a) == __double_as_longlong(ref) || (isnan(a) && isnan(ref));
        const bool ok_c = __double_as_longlong(c) == __double_as_longlong(ref) || (isnan(c) && isnan(ref));
        local += (ok_a ? 0 : 1) + (ok_c ? 0 : 1);
    }
    if (local) atomicAdd(bad, local);
}

// Eight independent DFMA chains per thread: issue-rate bound, not latency bound.
constexpr int kRateIters = 2048, kRateChains = 8;
__global__ void k_fp64_rate(double* out, double seed) {
    double a[kRateChains];
#pragma unroll
    for (int c = 0; c < kRateChains; ++c) a[c] = seed + threadIdx.x + c;
    const double m = 0.999999999, k = 1e-9;
    for (int i = 0; i < kRateIters; ++i) {
#pragma unroll
        for (int c = 0; c < kRateChains; ++c) a[c] = __fma_rn(a[c], m, k);
    }
    double s = 0;
#pragma unroll
    for (int c = 0; c < kRateChains; ++c) s += a[c];
    if (s == 12345.678) out[0] = s;  // keeps the chains live
}

}  // namespace

// dadd_int against __dadd_rn on pairs built to hit every path: random bit
// patterns, close exponents (cancellation), exact ties, far exponents.
__global__ void k_selftest_dadd(unsigned long long n, unsigned long long seed, unsigned long long* bad) {
    unsigned long long local = 0;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        auto mix = [](unsigned long long z) {
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
            z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
            return z ^ (z >> 31);
        };
        const unsigned long long r1 = mix(seed + (2 * i + 1) * 0x9E3779B97F4A7C15ull);
        const unsigned long long r2 = mix(seed + (2 * i + 2) * 0x9E3779B97F4A7C15ull);
        const unsigned long long ua = r1;
        unsigned long long ub;
        switch (i & 3) {
        case 0: ub = r2; break;  // independent
        case 1: {                // exponent within +-60 of a's, random sign
            const long long ea = (long long)((ua >> 52) & 0x7FF);
            long long eb = ea + (long long)(r2 % 121) - 60;
            eb = eb < 0 ? 0 : (eb > 0x7FF ? 0x7FF : eb);
            ub = (r2 & 0x8000000000000000ull) | ((unsigned long long)eb << 52) | ((r2 >> 11) & 0xFFFFFFFFFFFFFull);
            break;
        }
        case 2: {                // same exponent and close significand: cancellation
            ub = (r2 & 0x8000000000000000ull) | (ua & 0x7FF0000000000000ull) |
                 ((ua + (r2 & 0xFFF) - 0x800) & 0xFFFFFFFFFFFFFull);
            break;
        }
        default: {               // half an ulp of a (a tie) times a small power of two
            const unsigned long long ea = (ua >> 52) & 0x7FF;
            const unsigned long long sh = 53 + (r2 & 3);
            const unsigned long long eb = ea > sh ? ea - sh : 0;
            ub = (r2 & 0x8000000000000000ull) | (eb << 52) | (r2 & 0xFull);
            break;
        }
        }
        const double a = __longlong_as_double((long long)ua), b = __longlong_as_double((long long)ub);
        const double ref = __dadd_rn(a, b), got = dadd_int(a, b), got2 = dsub_int(a, b), ref2 = __dsub_rn(a, b);
        const bool ok = __double_as_longlong(got) == __double_as_longlong(ref) || (isnan(got) && isnan(ref));
        const bool ok2 = __double_as_longlong(got2) == __double_as_longlong(ref2) || (isnan(got2) && isnan(ref2));
        local += (ok ? 0 : 1) + (ok2 ? 0 : 1);
    }
    if (local) atomicAdd(bad, local);
}

bool selftest_dadd(unsigned long long n, unsigned long long seed, unsigned long long* mismatches) {
    unsigned long long* bad = nullptr;
    if (cudaMalloc(&bad, sizeof *bad) != cudaSuccess) return false;
    cudaMemset(bad, 0, sizeof *bad);
    k_selftest_dadd<<<152 * 8, 256>>>(n, seed, bad);
    const bool ok = cudaMemcpy(mismatches, bad, sizeof *bad, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(bad);
    return ok && cudaGetLastError() == cudaSuccess;
}

bool selftest_div6(unsigned long long n, unsigned long long seed, unsigned long long* mismatches) {
    unsigned long long* bad = nullptr;
    if (cudaMalloc(&bad, sizeof *bad) != cudaSuccess) return false;
    cudaMemset(bad, 0, sizeof *bad);
    k_selftest_div6<<<152 * 8, 256>>>(n, seed, bad);
    const bool ok = cudaMemcpy(mismatches, bad, sizeof *bad, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(bad);
    return ok && cudaGetLastError() == cudaSuccess;
}

bool measure_fp64_rate(double* fma_per_s) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
    double* out = nullptr;
    if (cudaMalloc(&out, sizeof(double)) != cudaSuccess) return false;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    const int blocks = sms * 8, threads = 256;
    k_fp64_rate<<<blocks, threads>>>(out, 1.0);  // warm-up
    cudaEventRecord(a);
    const int reps = 5;
    for (int r = 0; r < reps; ++r) k_fp64_rate<<<blocks, threads>>>(out, 1.0 + r);
    cudaEventRecord(b);
    bool ok = cudaEventSynchronize(b) == cudaSuccess;
    float ms = 0;
    ok = ok && cudaEventElapsedTime(&ms, a, b) == cudaSuccess;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(out);
    if (!ok || ms <= 0) return false;
    *fma_per_s = (double)blocks * threads * kRateIters * kRateChains * reps / (ms * 1e-3);
    return true;
}

namespace {
}  // namespace

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
void launch_velocity_bc(const Geom& g, double* u, double* v, double* w, Status* st, int gate, cudaStream_t s) {
    long long mx = 0;
    const int N[3][3] = {{g.NX, g.NY, g.NZ}, {g.NY, g.NX, g.NZ}, {g.NZ, g.NX, g.NY}};  // Nn, N1, N2 per component
    for (const auto& n : N) {
        mx = std::max(mx, 2ll * n[1] * n[2]);
        mx = std::max(mx, 2ll * (n[0] + 1) * n[2]);
        mx = std::max(mx, 2ll * (n[0] + 1) * (n[1] + 2));
    }
    dim3 grid(cdiv(mx, 256), 9);
    launch_pdl(k_velocity_bc, grid, dim3(256), 0, s, g, u, v, w, st, gate);
}

void launch_sweep_fp64(const Geom& g, int axis, const Fields& f, double dt, double invH, double lam, Status* st,
                       int phase, cudaStream_t s) {
    SweepArgs a;
    a.u = view((const double*)f.u, g.u.count, DK_F64_SWEEP, 0);
    a.v = view((const double*)f.v, g.v.count, DK_F64_SWEEP, 0);
    a.w = view((const double*)f.w, g.w.count, DK_F64_SWEEP, 0);
    a.tu = view(f.t0, g.u.count, DK_F64_SWEEP, 0);
    a.tv = view(f.t1, g.v.count, DK_F64_SWEEP, 0);
    a.tw = view(f.t2, g.w.count, DK_F64_SWEEP, 0);
    a.du = g.u; a.dv = g.v; a.dw = g.w;
    a.NX = g.NX; a.NY = g.NY; a.NZ = g.NZ; a.G = g.G;
    a.set_scheme(axis, dt, invH, lam);
    a.st = st; a.phase = phase;
    const dim3 block(32, 8), grid = face_grid(g, block);
    launch_pdl(axis == 0 ? k_sweep_fp64<0> : (axis == 1 ? k_sweep_fp64<1> : k_sweep_fp64<2>), grid, block, 0, s, a);
}

void launch_maccormack_fp64(const Geom& g, int axis, const Fields& f, const Fields& fwd, double dt, double invH,
                            double lam, Status* st, int phase, cudaStream_t s) {
    // Forward step: the reference sweep without diffusion, into fwd.t0..t2.
    launch_sweep_fp64(g, axis, fwd, dt, invH, 0.0, st, phase, s);
    SweepArgs a;
    a.u = view((const double*)f.u, g.u.count, DK_F64_SWEEP, 0);
    a.v = view((const double*)f.v, g.v.count, DK_F64_SWEEP, 0);
    a.w = view((const double*)f.w, g.w.count, DK_F64_SWEEP, 0);
    a.tu = view(f.t0, g.u.count, DK_F64_SWEEP, 0);
    a.tv = view(f.t1, g.v.count, DK_F64_SWEEP, 0);
    a.tw = view(f.t2, g.w.count, DK_F64_SWEEP, 0);
    a.du = g.u; a.dv = g.v; a.dw = g.w;
    a.NX = g.NX; a.NY = g.NY; a.NZ = g.NZ; a.G = g.G;
    a.set_scheme(axis, dt, invH, lam);
    a.st = st; a.phase = phase;
    const dim3 block(32, 8), grid = face_grid(g, block);
    launch_pdl(axis == 0 ? k_maccormack_fp64<0> : (axis == 1 ? k_maccormack_fp64<1> : k_maccormack_fp64<2>), grid, block,
               0, s, a, fwd.t0, fwd.t1, fwd.t2);
}

void launch_divergence_fp64(const Geom& g, const Fields& f, const Split* split, double scale, double h2, Status* st,
                            int gate, cudaStream_t s) {
    const dim3 block(32, 8), grid(cdiv(g.NX, 32), cdiv(g.NY, 8), g.NZ);
    launch_pdl(k_divergence_fp64, grid, block, 0, s, g, f.u, f.v, f.w, f.div, split ? *split : Split{}, split ? 1 : 0,
               exact::mul_const(scale), exact::mul_const(h2), st, gate);
}

void launch_split_from_div(const Geom& g, const double* div, const Split& split, double h2, cudaStream_t s) {
    const dim3 block(32, 8), grid(cdiv(g.NX, 32), cdiv(g.NY, 8), g.NZ);
    k_split_from_div<<<grid, block, 0, s>>>(g, div, split, exact::mul_const(h2));
}

// Integer-pipe share of the red-black chain.  Of the update's six additions
// the first and the last (the subtraction, which feeds the division unpacked)
// run there: at 256^3 a launch takes 101 us with none, 86 with either, 77
// with both -- both pipes then about 70 % busy -- 88 with a third and 140
// with all six (the logic pipe bounds).
constexpr int kRbEmu = 0x21;

void launch_rbgs_fp64(const Split& split, int color, cudaStream_t s) {
    const dim3 grid(cdiv((long long)split.hx * split.NY, 128), split.NZ);
    launch_pdl(k_rbgs_fp64<kRbEmu>, grid, dim3(128), 0, s, split, color);
}

// The cluster kernel for this grid, its cells a thread in *nc; null where the
// grid is too large for it or the device cannot hold such a cluster.
typedef void (*RbClusterKernel)(const Split, long long);
static RbClusterKernel rbgs_cluster_kernel(const Split& S, size_t* smem) {
    if ((long long)S.NX * S.NY * S.NZ > kRbMaxCells) return nullptr;
    const int rows = (S.NY * S.NZ + kRbCluster - 1) / kRbCluster, n = rows * S.hx;
    *smem = (size_t)2 * n * sizeof(double);
    const RbClusterKernel k = n <= kRbThreads ? k_rbgs_cluster<1> : (n <= 2 * kRbThreads ? k_rbgs_cluster<2> : nullptr);
    if (!k) return nullptr;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return k;
}

bool launch_rbgs_all_fp64(const Split& split, long long pairs, cudaStream_t s) {
    size_t smem = 0;
    const RbClusterKernel k = rbgs_cluster_kernel(split, &smem);
    if (!k) return false;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kRbCluster);
    cfg.blockDim = dim3(kRbThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kRbCluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess || clusters < 1) {
        cudaGetLastError();
        return false;
    }
    if (cudaLaunchKernelEx(&cfg, k, split, pairs) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return true;
}

void launch_join_fp64(const Geom& g, const Split& split, double* p, Status* st, int gate, cudaStream_t s) {
    const dim3 block(64, 4), grid(cdiv(g.p.nx, 64), cdiv(g.p.ny, 4), g.p.nz);
    launch_pdl(k_join_fp64, grid, block, 0, s, g, split, p, st, gate);
}

void launch_pressure_bc_fp64(const Geom& g, double* p, Status* st, int gate, cudaStream_t s) {
    long long mx = std::max(2ll * g.NY * g.NZ, std::max(2ll * (g.NX + 2) * g.NZ, 2ll * (g.NX + 2) * (g.NY + 2)));
    dim3 grid(cdiv(mx, 256), 3);
    k_pressure_bc<<<grid, 256, 0, s>>>(g, p, st, gate);
}

void launch_gradient_fp64(const Geom& g, const Fields& f, double scale, Status* st, int gate, cudaStream_t s) {
    const dim3 grid(cdiv((long long)(g.NX + 1) * (g.NY + 1), 256), g.NZ + 1);
    launch_pdl(k_gradient_fp64, grid, dim3(256), 0, s, g, FastDiv((unsigned)(g.NX + 1)), f.p, f.u, f.v, f.w,
               exact::mul_const(scale), st, gate);
}

void launch_step_tick(Status* st, cudaStream_t s) { launch_pdl(k_step_tick, dim3(1), dim3(1), 0, s, st); }

void launch_max_divergence(const Geom& g, const double* u, const double* v, const double* w, unsigned long long* out,
                           cudaStream_t s) {
    k_max_divergence<<<dim3(cdiv(g.NY, kDiagRows), g.NZ), kDiagThreads, 0, s>>>(g, u, v, w, out);
}

void launch_max_abs3(const double* u, long long nu, const double* v, long long nv, const double* w, long long nw,
                     unsigned long long* out, cudaStream_t s) {
    const long long n = std::max(nu, std::max(nv, nw));
    const unsigned blocks = (unsigned)std::min<long long>(cdiv(n, kDiagThreads), 152 * 8);
    k_max_abs3<<<blocks, kDiagThreads, 0, s>>>(u, nu, v, nv, w, nw, out);
}

bool fp64_debug_bounds(unsigned long long* first, unsigned* count, bool reset) {
#if AEROFLUX_DEBUG_BOUNDS
    if (cudaMemcpyFromSymbol(first, g_dbg_first, sizeof *first) != cudaSuccess ||
        cudaMemcpyFromSymbol(count, g_dbg_count, sizeof *count) != cudaSuccess)
        return false;
    if (reset) {
        const unsigned long long none = ~0ull;
        const unsigned zero = 0;
        cudaMemcpyToSymbol(g_dbg_first, &none, sizeof none);
        cudaMemcpyToSymbol(g_dbg_count, &zero, sizeof zero);
    }
#else
    (void)reset;
    *first = ~0ull;
    *count = 0;
#endif
    return true;
}

int kinetic_energy_partials(const Geom& g) { return g.NZ * (int)cdiv(g.NY, ke_rows(g)); }

void launch_kinetic_energy(const Geom& g, const double* u, const double* v, const double* w, double* partials,
                           double* out, cudaStream_t s) {
    const int rows = ke_rows(g);
    const dim3 grid(g.NZ, cdiv(g.NY, rows));
    const auto k = ke_dense(g) ? k_ke_planes<true> : k_ke_planes<false>;
    k<<<grid, kKeThreads, 0, s>>>(g, FastDiv((unsigned)g.NX), u, v, w, rows, partials);
    k_ke_final<<<1, kKeThreads, 0, s>>>(partials, (int)(grid.x * grid.y), out);
}

}  // namespace af

// ---------------------------------------------------------------------------
// Kinetic energy without any allocation.
//
// Some callers cannot allocate device memory while they run: hosts that hand
// all device memory to their own pool up front and forbid cudaMalloc
// afterwards, and latency-bound loops that cannot afford the implicit
// device-wide synchronisation of cudaMalloc/cudaFree.  This entry point runs
// the same fixed-order reduction as af_kinetic_energy over caller-owned
// device fields, with its scratch (the partial sums plus the final
// sum) in the file-scope array below.  Every GPU that loads the library holds
// the array until the process exits.
// ---------------------------------------------------------------------------
namespace af {
namespace {

constexpr int kNoAllocMaxPlanes = kKeMaxPartials;  // 128 KiB of partials
static __device__ __align__(256) double g_ke_scratch[kNoAllocMaxPlanes + 1];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
double* g_scratch_ptr[kMaxDevices] = {};

// Device address of g_ke_scratch on the current device, resolved once per
// device (host code only sees a host-side stand-in for the symbol).
cudaError_t scratch_address(int dev, double** out) {
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        cudaError_t rc = cudaGetSymbolAddress(&p, g_ke_scratch);
        if (rc != cudaSuccess) return rc;
        g_scratch_ptr[dev] = static_cast<double*>(p);
    }
    *out = g_scratch_ptr[dev];
    return cudaSuccess;
}

void put(char* err, size_t errlen, const char* msg) {
    if (err && errlen) snprintf(err, errlen, "%s", msg);
}

}  // namespace
}  // namespace af

extern "C" int af_kinetic_energy_noalloc(const af_config* cfg, const double* u, const double* v, const double* w,
                                         void* stream, double* out, char* err, size_t errlen) {
    using namespace af;
    if (!cfg || !u || !v || !w || !out) {
        put(err, errlen, "aeroflux: kinetic energy without allocation: NULL argument");
        return AF_ERR_ARG;
    }
    if (cfg->nx < 1 || cfg->ny < 1 || cfg->nz < 1 || cfg->ghost < 1 || !(cfg->h > 0) || std::isinf(cfg->h)) {
        put(err, errlen, "aeroflux: kinetic energy without allocation: extents, ghost and h must be positive");
        return AF_ERR_ARG;
    }
    // The kernels index planes and rows in int: extents and the ghost stay
    // below 2^20 so every padded coordinate fits.
    if (cfg->nz > kNoAllocMaxPlanes || cfg->nx >= (1 << 20) || cfg->ny >= (1 << 20) || cfg->ghost >= (1 << 20)) {
        char m[256];
        snprintf(m, sizeof m,
                 "aeroflux: kinetic energy without allocation supports at most %d z-planes (and nx, ny, ghost "
                 "< 2^20), got %lldx%lldx%lld ghost %lld",
                 kNoAllocMaxPlanes, (long long)cfg->nx, (long long)cfg->ny, (long long)cfg->nz,
                 (long long)cfg->ghost);
        put(err, errlen, m);
        return AF_ERR_ARG;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        put(err, errlen, "aeroflux: kinetic energy without allocation: no usable current device");
        return AF_ERR_CUDA;
    }
    double* scratch = nullptr;
    cudaError_t rc = scratch_address(dev, &scratch);
    if (rc != cudaSuccess) {
        put(err, errlen, cudaGetErrorString(rc));
        return AF_ERR_CUDA;
    }
    Geom g{};
    g.NX = (int)cfg->nx;
    g.NY = (int)cfg->ny;
    g.NZ = (int)cfg->nz;
    g.G = (int)cfg->ghost;
    const long long cx = cfg->nx + 2 * cfg->ghost, cy = cfg->ny + 2 * cfg->ghost;
    g.u.sy = cx + 1;
    g.u.sz = (cx + 1) * cy;
    g.v.sy = cx;
    g.v.sz = cx * (cy + 1);
    g.w.sy = cx;
    g.w.sz = cx * cy;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // Every partial the final pass reads is rewritten by this call, so the
    // array needs no clearing; concurrent calls on the GPU share it and race.
    launch_kinetic_energy(g, u, v, w, scratch, scratch + kNoAllocMaxPlanes, s);
    double sum = 0;
    if ((rc = cudaGetLastError()) != cudaSuccess ||
        (rc = cudaMemcpyAsync(&sum, scratch + kNoAllocMaxPlanes, sizeof sum, cudaMemcpyDeviceToHost, s)) !=
            cudaSuccess ||
        (rc = cudaStreamSynchronize(s)) != cudaSuccess) {
        put(err, errlen, cudaGetErrorString(rc));
        return AF_ERR_CUDA;
    }
    const double h = cfg->h;
    const double vol = h * h * h;
    *out = 0.5 * sum * vol;
    return AF_OK;
}
