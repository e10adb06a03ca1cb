// af_batch.cu -- batched mixed-precision fractional step.
//
// Many independent grids (slots) of uneven sizes step together.  Every stage
// is ONE persistent launch over a device-side work list: per stage, a prefix
// array gives each slot's number of tiles, a block finds its slot by binary
// search and processes one tile of that slot's iteration space, and the grid
// (a fixed multiple of the SM count) strides over all tiles.  Because the
// work lists live in device memory, slots can be assigned, released,
// activated and deactivated between steps without recapturing the step
// graph (continuous batching); the graph is recaptured only when the
// deepest multigrid hierarchy grows or the launch shapes are retuned.
//
// Arithmetic: binary32 advection/diffusion with integer-pipe conversions
// (af_cells.cuh); binary64 divergence, residual, pressure accumulator,
// gradient and BCs (bit-identical to the FP64 form's cells); binary32
// multigrid V-cycles with over-relaxed red-black smoothing inside binary64
// refinement.  The
// refinement loop is one WHILE node for the whole batch: it runs while any
// slot is unconverged, and a converged slot skips every later pass, so each
// slot performs exactly the passes it performs alone.  Every cell's result is
// independent of the tile that computes it, and reductions are exact maxima
// or fixed trees over one slot, so a slot's bits do not depend on the other
// slots or on the tuned launch shapes.
#include "af_batch.h"
#include "af_cells.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

namespace af {
namespace {

using namespace cells;

constexpr int kMaxLev = 16;
constexpr int kCoarseThreads = 512;
constexpr int kCoarseMax = 4096;

struct Lvl {
    int nx, ny, nz;
    float wx, wy, wz;   // (h0 / h_axis)^2
    int cx, cy, cz;     // 1 when the axis coarsens into the next level
    float* e;
    float* r;
    FastDiv fnx, fny, fhx;  // nx, ny, (nx+1)/2
    float* e2;              // second buffer of the fused red-black pair (levels below the tail)
    FastDiv ftx;            // fused-pair wide tiles along x
    FastDiv fty[3];         // fused-pair tiles along y, per tile variant (kPairVarTY)
    int nxw;                // 64 x the wide pair tiles along x; a narrow tile column covers nxw .. nx-1
    // Marching pair (kb_smooth_march), per block size (kMarchT): the quads of
    // a tile column (0 when the level cannot run it) and of its loaded rows,
    // the output rows of a tile, the tile columns and the tiles along y.
    struct March {
        int w, q, rows;
        FastDiv fq, fcol, fty;
    } march[3];
    int v4;  // every axis coarsens, rows of whole quads, e, r and the next level's on 16-byte boundaries
};

struct Ctl {
    unsigned long long maxr_bits;  // max |r| of the current pass (binary64 bits)
    unsigned int passes;
    unsigned int stopped;
    double last_div;               // dt/(rho h^2) * max|r| at the last check
    unsigned int nv;               // V-cycles the next pass runs (0: all of them)
    double vfac;                   // measured max|div| reduction per V-cycle (0: none yet); kept across projections
    unsigned int vtotal;           // V-cycles the current projection has run
};

// Whether the multigrid kernels of V-cycle vc of a pass skip a slot.
__device__ __forceinline__ bool mg_off(const Ctl& c, int vc) { return c.stopped || (c.nv && (unsigned)vc >= c.nv); }
// ctl[n] (n = the batch's capacity) is the batch's own record: its nv is the
// number of V-cycles some slot runs in the current pass, so a V-cycle no
// slot runs returns at once instead of walking the slots' tiles.
__device__ __forceinline__ bool vc_idle(const Ctl* ctl, int n, int vc) { return (unsigned)vc >= ctl[n].nv; }

struct InstDev {
    Geom g;
    double* slot[8];   // arena field slots P, U, V, W, Div, Tmp0, Tmp1, Tmp2
    double* b;         // h^2 * Div, P-shaped
    float dt_invh;     // (DT/2)/H for the sweeps
    float lam;         // nu*(DT/2)/H^2
    exact::MulC div_scale;   // rho/(DT*H)
    exact::MulC h2;          // H^2
    exact::MulC grad_scale;  // DT/(rho*H)
    double res_scale;   // DT/(rho*H^2): max|div| per unit residual
    double thresh;      // 0.5 * div_tol
    unsigned max_refine;
    int nlev;
    int coarse_sweeps;  // sweeps of the coarsest solve inside the tail V-cycle
    int tail;           // first level of the one-block tail V-cycle; -1: coarsest too large, smoothed instead
    int tail_floats;    // shared-memory floats of the tail levels (e and r)
    int res_lg;         // log2 of the planes a thread of the residual takes (at most kResMaxLg)
    int parity;         // 1 when U/V/W live in the Tmp slots
    int active;
    FastDiv fpx, fpy;        // padded P extents
    FastDiv ffx, ffy, ffz;   // NX+1, NY+1, NZ+1 (the face box)
    FastDiv fnx, fny;        // NX, NY
    float* sh[3];            // binary32 shadow of the current U, V, W (the sweeps' taps)
    int shp[3];              // row pitch of each shadow (floats): its padded x extent rounded up to 4
    int shq[4];              // shadow conversion: prefix of the components' (row, quad) counts
    FastDiv fsq[3];          // quads per shadow row
    const CUtensorMap* tmap; // 12 tensor maps over the shadows: [component][role], role 0-2 the staged
                             // tile of a sweep along axis 0-2, role 3 the axis-velocity tile
    int sw_tiles;            // staged sweep: work items (3 components x the spatial tiles)
    FastDiv swx, swy;        // staged sweep: spatial tiles along x and along y
    int warm;                // 1: a projection starts from the last pressure, 0: from zero
    int bc_off[10];          // velocity BC write sets: prefix of the nine (component, set) counts
    FastDiv bcd[9][2];       // their index decoding's divisors (bc_cell_div's d1, d2)
    Lvl lev[kMaxLev];
};

// Stage ids.  Level stages take kMaxLev consecutive ids.
enum {
    S_BC = 0, S_SWEEP, S_DIV, S_INT, S_PBC, S_GRAD, S_COARSE, S_SHADOW, S_CORR,
    S_SMOOTH = 9,
    S_RESTRICT = S_SMOOTH + kMaxLev,
    S_PROLONG = S_RESTRICT + kMaxLev,
    S_BIGCOARSE = S_PROLONG + kMaxLev,
    S_PAIR = S_BIGCOARSE + kMaxLev,
    S_PAIRN = S_PAIR + kMaxLev,
    S_SWEEPT = S_PAIRN + kMaxLev,
    S_MARCH = S_SWEEPT + 1,
    S_COUNT = S_MARCH + kMaxLev
};

struct Shape {
    int tpb = 256;   // threads per block
    int ept = 1;     // elements per thread
    int bpsm = 8;    // persistent blocks per SM
    int var = 0;     // fused-pair stages: the tile variant (kPairVarTY, kPairVarTZ)
};

// A stage's device work list: prefix[0..n] of tiles per slot.
struct Tab {
    const int* prefix;
    int n;
    int ept;
};

// Every lane of a warp asks for the same item (callers are block-uniform
// and blocks are whole warps): lane 0 searches, the warp shares the result.
__device__ __forceinline__ int find_slot(const int* prefix, int n, int item) {
    int lo = 0;
    if ((threadIdx.x & 31) == 0) {
        int hi = n;  // prefix[lo] <= item < prefix[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (prefix[mid] <= item) lo = mid;
            else hi = mid;
        }
    }
    return __shfl_sync(0xffffffffu, lo, 0);
}

// The start of every batched kernel.  Its launch may overlap the end of the
// kernel before it (launch_pdl): the block waits before it reads anything a
// kernel wrote.  What no kernel writes -- with one slot, its record (`bytes`
// from `off`) and work list -- it fetches into its L1 before it waits (with
// many slots the search for the block's own costs as much as it saves).
// Measured per Step, launches one after the other / overlapped: 16^3 0.690 /
// 0.678 ms, 48x32x64 1.56 / 1.50, 128^3 2.755 / 2.69, 256^3 9.19 / 9.12, the
// 256-grid batch unchanged.
__device__ __forceinline__ void touch(const void* p) {
    unsigned v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
}
__device__ __forceinline__ void begin(const InstDev* inst, const Tab& tab, size_t off, size_t bytes) {
    if (tab.n == 1) {
        const char* p = (const char*)inst + off;
        if (threadIdx.x * 128u < bytes) touch(p + threadIdx.x * 128u);
        if (threadIdx.x == 0) touch(tab.prefix);
    }
    pdl_wait();
    // A grid that takes at most a quarter of the SMs' threads leaves the next
    // kernel's blocks room to get this far while it runs.
    if (gridDim.x * blockDim.x <= 152u * 512u) pdl_trigger();
}
// The record up to its levels, or level l (and the next).
__device__ __forceinline__ void begin_slot(const InstDev* inst, const Tab& tab) {
    begin(inst, tab, 0, offsetof(InstDev, lev) + sizeof(Lvl));
}
__device__ __forceinline__ void begin_level(const InstDev* inst, const Tab& tab, int l, int levels) {
    begin(inst, tab, offsetof(InstDev, lev) + l * sizeof(Lvl), levels * sizeof(Lvl));
}

// Loop over this block's tiles; `s` is the slot, `first` the first element
// of the tile; body sees element index `el` (< the slot's count, checked by
// the body).
#define FOR_TILES(tab)                                                                   \
    for (int item = blockIdx.x, total = (tab).prefix[(tab).n]; item < total; item += gridDim.x) { \
        const int s = find_slot((tab).prefix, (tab).n, item);                            \
        const long long first = (long long)(item - (tab).prefix[s]) * blockDim.x * (tab).ept;
#define FOR_ELEMS(tab) \
        for (int k_ = 0; k_ < (tab).ept; ++k_) {      \
            const long long el = first + (long long)k_ * blockDim.x + threadIdx.x;
#define END_ELEMS }
#define END_TILES }

__device__ __forceinline__ double* cur(const InstDev& I, int field, int parity) {
    const int p = parity ^ I.parity;
    if (!p || field == 0 || field == 4) return I.slot[field];
    return I.slot[field <= 3 ? field + 4 : field - 4];
}

// --- counts of each stage's iteration space -------------------------------
__host__ __device__ inline long long bc_count(const Geom& g) {
    const long long N[3][3] = {{g.NX, g.NY, g.NZ}, {g.NY, g.NX, g.NZ}, {g.NZ, g.NX, g.NY}};
    long long c = 0;
    for (int k = 0; k < 3; ++k) c += 2 * N[k][1] * N[k][2] + 2 * (N[k][0] + 1) * N[k][2] + 2 * (N[k][0] + 1) * (N[k][1] + 2);
    return c;
}
__host__ __device__ inline long long face_box(const Geom& g) {
    return (long long)(g.NX + 1) * (g.NY + 1) * 3 * (g.NZ + 1);
}
__host__ __device__ inline long long pbc_count(const Geom& g) {
    return 2ll * g.NY * g.NZ + 2ll * (g.NX + 2) * g.NZ + 2ll * (g.NX + 2) * (g.NY + 2);
}
constexpr int kResMaxLg = 3;
constexpr int kCorrZ = 4;  // cells of a column a thread of the correction takes
__host__ __device__ inline long long correct_items(const Geom& g) {
    return (long long)g.NX * g.NY * ((g.NZ + kCorrZ - 1) / kCorrZ);
}
__host__ __device__ inline long long residual_items(const Geom& g, int lg) {
    return (long long)g.NX * g.NY * ((g.NZ + (1 << lg) - 1) >> lg);
}
__host__ __device__ inline long long lvl_cells(const Lvl& L) { return (long long)L.nx * L.ny * L.nz; }

// --- binary64 stages (bit-identical to the FP64 form's cells) -------------
__global__ void kb_bc(const InstDev* inst, Status* st, Tab tab, int parity, int gate) {
    begin_slot(inst, tab);
    FOR_TILES(tab)
    const InstDev& I = inst[s];
    if (gated(&st[s], gate)) continue;
    AF_PTR(double) u = view(cur(I, 1, parity), I.g.u.count, DK_BC, s);
    AF_PTR(double) v = view(cur(I, 2, parity), I.g.v.count, DK_BC, s);
    AF_PTR(double) w = view(cur(I, 3, parity), I.g.w.count, DK_BC, s);
    int off[10];  // the offsets in registers: no reload per element
#pragma unroll
    for (int j = 0; j < 10; ++j) off[j] = I.bc_off[j];
    FOR_ELEMS(tab)
    if (el >= off[9]) break;
    // Write set k = 3 * component + set holds elements bc_off[k] ..
    // bc_off[k+1]-1 (bc_set_count in that order).
    const int e = (int)el;
    int k = 0, base = 0;
#pragma unroll
    for (int j = 1; j < 9; ++j)
        if (e >= off[j]) {
            k = j;
            base = off[j];
        }
    const int comp = k / 3;
    bc_cell_div(bc_comp(I.g, comp, u, v, w), I.g.G, k - 3 * comp, (unsigned)(e - base), I.bcd[k][0], I.bcd[k][1]);
    END_ELEMS
    END_TILES
}

__global__ void kb_div(const InstDev* inst, Status* st, Tab tab, int parity, int gate) {
    begin_slot(inst, tab);
    FOR_TILES(tab)
    const InstDev& I = inst[s];
    if (gated(&st[s], gate)) continue;
    const Geom& g = I.g;
    const long long n = (long long)g.p.nx * g.p.ny * g.p.nz;
    FOR_ELEMS(tab)
    if (el >= n) break;
    const unsigned e = (unsigned)el, r = I.fpx.div(e), z = I.fpy.div(r);
    div_cell(g, view((const double*)cur(I, 1, parity), g.u.count, DK_DIV, s),
             view((const double*)cur(I, 2, parity), g.v.count, DK_DIV, s),
             view((const double*)cur(I, 3, parity), g.w.count, DK_DIV, s), view(I.slot[0], g.p.count, DK_DIV, s),
             view(I.slot[4], g.p.count, DK_DIV, s), view(I.b, g.p.count, DK_DIV, s), I.div_scale, I.h2, !I.warm,
             (int)(e - r * g.p.nx), (int)(r - z * g.p.ny), (int)z);
    END_ELEMS
    END_TILES
}

__global__ void kb_pbc(const InstDev* inst, Status* st, Tab tab, int gate) {
    begin_slot(inst, tab);
    FOR_TILES(tab)
    const InstDev& I = inst[s];
    if (gated(&st[s], gate)) continue;
    const Geom& g = I.g;
    const long long c0 = pbc_set_count(g, 0), c1 = pbc_set_count(g, 1), n = pbc_count(g);
    FOR_ELEMS(tab)
    if (el >= n) break;
    AF_PTR(double) p = view(I.slot[0], g.p.count, DK_PBC, s);
    if (el < c0) pbc_cell(g, p, 0, el);
    else if (el < c0 + c1) pbc_cell(g, p, 1, el - c0);
    else pbc_cell(g, p, 2, el - c0 - c1);
    END_ELEMS
    END_TILES
}

// subtractGradient, a thread per cell of the face box (grad_cell), the slot's
// record in registers (read again a tile: 265 instead of 228 us at 256^3; a
// thread a face: 311).
// scratch = 1 (the autotuner's timing runs) stores the new values into the
// Tmp fields instead, so timing leaves the slots' velocities untouched.
__global__ void kb_grad(const InstDev* inst, Status* st, Tab tab, int parity, int gate, int scratch) {
    begin_slot(inst, tab);
    int held = -1;  // the slot whose record is in registers
    Geom g{};
    exact::MulC scale{};
    FastDiv fx, fy;
    const double* pp = nullptr;
    double *pf[3] = {}, *po[3] = {};
    bool off = true;
    FOR_TILES(tab)
    if (s != held) {
        held = s;
        const InstDev& I = inst[s];
        off = gated(&st[s], gate);
        g = I.g, scale = I.grad_scale, fx = I.ffx, fy = I.ffy, pp = I.slot[0];
        for (int c = 0; c < 3; ++c) {
            pf[c] = cur(I, 1 + c, parity);
            po[c] = scratch ? cur(I, 5 + c, parity) : pf[c];
        }
    }
    if (off) continue;
    const unsigned n = fx.d * fy.d * (unsigned)(g.NZ + 1);
    FOR_ELEMS(tab)
    if (el >= n) break;
    const unsigned e = (unsigned)el, r = fx.div(e), z = fy.div(r);
    grad_cell(g, view(pp, g.p.count, DK_GRAD, s), view((const double*)pf[0], g.u.count, DK_GRAD, s),
              view((const double*)pf[1], g.v.count, DK_GRAD, s), view((const double*)pf[2], g.w.count, DK_GRAD, s),
              view(po[0], g.u.count, DK_GRAD, s), view(po[1], g.v.count, DK_GRAD, s),
              view(po[2], g.w.count, DK_GRAD, s), scale, g.G + (int)(e - r * fx.d), g.G + (int)(r - z * fy.d),
              g.G + (int)z);
    END_ELEMS
    END_TILES
}

// binary32 shadow of the current U, V, W (every element, ghosts included),
// converted once per sweep instead of once per tap.  A shadow row holds the
// field row's nx values and is padded to a multiple of four floats (the row
// pitch shp), so rows start on 16-byte boundaries and a TMA tensor map can
// describe the shadow.  A thread converts four consecutive elements of one
// row and stores them with one 16-byte store (padding: zeros).
__global__ void kb_shadow(const InstDev* inst, Tab tab, int parity) {
    begin_slot(inst, tab);
    FOR_TILES(tab)
    const InstDev& I = inst[s];
    const long long n = I.shq[3];
    FOR_ELEMS(tab)
    if (el >= n) break;
    const int e = (int)el;
    const int f = e < I.shq[1] ? 0 : (e < I.shq[2] ? 1 : 2);
    const unsigned r = (unsigned)(e - I.shq[f]);
    const unsigned row = I.fsq[f].div(r), q = r - row * I.fsq[f].d;
    const Dims& d = f == 0 ? I.g.u : (f == 1 ? I.g.v : I.g.w);
    AF_PTR(const double) src =
        view((const double*)cur(I, 1 + f, parity), d.count, DK_SHADOW, s) + ((long long)row * d.nx + 4 * q);
    AF_PTR(float) dst = view(I.sh[f], (long long)I.shp[f] * d.ny * d.nz, DK_SHADOW, s) +
                        ((long long)row * I.shp[f] + 4 * q);
    const int left = d.nx - 4 * (int)q;
    float4 o;
    o.x = f64_to_f32(src[0]);
    o.y = left > 1 ? f64_to_f32(src[1]) : 0.0f;
    o.z = left > 2 ? f64_to_f32(src[2]) : 0.0f;
    o.w = left > 3 ? f64_to_f32(src[3]) : 0.0f;
    AF_VEC(float4, dst, 0, 4) = o;
    END_ELEMS
    END_TILES
}

// One axis sweep of every face.  A warp owns one (component, y, z) face row
// (32 lanes per row of the face box) and its lanes stride over x; taps come
// from the binary32 shadow.  Per row the kernel fixes the component (a
// template parameter), the row pointers of the face's own field and of the
// axis component that gives the face velocity, and the four 32-bit offsets
// of that velocity's taps, so a face costs its nine loads, the arithmetic
// of mx_face_update and one store.
template <int AX, int C>
__device__ __forceinline__ void sweep_row(const InstDev& I, Status* st, AF_PTR(double) AF_RESTRICT dd, int y, int z,
                                          int x0, int x1, int phase, int slot) {
    const Geom& g = I.g;
    const Dims& d = C == 0 ? g.u : (C == 1 ? g.v : g.w);
    const Dims& a = AX == 0 ? g.u : (AX == 1 ? g.v : g.w);
    const long long py = I.shp[C], pz = py * d.ny;  // shadow strides
    AF_PTR(const float) AF_RESTRICT src =
        view((const float*)I.sh[C], py * d.ny * d.nz, DK_SWEEP_ROWS, slot) + (y * py + z * pz);
    dd += (long long)y * d.sy + (long long)z * d.sz;
    const long long s = AX == 0 ? 1 : (AX == 1 ? py : pz);
    const int na = AX == 0 ? d.nx : (AX == 1 ? d.ny : d.nz);
    // Face velocity taps (summed by mx_face_vel4): offsets from (x, y, z) in the axis
    // component's shadow, in the order they are summed.
    const int ay = I.shp[AX], az = I.shp[AX] * a.ny;
    AF_PTR(const float) AF_RESTRICT va = view((const float*)I.sh[AX], (long long)az * a.nz, DK_SWEEP_ROWS, slot) +
                                         ((long long)y * ay + (long long)z * az);
    int o0 = 0, o1 = 0, o2 = 0, o3 = 0;
    if (C == 0 && AX == 1) { o0 = -1; o1 = 0; o2 = ay - 1; o3 = ay; }
    if (C == 0 && AX == 2) { o0 = -1; o1 = 0; o2 = az - 1; o3 = az; }
    if (C == 1 && AX == 0) { o0 = -ay; o1 = 1 - ay; o2 = 0; o3 = 1; }
    if (C == 1 && AX == 2) { o0 = -ay; o1 = 0; o2 = az - ay; o3 = az; }
    if (C == 2 && AX == 0) { o0 = -az; o1 = 1 - az; o2 = 0; o3 = 1; }
    if (C == 2 && AX == 1) { o0 = -az; o1 = ay - az; o2 = 0; o3 = ay; }
    const float dt_invh = I.dt_invh, lam = I.lam;
    auto vel_at = [&](int x) {
        return C == AX ? src[x] : mx_face_vel4(va[x + o0], va[x + o1], va[x + o2], va[x + o3]);
    };
    // The next face's velocity taps load before this face's dependent taps,
    // so a lane keeps two faces' loads in flight.
    float vel_next = x0 < x1 ? vel_at(x0) : 0.0f;
    for (int x = x0; x < x1; x += 32) {
        const float vel = vel_next;
        if (x + 32 < x1) vel_next = vel_at(x + 32);
        const int ca = AX == 0 ? x : (AX == 1 ? y : z);
        float res;
        if (!mx_face_update(src + x, s, vel, ca, na, dt_invh, lam, &res)) {
            atomicMin(&st->fault_gate, st->step * 8u + (unsigned)phase);
            atomicMin(&st->fault_key, fault_key(C, x, y, z));
            continue;
        }
        dd[x] = (double)res;  // widening is exact
    }
}

// Iteration space of the sweep: 32 lanes per face row of the three
// components, then the U rows' last faces (x = G + NX), 32 rows to a warp:
// a U row has NX + 1 faces, and with NX a multiple of 32 its last face would
// otherwise cost a whole warp iteration of one lane.
__host__ __device__ inline long long sweep_box(const Geom& g) {
    return 32ll * (3ll * (g.NY + 1) * (g.NZ + 1) + ((long long)g.NY * g.NZ + 31) / 32);
}

template <int AX>
__global__ void kb_sweep(const InstDev* inst, Status* st, Tab tab, int parity, int phase) {
    begin_slot(inst, tab);
    FOR_TILES(tab)
    const InstDev& I = inst[s];
    if (gated(&st[s], phase)) continue;
    const Geom& g = I.g;
    const long long rows = 3ll * (g.NY + 1) * (g.NZ + 1), n = sweep_box(g);
    FOR_ELEMS(tab)
    if (el >= n) break;
    const long long row = el >> 5;
    const int lane = (int)(el & 31);
    if (row >= rows) {
        // Last U face of U row q.
        const long long q = (row - rows) * 32 + lane;
        if (q >= (long long)g.NY * g.NZ) continue;
        const unsigned zz = I.fny.div((unsigned)q);
        const int y = g.G + (int)((unsigned)q - zz * (unsigned)g.NY), z = g.G + (int)zz;
        sweep_row<AX, 0>(I, st + s, view(cur(I, 5, parity), g.u.count, DK_SWEEP_ROWS, s), y, z, g.G + g.NX,
                         g.G + g.NX + 1, phase, s);
        continue;
    }
    const unsigned r = (unsigned)row, r2 = I.ffy.div(r), cc = I.ffz.div(r2);
    const int c = (int)cc;
    const int y = g.G + (int)(r - r2 * (unsigned)(g.NY + 1)), z = g.G + (int)(r2 - cc * (unsigned)(g.NZ + 1));
    if (y >= g.G + g.NY + (c == 1) || z >= g.G + g.NZ + (c == 2)) continue;
    const int x0 = g.G + lane, x1 = g.G + g.NX;  // the U rows' last faces come after the rows
    if (c == 0) sweep_row<AX, 0>(I, st + s, view(cur(I, 5, parity), g.u.count, DK_SWEEP_ROWS, s), y, z, x0, x1, phase, s);
    else if (c == 1)
        sweep_row<AX, 1>(I, st + s, view(cur(I, 6, parity), g.v.count, DK_SWEEP_ROWS, s), y, z, x0, x1, phase, s);
    else sweep_row<AX, 2>(I, st + s, view(cur(I, 7, parity), g.w.count, DK_SWEEP_ROWS, s), y, z, x0, x1, phase, s);
    END_ELEMS
    END_TILES
}

// --- staged tile sweep ---------------------------------------------------
// The same sweep with its gathers served from shared memory.  A block owns a
// tile of kSwTX x kSwTY x kSwTZ faces of one component, x tiles starting at
// the first interior face (G + 32k; a U row's extra last face joins its last
// tile).  One thread stages, with TMA tensor loads over the binary32
// shadows, the tile of the face's own component with a halo along the sweep
// axis (at least 4 cells along x, kSwHA along y or z: the diffusion taps and
// every backtrace with |dt*vel/h| < kSwHA) and, when the component is not
// the sweep axis's, the tile of the axis component whose four faces give the
// face velocity (a one-cell halo).  A TMA box must start on a 16-byte
// boundary, so each box starts at the x below its tile's halo rounded down
// to a multiple of four (sw_box_x) and is wide enough for any rounding.
// Backtraces that leave the staged halo read the shadow in global memory
// instead.  Every face's arithmetic is the row kernel's (mx_face_vel4,
// mx_backtrace, mx_face_value): the same bits.
// Six planes deep: a thread computes six faces per tile, so the tile's
// set-up (transfer wait, barrier, indices) is spread over more faces than
// with four planes, while four blocks still fit an SM (measured per sweep
// launch at 256^3, with the tile decoded by every thread: 4 planes 268-281 us,
// 6 planes 236-250 us, 8 planes at three blocks per SM 290-311 us).
//
// Bound by issue (two thirds of the slots; 3.8 TB/s from memory), so the work
// is in what a face costs: a backtrace of less than a cell interpolates
// between values the diffusion has loaded anyway, values shared along z stay
// in registers, the result is widened on the integer pipe, and a warp of its
// own decodes tiles.  113 -> 68 instructions a face, 256^3 235-243 ->
// 156-162 us a sweep (207-218 without the loading warp; 158-168 with the z
// loop not unrolled).
constexpr int kSwTX = 32, kSwTY = 8, kSwTZ = 6, kSwHA = 2, kSwThreads = kSwTX * kSwTY;
constexpr int kSwBlock = kSwThreads + 32;  // and the loading warp
// Box roles: 0-2 the own component for a sweep along x, y, z; 3 the axis
// component.  First x of a box (a multiple of 4) and its width.
__host__ __device__ constexpr int sw_box_x(int role, int x0) {
    return (role == 0 ? x0 - 4 : (role == 3 ? x0 - 1 : x0)) & ~3;
}
__host__ __device__ constexpr int sw_bx(int role) {
    return role == 0 ? kSwTX + 12 : (role == 3 ? kSwTX + 8 : kSwTX + 4);
}
__host__ __device__ constexpr int sw_by(int role) {
    return role == 1 ? kSwTY + 2 * kSwHA : (role == 3 ? kSwTY + 2 : kSwTY);
}
__host__ __device__ constexpr int sw_bz(int role) {
    return role == 2 ? kSwTZ + 2 * kSwHA : (role == 3 ? kSwTZ + 2 : kSwTZ);
}
__host__ __device__ constexpr int sw_box_floats(int role) { return sw_bx(role) * sw_by(role) * sw_bz(role); }
__host__ __device__ constexpr int sw_max(int a, int b) { return a > b ? a : b; }
// Floats of the largest own-component box, rounded up to 32 (128 bytes: the
// buffers are TMA destinations).
constexpr int kSwOwnMax = (sw_max(sw_box_floats(0), sw_max(sw_box_floats(1), sw_box_floats(2))) + 31) / 32 * 32;
constexpr int kSwAxCount = (kSwTX + 8) * (kSwTY + 2) * (kSwTZ + 2);
static_assert(kSwAxCount % 32 == 0, "axis-box buffers start on 128-byte boundaries");
// Two buffer pairs (own, axis) per block, in dynamic shared memory.
constexpr size_t kSwSmem = (size_t)2 * (kSwOwnMax + kSwAxCount) * sizeof(float);
static_assert(sw_bx(0) * sw_by(0) * sw_bz(0) <= kSwOwnMax && sw_bx(1) * sw_by(1) * sw_bz(1) <= kSwOwnMax &&
              sw_bx(2) * sw_by(2) * sw_bz(2) <= kSwOwnMax, "own box exceeds its buffer");
static_assert(sw_bx(3) * sw_by(3) * sw_bz(3) == kSwAxCount, "axis box size");
// A wait on a TMA transfer gives up after this many polls (each poll itself
// blocks for a bounded, hardware-defined time); the kernel then records the
// failure in the batch's diagnostic word and returns.
constexpr unsigned kSwSpinLimit = 1u << 22;

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// A wait also gives up after this long (a transfer lands in microseconds).
constexpr unsigned long long kWaitLimitNs = 200000000ull;
// Suspend-time hint of one poll: a waiting thread sleeps in the barrier
// until the phase completes (or this long) instead of re-issuing the poll,
// so waiting warps take no issue slots from the working ones.
constexpr unsigned kPollSuspendNs = 20000u;
__device__ __forceinline__ bool mbar_try_wait_sleep(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity), "n"(kPollSuspendNs)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Polls the barrier's phase `parity` at most kSwSpinLimit times and for at
// most kWaitLimitNs.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (unsigned it = 1; it < kSwSpinLimit; ++it) {
        if (mbar_try_wait_sleep(bar, parity)) return true;
        if ((it & 15u) == 0u && global_ns() - t0 > kWaitLimitNs) return false;
    }
    return false;
}
// Whether an earlier kernel of the work gave up a wait (its results are
// invalid, so later staged kernels return at once instead of waiting again).
__device__ __forceinline__ bool diag_set(const unsigned* diag) { return *(const volatile unsigned*)diag != 0u; }
__device__ __forceinline__ void tma_load_3d(float* dst, const CUtensorMap* map, int x, int y, int z,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
        : "memory");
}

// A tile of the staged sweep as the loading thread hands it to its block: the slot, the
// component and the first face, and what a face needs of the slot, so that
// the block's other threads neither decode the tile nor read the slot's
// record.
struct SwTile {
    int live;  // 0 past the work list, without faces, or when the slot is gated by a fault
    int s, c, x0, y0, z0;
    int xhi, yhi, zend;   // one past the tile's last face (the component's last row: yhi)
    int na, cmax;         // padded extent along the sweep axis; last coordinate a short backtrace is unclamped at
    int dsy, dsz;         // strides of the component's binary64 field
    int py, pz, dnz;      // row pitch and plane of its shadow, its planes
    float dt_invh, lam;
    double* dd;           // the binary64 field written
    long long count;
    const float* sh;      // the shadow
    Status* st;
};

// Faces of one tile of component C (the loads have landed in own / axv).
template <int AX, int C>
__device__ __forceinline__ void sweep_tile_faces(const SwTile& T, const float* own_, const float* axv_, int phase) {
    const int slot = T.s;
    AF_PTR(const float) own = view(own_, (long long)kSwOwnMax, DK_SWEEP_TMA, slot);
    AF_PTR(const float) axv = view(axv_, (long long)kSwAxCount, DK_SWEEP_TMA, slot);
    AF_PTR(double) AF_RESTRICT dd = view(T.dd, T.count, DK_SWEEP_TMA, slot);
    constexpr int BX = sw_bx(AX), BY = sw_by(AX), BZ = sw_bz(AX);
    constexpr int SO = AX == 0 ? 1 : (AX == 1 ? BX : BX * BY);  // own-box stride along the sweep axis
    constexpr int AXX = sw_bx(3), AXY = sw_by(3);
    // Axis-box strides along the component's axis and the sweep axis.
    constexpr int EC = C == 0 ? 1 : (C == 1 ? AXX : AXX * AXY);
    constexpr int EA = AX == 0 ? 1 : (AX == 1 ? AXX : AXX * AXY);
    const int x0 = T.x0, y0 = T.y0, z0 = T.z0;
    const int ox = sw_box_x(AX, x0), oy = y0 - (AX == 1 ? kSwHA : 0), oz = z0 - (AX == 2 ? kSwHA : 0);
    const int oa = AX == 0 ? ox : (AX == 1 ? oy : oz);  // own box's first coordinate along the axis
    const int ax0 = sw_box_x(3, x0);
    const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
    const int y = y0 + ly;
    if (y >= T.yhi) return;
    const int xhi = T.xhi, zend = T.zend, cmax = T.cmax, dsz = T.dsz;
    const float dt_invh = T.dt_invh, lam = T.lam;
    // A backtrace of less than a cell whose taps lie inside the field, which
    // mx_backtrace leaves unclamped: off > -1 and ca >= 1 give a position
    // above 0, off < 1 and ca <= na - 3 one below na - 1 (SwTile::cmax).
    for (int x = x0 + lx; x < xhi; x += kSwTX) {
        // Walk z with every index advanced by its plane stride: the face's
        // own box, the axis box and the binary64 destination.  What the next
        // plane's face reads again stays in registers: along z the face's own
        // values, and two of the four velocity taps where the component's or
        // the sweep's axis is z.
        int io = ((z0 - oz) * BY + (y - oy)) * BX + (x - ox);
        int ia = (AXY + (y - y0 + 1)) * AXX + (x - ax0);
        AF_PTR(double) dz = dd + (x + y * T.dsy + z0 * dsz);  // a field holds < 2^31 elements
        const bool in_xy = AX == 2 || (AX == 0 ? x : y) <= cmax;
        float m = 0.0f, c = 0.0f, v0 = 0.0f, v1 = 0.0f;
        if (AX == 2) m = own[io - SO], c = own[io];
        if (C != AX && AX == 2) v0 = axv[ia - EC], v1 = axv[ia];
        if (C != AX && C == 2) v0 = axv[ia - EC], v1 = axv[ia + EA - EC];
#pragma unroll 2
        for (int z = z0; z < zend; ++z, io += BX * BY, ia += AXX * AXY, dz += dsz) {
            if (AX != 2) m = own[io - SO], c = own[io];
            const float p = own[io + SO];
            float vel;
            // The row kernel's tap order: before the sweep axis's own
            // component, (-e_C, 0, e_AX - e_C, e_AX); after it,
            // (-e_C, e_AX - e_C, 0, e_AX).
            if (C == AX) {
                vel = c;
            } else if (AX == 2 || C == 2) {
                const float w0 = AX == 2 ? axv[ia + EA - EC] : axv[ia], w1 = axv[ia + EA];
                vel = mx_face_vel4(v0, v1, w0, w1);
                v0 = w0, v1 = w1;
            } else if (AX > C) {
                vel = mx_face_vel4(axv[ia - EC], axv[ia], axv[ia + EA - EC], axv[ia + EA]);
            } else {
                vel = mx_face_vel4(axv[ia - EC], axv[ia + EA - EC], axv[ia], axv[ia + EA]);
            }
            const int ca = AX == 0 ? x : (AX == 1 ? y : z);
            const float off = -__fmul_rn(vel, dt_invh);
            float t, d0, d1;
            if (fabsf(off) < 1.0f && (AX == 2 ? z <= cmax : in_xy)) {
                const bool back = off < 0.0f;
                t = __fadd_rn(off, back ? 1.0f : 0.0f);  // off - floor(off), and +0 of -0
                d0 = back ? m : c;
                d1 = back ? c : p;
            } else {
                int i0;
                if (!mx_backtrace(vel, ca, T.na, dt_invh, &i0, &t)) {
                    atomicMin(&T.st->fault_gate, T.st->step * 8u + (unsigned)phase);
                    atomicMin(&T.st->fault_key, fault_key(C, x, y, z));
                    if (AX == 2) m = c, c = p;
                    continue;
                }
                const int rel = i0 - ca;
                if (i0 >= oa && i0 + 1 < oa + (AX == 0 ? BX : (AX == 1 ? BY : BZ))) {
                    d0 = own[io + rel * SO];
                    d1 = own[io + (rel + 1) * SO];
                } else {
                    AF_PTR(const float) gp =
                        view(T.sh, (long long)T.pz * T.dnz, DK_SWEEP_TMA, slot) + (x + y * T.py + (long long)z * T.pz);
                    const int gs = AX == 0 ? 1 : (AX == 1 ? T.py : T.pz);
                    d0 = gp[(long long)rel * gs];
                    d1 = gp[(long long)(rel + 1) * gs];
                }
            }
            dz[0] = widen(mx_face_value(t, d0, d1, m, c, p, lam));
            if (AX == 2) m = c, c = p;
        }
    }
}

// Called by a whole warp (find_slot); its first lane writes the tile.
template <int AX>
__device__ __forceinline__ void sw_decode(const InstDev* inst, Status* st, const Tab& tab, int item, int total,
                                          int parity, int phase, SwTile* t) {
    const int s = item < total ? find_slot(tab.prefix, tab.n, item) : -1;
    if ((threadIdx.x & 31) != 0) return;
    t->live = 0;
    if (s < 0) return;
    const InstDev& I = inst[s];
    if (gated(&st[s], phase)) return;
    // The three components of one spatial tile are consecutive items, so
    // the axis component's box, staged again for the other two, is still in
    // L2.  A spatial tile past one component's last face row or plane holds
    // no faces of it.
    const Geom& g = I.g;
    const unsigned local = (unsigned)(item - tab.prefix[s]);
    const unsigned r = local / 3u;
    const int c = (int)(local - 3u * r);
    const unsigned q1 = I.swx.div(r), q2 = I.swy.div(q1);
    t->s = s;
    t->c = c;
    t->x0 = g.G + (int)(r - q1 * I.swx.d) * kSwTX;
    t->y0 = g.G + (int)(q1 - q2 * I.swy.d) * kSwTY;
    t->z0 = g.G + (int)q2 * kSwTZ;
    t->yhi = g.G + g.NY + (c == 1);
    t->zend = min(t->z0 + kSwTZ, g.G + g.NZ + (c == 2));
    if (t->y0 >= t->yhi || t->z0 >= t->zend) return;
    // The last tile of a row runs to the component's last face.
    t->xhi = t->x0 + kSwTX >= g.G + g.NX ? g.G + g.NX + (c == 0) : t->x0 + kSwTX;
    const Dims& d = c == 0 ? g.u : (c == 1 ? g.v : g.w);
    t->na = AX == 0 ? d.nx : (AX == 1 ? d.ny : d.nz);
    t->cmax = g.G >= 1 ? t->na - 3 : -1;
    t->dsy = (int)d.sy;
    t->dsz = (int)d.sz;
    t->py = I.shp[c];
    t->pz = I.shp[c] * d.ny;
    t->dnz = d.nz;
    t->dt_invh = I.dt_invh;
    t->lam = I.lam;
    t->dd = cur(I, 5 + c, parity);
    t->count = d.count;
    t->sh = I.sh[c];
    t->st = st + s;
    t->live = 1;
}

// The loading thread: the TMA loads of tile t into one buffer pair.  The buffers' last
// reads (generic proxy) finished before the caller's barrier; the fence
// orders them before these writes (async proxy).
template <int AX>
__device__ __forceinline__ void sw_issue(const InstDev& I, const SwTile& t, float* own, float* axv,
                                         unsigned long long* bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    constexpr unsigned own_bytes = sw_bx(AX) * sw_by(AX) * sw_bz(AX) * 4u;
    mbar_expect_tx(bar, own_bytes + (t.c != AX ? kSwAxCount * 4u : 0u));
    tma_load_3d(own, I.tmap + t.c * 4 + AX, sw_box_x(AX, t.x0), t.y0 - (AX == 1 ? kSwHA : 0),
                t.z0 - (AX == 2 ? kSwHA : 0), bar);
    if (t.c != AX) tma_load_3d(axv, I.tmap + AX * 4 + 3, sw_box_x(3, t.x0), t.y0 - 1, t.z0 - 1, bar);
}

// Persistent blocks walk their tiles with two buffer pairs: a warp of its own
// decodes the next tile and issues its loads while the others compute the
// current one's faces.
template <int AX>
__global__ void __launch_bounds__(kSwBlock, 4)
    kb_sweep_tma(const InstDev* inst, Status* st, Tab tab, int parity, int phase, unsigned* diag) {
    begin_slot(inst, tab);
    extern __shared__ __align__(128) float swsm[];
    // Buffer pair k: own-component box and axis box.
    auto own = [&](int k) { return swsm + k * kSwOwnMax; };
    auto axv = [&](int k) { return swsm + 2 * kSwOwnMax + k * kSwAxCount; };
    __shared__ __align__(8) unsigned long long bar[2];
    __shared__ unsigned stop;
    if (smem_addr(swsm) & 127u) {  // the buffers are TMA destinations: 128-byte aligned base
        if (threadIdx.x == 0) atomicOr(diag, 4u);
        return;
    }
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        stop = diag_set(diag) ? 1u : 0u;
    }
    __syncthreads();
    if (stop) return;
    const int total = tab.prefix[tab.n];
    unsigned ph = 0u;  // bit k: the phase parity buffer k waits for next
    int item = blockIdx.x, k = 0;
    __shared__ __align__(8) SwTile tile[2];  // of buffer pair k
    // The loading warp, all its lanes; the first one does the work.
    const bool loading = threadIdx.x >= kSwThreads, loader = threadIdx.x == kSwThreads;
    auto begin_tile = [&](int it, int kk) {
        sw_decode<AX>(inst, st, tab, it, total, parity, phase, &tile[kk]);
        if (loader && tile[kk].live) sw_issue<AX>(inst[tile[kk].s], tile[kk], own(kk), axv(kk), &bar[kk]);
    };
    if (loading) begin_tile(item, 0);
    __syncthreads();
    while (item < total) {
        const int next_item = item + gridDim.x;
        const SwTile& T = tile[k];
        bool ok = true;
        if (loading) {
            begin_tile(next_item, k ^ 1);
        } else if (T.live) {
            ok = mbar_wait_bounded(&bar[k], (ph >> k) & 1u);
            if (!ok) {
            } else if (T.c == 0) {
                sweep_tile_faces<AX, 0>(T, own(k), axv(k), phase);
            } else if (T.c == 1) {
                sweep_tile_faces<AX, 1>(T, own(k), axv(k), phase);
            } else {
                sweep_tile_faces<AX, 2>(T, own(k), axv(k), phase);
            }
        }
        if (T.live) ph ^= 1u << k;
        // Every thread is done with buffer pair k before it is loaded again.
        if (__syncthreads_or(ok ? 0 : 1)) {
            // A transfer did not land in time: record it, give the copies in
            // flight a second bounded wait, and stop.
            if (loader) {
                atomicOr(diag, 1u);
                mbar_wait_bounded(&bar[k], ((ph >> k) & 1u) ^ 1u);
                if (tile[k ^ 1].live) mbar_wait_bounded(&bar[k ^ 1], (ph >> (k ^ 1)) & 1u);
            }
            __syncthreads();
            return;
        }
        item = next_item;
        k ^= 1;
    }
}

__global__ void kb_tick(const InstDev* inst, Status* st, int n) {
    pdl_wait();
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x)
        if (inst[s].active) st[s].step += 1;
}

// --- refinement control ---------------------------------------------------
__global__ void kb_init(const InstDev* inst, Ctl* ctl, int n) {
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl[n].nv = 0xFFFFFFFFu;  // until a check counts them
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        ctl[s].maxr_bits = 0;
        ctl[s].passes = 0;
        ctl[s].stopped = inst[s].active ? 0u : 1u;
        ctl[s].nv = 0u;
        ctl[s].vtotal = 0u;
        ctl[s].last_div = 0;
    }
}

// r = b - L(p) in binary64 over the interior, r (binary32) for the inner
// solve, inner solution zeroed, max|r| reduced per slot.  In the loop a
// converged slot is skipped.
__device__ __forceinline__ void warp_max_commit(unsigned long long m, unsigned long long* out) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, o);
        m = t > m ? t : m;
    }
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

// r = b - L(p) in binary64 over the interior, r (binary32) for the inner
// solve, inner solution zeroed, max|r| reduced per slot.  A block keeps its
// running maximum over consecutive tiles of one slot and commits it (one
// atomic per warp) when the slot changes or the block finishes, so the
// atomics are per block, not per warp-sized tile.  In the loop a converged
// slot is skipped.  Bound by the binary64 pipe: of the seven operations the x
// and y neighbour sums run on the integer pipe (the last difference cancels
// too deeply for it; a third sum there costs more issue than it saves).  A
// thread takes 2^res_lg cells of a column, so that their indices are worked
// out once and a cell's z neighbours stay in registers (residual_planes_log).
// 256^3: 268 us with no integer sums, 222 a cell a thread, 186 with eight.
__global__ void kb_residual(const InstDev* inst, Status* st, Ctl* ctl, Tab tab, int gate, int in_loop) {
    begin_slot(inst, tab);
    int held = -1;
    unsigned long long m = 0;
    for (int item = blockIdx.x, total = tab.prefix[tab.n]; item < total; item += gridDim.x) {
        const int s = find_slot(tab.prefix, tab.n, item);
        const long long first = (long long)(item - tab.prefix[s]) * blockDim.x * tab.ept;
        const InstDev& I = inst[s];
        if (gated(&st[s], gate) || (in_loop && ctl[s].stopped)) continue;
        if (s != held) {
            if (held >= 0) warp_max_commit(m, &ctl[held].maxr_bits);
            held = s;
            m = 0;
        }
        const Geom& g = I.g;
        const long long nl0 = lvl_cells(I.lev[0]);
        AF_PTR(const double) AF_RESTRICT p = view((const double*)I.slot[0], g.p.count, DK_RESIDUAL, s);
        AF_PTR(const double) AF_RESTRICT bb = view((const double*)I.b, g.p.count, DK_RESIDUAL, s);
        AF_PTR(float) AF_RESTRICT r0 = view(I.lev[0].r, nl0, DK_RESIDUAL, s);
        AF_PTR(float) AF_RESTRICT e0 = view(I.lev[0].e, nl0, DK_RESIDUAL, s);
        const int planes = 1 << I.res_lg;
        const long long n = residual_items(g, I.res_lg);
        for (int k = 0; k < tab.ept; ++k) {
            const long long el = first + (long long)k * blockDim.x + threadIdx.x;
            if (el >= n) continue;
            const unsigned e = (unsigned)el, r2 = I.fnx.div(e), zz = I.fny.div(r2);
            const int xi = (int)(e - r2 * (unsigned)g.NX), yi = (int)(r2 - zz * (unsigned)g.NY), z0 = (int)zz << I.res_lg;
            const int sy = (int)g.p.sy, sz = (int)g.p.sz;  // a field holds < 2^31 elements
            int i = (g.G + xi) + (g.G + yi) * sy + (g.G + z0) * sz;
            int j = xi + g.NX * (yi + g.NY * z0);
            // A neighbour across a wall is the cell itself.
            const int xm = xi > 0 ? -1 : 0, xp = xi < g.NX - 1 ? 1 : 0;
            const int ym = yi > 0 ? -sy : 0, yp = yi < g.NY - 1 ? sy : 0;
            double below = p[z0 > 0 ? i - sz : i], pc = p[i];
            // A constant count with an early exit: 186 us where a computed one
            // takes 200.
#pragma unroll 1
            for (int c = 0; c < 1 << kResMaxLg; ++c, i += sz, j += g.NX * g.NY) {
                const int z = z0 + c;
                if (z >= g.NZ || c >= planes) break;
                const double above = p[z < g.NZ - 1 ? i + sz : i];
                const double sum = dadd(dadd(dadd_int(p[i + xm], p[i + xp]), dadd_int(p[i + ym], p[i + yp])),
                                        dadd(below, above));
                const double res = dsub(bb[i], __fma_rn(-6.0, pc, sum));
                r0[j] = f64_to_f32(res);
                e0[j] = 0.0f;
                below = pc;
                pc = above;
                // |res| and NaN on the bit pattern (integer pipe); NaN reads as
                // +Inf so the loop stops.
                const unsigned long long a = dbits(res) & ~kSign;
                const unsigned long long v = a > 0x7FF0000000000000ull ? 0x7FF0000000000000ull : a;
                m = v > m ? v : m;
            }
        }
    }
    if (held >= 0) warp_max_commit(m, &ctl[held].maxr_bits);
}

// p += e over the interior.  Bound by memory (20 bytes a cell).  A thread takes
// kCorrZ cells of a column, loads before stores, and neighbouring threads
// neighbouring cells across the ends of rows: a warp per row left lanes idle
// on rows that are no multiple of 32 and had one load in flight.  48x32x64 5.8 ->
// 4.8 us, 256^3 60 -> 58, a 256-grid batch 512 -> 453; a warp per row with four
// cells a lane: 54.7 at 256^3, 712 for the batch.
__global__ void kb_correct(const InstDev* inst, Ctl* ctl, Tab tab) {
    begin_slot(inst, tab);
    FOR_TILES(tab)
    const InstDev& I = inst[s];
    if (ctl[s].stopped) continue;
    const Geom& g = I.g;
    AF_PTR(double) AF_RESTRICT p = view(I.slot[0], g.p.count, DK_CORRECT, s);
    AF_PTR(const float) AF_RESTRICT e0 = view((const float*)I.lev[0].e, lvl_cells(I.lev[0]), DK_CORRECT, s);
    const long long n = correct_items(g);
    FOR_ELEMS(tab)
    if (el >= n) break;
    const unsigned q = (unsigned)el, r2 = I.fnx.div(q), zz = I.fny.div(r2);
    const int x = (int)(q - r2 * (unsigned)g.NX), y = (int)(r2 - zz * (unsigned)g.NY), z = (int)zz * kCorrZ;
    const int sy = (int)g.p.sy, sz = (int)g.p.sz, se = g.NX * g.NY;
    const int i = (g.G + x) + (g.G + y) * sy + (g.G + z) * sz, j = x + g.NX * y + se * z;
    double v[kCorrZ];
    float d[kCorrZ];
#pragma unroll
    for (int k = 0; k < kCorrZ; ++k)
        if (z + k < g.NZ) v[k] = p[i + k * sz], d[k] = e0[j + k * se];
#pragma unroll
    for (int k = 0; k < kCorrZ; ++k)
        if (z + k < g.NZ) p[i + k * sz] = v[k] + f32_to_f64(d[k]);
    END_ELEMS
    END_TILES
}

// One block: per slot, whether another refinement pass runs; the WHILE
// condition is "any slot continues".  Bounded by each slot's max_refine.
__global__ void kb_check(const InstDev* inst, Status* st, Ctl* ctl, int n, cudaGraphConditionalHandle h, int use_cond,
                         int count_pass, int gate, int vcycles, double pass_floor) {
    pdl_wait();
    __shared__ unsigned most;  // V-cycles of the next pass, most over the slots
    if (threadIdx.x == 0) most = 0u;
    __syncthreads();
    int any = 0;
    for (int s = threadIdx.x; s < n; s += blockDim.x) {
        const InstDev& I = inst[s];
        if (!I.active) continue;
        Ctl& c = ctl[s];
        const double r = __longlong_as_double((long long)c.maxr_bits);
        c.maxr_bits = 0;
        if (c.stopped) continue;
        const double div = I.res_scale * r;
        // A pass that removes less than a tenth of max|r| has reached the
        // binary64 round-off floor of the residual (|B| * 2^-53 and up):
        // stop there rather than spin to the pass cap.
        const bool stalled = count_pass && div > 0.9 * c.last_div;
        const double prev = c.last_div;
        c.last_div = div;
        if (count_pass) c.passes += 1;
        const bool more =
            !gated(&st[s], gate) && div > I.thresh && !isinf(div) && !stalled && c.passes < I.max_refine;
        // The last pass often needs fewer V-cycles than the others: from the
        // reduction per V-cycle the pass just achieved, predict how many more
        // bring max|div| below half the threshold, and run only those.
        // The first pass of a projection uses the factor the slot's last
        // projection measured.
        if (count_pass) c.vtotal += c.nv ? c.nv : (unsigned)vcycles;
        if (count_pass && prev > 0.0) {
            const double ran = c.nv ? (double)c.nv : (double)vcycles;
            const double f = pow(div / prev, 1.0 / ran);
            if (f < 1.0) c.vfac = f;
        }
        // A pass cannot take max|r| below its binary32 floor (the inner
        // solve's correction carries about 24 bits), so V-cycles past
        // log(pass_floor) / log(vfac) are cut as well (pass_floor = 0: no
        // such cut).
        unsigned nv = 0u;
        if (more && c.vfac > 0.0 && c.vfac < 1.0) {
            double k = ceil(log(0.5 * I.thresh / div) / log(c.vfac));
            if (pass_floor > 0.0) k = fmin(k, ceil(log(pass_floor) / log(c.vfac)));
            if (k < 1.0) k = 1.0;
            if (k < (double)vcycles) nv = (unsigned)k;
        }
        c.nv = nv;
        if (!more) c.stopped = 1;
        else atomicMax(&most, nv ? nv : (unsigned)vcycles);
        any |= more ? 1 : 0;
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) ctl[n].nv = most;
    if (threadIdx.x == 0 && use_cond) cudaGraphSetConditional(h, any ? 1u : 0u);
}

// --- binary32 multigrid ---------------------------------------------------
__device__ __forceinline__ long long lidx(int x, int y, int z, int nx, int ny) {
    return x + (long long)nx * (y + (long long)ny * z);
}

// Binary32 cell formulas of the multigrid with every rounding written out
// (no contraction left to the compiler), so the per-level kernels, the fused
// red-black pair and the one-block tail V-cycle compute the same bits.
// Over-relaxed update of one cell from its value c:
//   c + omega * ((wx*sx + wy*sy + wz*sz - r) / (2*(wx+wy+wz)) - c).
// omega = 1.5 was measured best on cubes of 128^3-512^3 (refinement passes
// to max|div| <= 1e-10 per projection at 256^3: 8 at omega = 1, 6 at 1.3,
// 5 at 1.5, 7 at 1.6).
constexpr float kMgOmega = 1.5f;
struct MgW {  // a level's weights
    float wx, wy, wz;
};
template <class LevelOrWeights>
__device__ __forceinline__ float mg_relax(const LevelOrWeights& L, float sx, float sy, float sz, float r, float inv, float c) {
    const float v = __fmul_rn(__fsub_rn(__fmaf_rn(L.wz, sz, __fmaf_rn(L.wy, sy, __fmul_rn(L.wx, sx))), r), inv);
    return __fmaf_rn(kMgOmega, __fsub_rn(v, c), c);
}
// Residual of one cell: r - (wx*dxx + wy*dyy + wz*dzz), d** the second differences.
template <class LevelOrWeights>
__device__ __forceinline__ float mg_res(const LevelOrWeights& L, float sx, float sy, float sz, float c, float r) {
    const float c2 = 2.0f * c;
    return __fsub_rn(r, __fmaf_rn(L.wz, __fsub_rn(sz, c2), __fmaf_rn(L.wy, __fsub_rn(sy, c2), __fmul_rn(L.wx, __fsub_rn(sx, c2)))));
}
// Trilinear weights (a* on the parent, b* = 1 - a* on its neighbour).
__device__ __forceinline__ float mg_interp(float ax, float ay, float az, float e000, float e100, float e010, float e110,
                                           float e001, float e101, float e011, float e111) {
    const float bx = 1.0f - ax, by = 1.0f - ay, bz = 1.0f - az;
    auto lx = [&](float p, float q) { return __fmaf_rn(bx, q, __fmul_rn(ax, p)); };
    auto ly = [&](float p, float q) { return __fmaf_rn(by, q, __fmul_rn(ay, p)); };
    const float z0 = ly(lx(e000, e100), lx(e010, e110)), z1 = ly(lx(e001, e101), lx(e011, e111));
    return __fmaf_rn(bz, z1, __fmul_rn(az, z0));
}

// One red-black colour sweep of L e = r in place.  A warp owns one (y, z) row
// and its lanes stride over the row's cells of the colour; the neighbour
// rows are addressed through pointers clamped to the row itself at the
// walls (the Neumann reflection, the same values as per-cell selects), so a
// cell costs its eight loads, the relaxation and a store.  The iteration
// space counts 32 lanes per row (row_box).
__host__ __device__ inline long long row_box(const Lvl& L) { return 32ll * L.ny * L.nz; }

__global__ void kb_smooth(const InstDev* inst, const Ctl* ctl, Tab tab, int l, int color, int vc) {
    begin_level(inst, tab, l, 1);
    if (vc_idle(ctl, tab.n, vc)) return;
    FOR_TILES(tab)
    if (mg_off(ctl[s], vc)) continue;
    const Lvl L = inst[s].lev[l];
    const long long rows = (long long)L.ny * L.nz;
    const long long nxy = (long long)L.nx * L.ny;
    const float inv = 1.0f / (2.0f * (L.wx + L.wy + L.wz));
    FOR_ELEMS(tab)
    const long long row = el >> 5;
    if (row >= rows) break;
    const int lane = (int)(el & 31);
    const unsigned zz = L.fny.div((unsigned)row);
    const int y = (int)((unsigned)row - zz * (unsigned)L.ny), z = (int)zz;
    AF_PTR(float) AF_RESTRICT e = view(L.e, lvl_cells(L), DK_SMOOTH, s) + ((long long)L.nx * y + nxy * z);
    AF_PTR(const float) AF_RESTRICT rr =
        view((const float*)L.r, lvl_cells(L), DK_SMOOTH, s) + ((long long)L.nx * y + nxy * z);
    AF_PTR(const float) ym = y > 0 ? e - L.nx : e;
    AF_PTR(const float) yp = y < L.ny - 1 ? e + L.nx : e;
    AF_PTR(const float) zm = z > 0 ? e - nxy : e;
    AF_PTR(const float) zp = z < L.nz - 1 ? e + nxy : e;
    const int p = ((y + z) & 1) != color ? 1 : 0;
    for (int x = p + 2 * lane; x < L.nx; x += 64) {
        const int xm = x > 0 ? x - 1 : x, xp = x < L.nx - 1 ? x + 1 : x;
        const float c = e[x];
        const float sx = e[xm] + e[xp];
        const float sy = ym[x] + yp[x];
        const float sz = zm[x] + zp[x];
        e[x] = mg_relax(L, sx, sy, sz, rr[x], inv, c);
    }
    END_ELEMS
    END_TILES
}

__device__ __forceinline__ float mg_residual(const Lvl& L, int x, int y, int z, int slot) {
    const long long nxy = (long long)L.nx * L.ny;
    const long long i = lidx(x, y, z, L.nx, L.ny);
    AF_PTR(const float) le = view((const float*)L.e, lvl_cells(L), DK_RESTRICT, slot);
    AF_PTR(const float) lr = view((const float*)L.r, lvl_cells(L), DK_RESTRICT, slot);
    const float c = le[i];
    const float sx = (x > 0 ? le[i - 1] : c) + (x < L.nx - 1 ? le[i + 1] : c);
    const float sy = (y > 0 ? le[i - L.nx] : c) + (y < L.ny - 1 ? le[i + L.nx] : c);
    const float sz = (z > 0 ? le[i - nxy] : c) + (z < L.nz - 1 ? le[i + nxy] : c);
    return mg_res(L, sx, sy, sz, c, lr[i]);
}

// Four cells of a level's row from an even one on.  V4: rows and arrays start
// on 16-byte boundaries (Lvl::v4), one access; otherwise two of 8 bytes, the
// second of them (cells 2 and 3) only where `two` (nx is even, so each pair is
// whole).
template <bool V4, class P>
__device__ __forceinline__ float4 ld_quad(P p, long long i, bool two) {
    if (V4) return AF_VEC(const float4, p, i, 4);
    const float2 a = AF_VEC(const float2, p, i, 2), b = AF_VEC(const float2, p, i + (two ? 2 : 0), 2);
    return make_float4(a.x, a.y, b.x, b.y);
}

// Means of the residuals of two coarse cells' children, from the 2 x 2 rows of
// four fine cells at b (e) and rb (r); a neighbour across a wall is the cell
// itself.  The children in the order z, y, x with x fastest.
template <bool V4, class P>
__device__ __forceinline__ float2 restrict_two(const Lvl& F, P b, P rb, int x0, int y0, int z0, bool two, float inv) {
    const long long sy = F.nx, sz = (long long)F.nx * F.ny;
    const int xm = x0 > 0 ? -1 : 0, xp = x0 + 4 < F.nx ? 4 : (two ? 3 : 1);
    const long long ym = y0 > 0 ? -sy : 0, yp = y0 + 2 < F.ny ? 2 * sy : sy;
    const long long zm = z0 > 0 ? -sz : 0, zp = z0 + 2 < F.nz ? 2 * sz : sz;
    float4 E[2][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) E[k >> 1][k & 1] = ld_quad<V4>(b, (k & 1) * sy + (k >> 1) * sz, two);
    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int dy = k & 1, dz = k >> 1;
        const long long o = dy * sy + dz * sz;
        const float4 c = E[dz][dy], R = ld_quad<V4>(rb, o, two);
        const float4 my = E[dz][dy ^ 1], ny = ld_quad<V4>(b, dz * sz + (dy ? yp : ym), two);
        const float4 mz = E[dz ^ 1][dy], nz = ld_quad<V4>(b, dy * sy + (dz ? zp : zm), two);
        const float l = b[o + xm], r = b[o + xp];
        s0 += mg_res(F, l + c.y, ny.x + my.x, nz.x + mz.x, c.x, R.x);
        s0 += mg_res(F, c.x + (two ? c.z : r), ny.y + my.y, nz.y + mz.y, c.y, R.y);
        s1 += mg_res(F, c.y + c.w, ny.z + my.z, nz.z + mz.z, c.z, R.z);
        s1 += mg_res(F, c.z + r, ny.w + my.w, nz.w + mz.w, c.w, R.w);
    }
    return make_float2(s0 * inv, s1 * inv);
}

// Coarse rhs = mean of the children's residuals; coarse solution = 0.  Where
// every axis coarsens a thread takes two coarse cells along x, whose children
// are rows of four cells: 16 wide loads and 8 narrow ones where a cell a
// thread made 80 narrow ones.  Bound by memory: e and r are read once from it
// (8 bytes a fine cell).  Measured at 256^3 / 512^3, a cell a thread / two:
// 38.8 / 34.7 and 239 / 214 us.  Otherwise a thread a coarse cell.
__host__ __device__ inline bool restrict_pairs(const Lvl& F) { return F.cx && F.cy && F.cz; }
__host__ __device__ inline long long restrict_items(const Lvl& F, const Lvl& C) {
    return restrict_pairs(F) ? (long long)((C.nx + 1) / 2) * C.ny * C.nz : lvl_cells(C);
}

__global__ void __launch_bounds__(1024, 1) kb_restrict(const InstDev* inst, const Ctl* ctl, Tab tab, int l, int vc) {
    begin_level(inst, tab, l, 2);
    if (vc_idle(ctl, tab.n, vc)) return;
    FOR_TILES(tab)
    if (mg_off(ctl[s], vc)) continue;
    const Lvl& F = inst[s].lev[l];
    const Lvl& C = inst[s].lev[l + 1];
    const long long n = restrict_items(F, C);
    const int ex = F.cx ? 2 : 1, ey = F.cy ? 2 : 1, ez = F.cz ? 2 : 1;
    const float inv = 1.0f / (float)(ex * ey * ez);
    AF_PTR(float) cr = view(C.r, lvl_cells(C), DK_RESTRICT, s);
    AF_PTR(float) ce = view(C.e, lvl_cells(C), DK_RESTRICT, s);
    FOR_ELEMS(tab)
    if (el >= n) break;
    const unsigned e = (unsigned)el;
    if (restrict_pairs(F)) {
        const unsigned row = C.fhx.div(e), zz = C.fny.div(row);
        const int X = 2 * (int)(e - row * C.fhx.d), Y = (int)(row - zz * (unsigned)C.ny), Z = (int)zz;
        const bool two = X + 1 < C.nx;
        const long long o = lidx(2 * X, 2 * Y, 2 * Z, F.nx, F.ny), i = lidx(X, Y, Z, C.nx, C.ny);
        AF_PTR(const float) b = view((const float*)F.e, lvl_cells(F), DK_RESTRICT, s) + o;
        AF_PTR(const float) rb = view((const float*)F.r, lvl_cells(F), DK_RESTRICT, s) + o;
        if (F.v4) {
            AF_VEC(float2, cr, i, 2) = restrict_two<true>(F, b, rb, 2 * X, 2 * Y, 2 * Z, true, inv);
            AF_VEC(float2, ce, i, 2) = make_float2(0.0f, 0.0f);
        } else {
            const float2 m = restrict_two<false>(F, b, rb, 2 * X, 2 * Y, 2 * Z, two, inv);
            cr[i] = m.x;
            ce[i] = 0.0f;
            if (two) cr[i + 1] = m.y, ce[i + 1] = 0.0f;
        }
        continue;
    }
    const unsigned r = C.fnx.div(e), zz = C.fny.div(r);
    const int X = (int)(e - r * (unsigned)C.nx), Y = (int)(r - zz * (unsigned)C.ny), Z = (int)zz;
    float sum = 0.0f;
    for (int dz = 0; dz < ez; ++dz)
        for (int dy = 0; dy < ey; ++dy)
            for (int dx = 0; dx < ex; ++dx) sum += mg_residual(F, X * ex + dx, Y * ey + dy, Z * ez + dz, s);
    cr[el] = sum * inv;
    ce[el] = 0.0f;
    END_ELEMS
    END_TILES
}

// e_fine += cell-centred trilinear interpolation of e_coarse: per coarsened
// axis the parent weighs 3/4 and the next coarse cell toward the fine cell
// 1/4 (clamped at the walls, the Neumann reflection).  A row of 2^lg lanes
// owns one fine (y, z) row, whose four coarse rows are fixed; short rows
// (at most 16 lane iterations) share a warp two or four to a warp, so the
// per-row setup is not paid by idle lanes.  The iteration space counts 32
// lanes per warp (prolong_box).
// Where every axis coarsens, a work row is a coarse row (Y0, Z0) and covers
// the four fine rows (2 Y0 + {0, 1}, 2 Z0 + {0, 1}); a lane takes two coarse
// cells of it, four cells of each fine row: 27 coarse loads (9 of them wide
// where rows allow it, Lvl::v4) and 4 wide accesses of e each way for 16 fine
// cells, all of a step's loads issued before its stores.  Bound by memory: e
// is read and written once (8 bytes a fine cell).  Measured at 256^3 / 512^3,
// one coarse cell a lane / two: 34.7 / 26.5 and 352 / 211 us.  Otherwise a work
// row is a fine row.
__host__ __device__ inline bool prolong_blocks(const Lvl& F) { return F.cx && F.cy && F.cz; }
__host__ __device__ inline int prolong_lanes_log(const Lvl& F, const Lvl& C) {
    // Lane iterations of a row.
    const int w = prolong_blocks(F) ? (C.nx + 1) / 2 : (F.cx ? C.nx : F.nx);
    return w > 16 ? 5 : (w > 8 ? 4 : 3);
}
__host__ __device__ inline long long prolong_rows(const Lvl& F, const Lvl& C) {
    return prolong_blocks(F) ? (long long)C.ny * C.nz : (long long)F.ny * F.nz;
}
__host__ __device__ inline long long prolong_box(const Lvl& F, const Lvl& C) {
    const int sh = 5 - prolong_lanes_log(F, C);
    return 32ll * ((prolong_rows(F, C) + (1 << sh) - 1) >> sh);
}

// Fine rows (2 Y0 + b, 2 Z0 + c), b, c in {0, 1}.  Row b takes neighbour row
// Y0 + 1 if b else Y0 - 1, and likewise c (clamped at the walls, as the fine
// cells' neighbours are); operands and order are mg_interp's.
template <bool V4>
__device__ __forceinline__ void prolong_rows4(const Lvl& F, const Lvl& C, int Y0, int Z0, int lane, int lanes, int s) {
    AF_PTR(const float) AF_RESTRICT ce = view((const float*)C.e, lvl_cells(C), DK_PROLONG, s);
    AF_PTR(float) AF_RESTRICT fe = view(F.e, lvl_cells(F), DK_PROLONG, s);
    const int Ys[3] = {max(Y0 - 1, 0), Y0, min(Y0 + 1, C.ny - 1)};
    const int Zm = max(Z0 - 1, 0), Zp = min(Z0 + 1, C.nz - 1);
    const long long f0 = lidx(0, 2 * Y0, 2 * Z0, F.nx, F.ny), sy = F.nx, sz = (long long)F.nx * F.ny;
    auto lerp = [](float p, float q) { return __fmaf_rn(0.25f, q, __fmul_rn(0.75f, p)); };
    for (int X = 2 * lane; X < C.nx; X += 2 * lanes) {
        const bool two = X + 1 < C.nx;
        const int Xm = max(X - 1, 0), Xp = min(X + 2, C.nx - 1);
        // Coarse plane Z interpolated along x and y: v[b][x].
        auto plane = [&](int Z, float(&v)[2][4]) {
            float lx[3][4];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const long long o = lidx(0, Ys[b], Z, C.nx, C.ny);
                float c0, c1;
                if (V4) {
                    const float2 c = AF_VEC(const float2, ce, o + X, 2);
                    c0 = c.x, c1 = c.y;
                } else {
                    c0 = ce[o + X], c1 = ce[o + X + (two ? 1 : 0)];
                }
                lx[b][0] = lerp(c0, ce[o + Xm]);
                lx[b][1] = lerp(c0, c1);
                lx[b][2] = lerp(c1, c0);
                lx[b][3] = lerp(c1, ce[o + Xp]);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) v[0][x] = lerp(lx[1][x], lx[0][x]), v[1][x] = lerp(lx[1][x], lx[2][x]);
        };
        float here[2][4];
        plane(Z0, here);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const long long o = f0 + c * sz + 2 * X;
            float4 f[2];
            f[0] = ld_quad<V4>((AF_PTR(const float))fe, o, two);
            f[1] = ld_quad<V4>((AF_PTR(const float))fe, o + sy, two);
            float next[2][4];
            plane(c ? Zp : Zm, next);
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                float4 g = f[b];
                g.x = __fadd_rn(g.x, lerp(here[b][0], next[b][0]));
                g.y = __fadd_rn(g.y, lerp(here[b][1], next[b][1]));
                g.z = __fadd_rn(g.z, lerp(here[b][2], next[b][2]));
                g.w = __fadd_rn(g.w, lerp(here[b][3], next[b][3]));
                if (V4) {
                    AF_VEC(float4, fe, o + b * sy, 4) = g;
                } else {
                    AF_VEC(float2, fe, o + b * sy, 2) = make_float2(g.x, g.y);
                    if (two) AF_VEC(float2, fe, o + b * sy + 2, 2) = make_float2(g.z, g.w);
                }
            }
        }
    }
}

__global__ void __launch_bounds__(1024) kb_prolong(const InstDev* inst, const Ctl* ctl, Tab tab, int l, int vc) {
    begin_level(inst, tab, l, 2);
    if (vc_idle(ctl, tab.n, vc)) return;
    FOR_TILES(tab)
    if (mg_off(ctl[s], vc)) continue;
    const Lvl F = inst[s].lev[l];
    const Lvl C = inst[s].lev[l + 1];
    const long long rows = prolong_rows(F, C);
    const int lg = prolong_lanes_log(F, C), lanes = 1 << lg;
    FOR_ELEMS(tab)
    const long long row = ((el >> 5) << (5 - lg)) + ((el & 31) >> lg);
    if (row >= rows) break;
    const int lane = (int)(el & (lanes - 1));
    if (prolong_blocks(F)) {
        const unsigned cz = C.fny.div((unsigned)row);
        const int Y0 = (int)((unsigned)row - cz * (unsigned)C.ny), Z0 = (int)cz;
        if (F.v4) prolong_rows4<true>(F, C, Y0, Z0, lane, lanes, s);
        else prolong_rows4<false>(F, C, Y0, Z0, lane, lanes, s);
        continue;
    }
    const unsigned zz = F.fny.div((unsigned)row);
    const int y = (int)((unsigned)row - zz * (unsigned)F.ny), z = (int)zz;
    int Y0 = y, Y1 = y, Z0 = z, Z1 = z;
    float ay = 1.0f, az = 1.0f;
    if (F.cy) { Y0 = y >> 1; Y1 = min(max(Y0 + ((y & 1) ? 1 : -1), 0), C.ny - 1); ay = 0.75f; }
    if (F.cz) { Z0 = z >> 1; Z1 = min(max(Z0 + ((z & 1) ? 1 : -1), 0), C.nz - 1); az = 0.75f; }
    AF_PTR(const float) ce = view((const float*)C.e, lvl_cells(C), DK_PROLONG, s);
    AF_PTR(const float) c00 = ce + lidx(0, Y0, Z0, C.nx, C.ny);
    AF_PTR(const float) c10 = ce + lidx(0, Y1, Z0, C.nx, C.ny);
    AF_PTR(const float) c01 = ce + lidx(0, Y0, Z1, C.nx, C.ny);
    AF_PTR(const float) c11 = ce + lidx(0, Y1, Z1, C.nx, C.ny);
    AF_PTR(float) fe = view(F.e, lvl_cells(F), DK_PROLONG, s) + lidx(0, y, z, F.nx, F.ny);
    if (F.cx) {
        // A lane owns the fine pair (2X, 2X+1): both take parent X, the even
        // one neighbour X-1 and the odd one X+1 (clamped at the walls), so
        // the pair shares its coarse loads and one 8-byte access of e (nx is
        // even and every row starts on an even element).
        for (int X = lane; X < C.nx; X += lanes) {
            const int Xm = max(X - 1, 0), Xp = min(X + 1, C.nx - 1);
            const float a00 = c00[X], a10 = c10[X], a01 = c01[X], a11 = c11[X];
            float2 f = AF_VEC(float2, fe, 2 * X, 2);
            f.x = __fadd_rn(f.x, mg_interp(0.75f, ay, az, a00, c00[Xm], a10, c10[Xm], a01, c01[Xm], a11, c11[Xm]));
            f.y = __fadd_rn(f.y, mg_interp(0.75f, ay, az, a00, c00[Xp], a10, c10[Xp], a01, c01[Xp], a11, c11[Xp]));
            AF_VEC(float2, fe, 2 * X, 2) = f;
        }
    } else {
        for (int x = lane; x < F.nx; x += lanes)
            fe[x] = __fadd_rn(fe[x], mg_interp(1.0f, ay, az, c00[x], c00[x], c10[x], c10[x], c01[x], c01[x], c11[x],
                                               c11[x]));
    }
    END_ELEMS
    END_TILES
}

__device__ float block_sum(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        float s = threadIdx.x < kCoarseThreads / 32 ? red[threadIdx.x] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) red[0] = s;
    }
    __syncthreads();
    const float s = red[0];
    __syncthreads();
    return s;
}

// --- fused red-black pair ---------------------------------------------------
// One red sweep then one black sweep of L e = r, from e_in into e_out.  The
// red values read only e_in (their black neighbours are unchanged by the red
// sweep); the black values read the new red values.  Each block owns an
// output tile of TX x TY x TZ cells.  It first computes the new
// red values of the tile plus a one-cell halo -- only the red cells, kept
// compactly in shared memory (a row of the halo alternates colours, so
// x >> 1 indexes its red cells) -- then, after one barrier, each lane writes
// an adjacent (x, x+1) pair of the tile, one red cell (from shared memory)
// and one black cell (from its red neighbours there), so lanes never diverge
// on colour.  Nothing reads what the kernel writes, so blocks never race, and
// the result equals the two in-place colour sweeps bit for bit (mg_relax in
// both).  Per pair it moves e and r once and writes e once.
//
// Wide tiles (LANES = 32, TX = 64, a warp per row) cover x < nxw; a level
// whose x extent leaves 1..32 cells past the last wide tile (nx = 32, 96,
// ...) covers them with one narrow tile column (LANES = 16, TX = 32, a warp
// per two rows) instead of a half-idle wide tile.
//
// Three tile variants trade the red halo's recomputation (1.45x the tile's
// red cells at 16 x 8 rows and planes, 1.9x at 8 x 4, 2.3x at 4 x 4) against
// parallelism: a 64^3 level holds 32 of the largest tiles for 152 SMs.  The
// autotuner picks a variant per level; untuned, the level's size does.
// Variant 3 is the marching pair (kb_smooth_march) on the slots whose level
// allows it.
// Variant 4: 64 x 16 x 16 tiles, the red halo recomputed over 1.27x the
// tile's red cells.
constexpr int kPairVarTY[5] = {16, 8, 4, 0, 16}, kPairVarTZ[5] = {8, 4, 4, 0, 16};
constexpr int kPairTileVars[4] = {0, 1, 2, 4};
constexpr int kPairWideX = 64;

template <int LANES, int V>
struct PairTile {
    static constexpr int TY = kPairVarTY[V];
    static constexpr int TZ = kPairVarTZ[V];
    static constexpr int FY = V == 4 ? 0 : V;  // Lvl::fty entry of TY
    static constexpr int HY = TY + 2, HZ = TZ + 2;
    static constexpr int TX = 2 * LANES;        // cells along x
    static constexpr int RX = LANES + 1;        // red cells of a halo row
    static constexpr int RPW = 32 / LANES;      // tile rows per warp
    static constexpr int THREADS = TY * LANES;
    // Resident threads per SM the launch bounds ask for: all 2048 for the
    // largest tiles (32 registers suffice), 1536 for the others (their
    // index arithmetic would spill at 32).
    static constexpr int RESIDENT = V == 0 || V == 4 ? 2048 : 1536;
};

template <int LANES, int V>
__global__ void __launch_bounds__(PairTile<LANES, V>::THREADS, PairTile<LANES, V>::RESIDENT / PairTile<LANES, V>::THREADS)
    kb_smooth_pair(const InstDev* inst, const Ctl* ctl, Tab tab, int l, int dir, int vc) {
    begin_level(inst, tab, l, 1);
    if (vc_idle(ctl, tab.n, vc)) return;
    using T = PairTile<LANES, V>;
    __shared__ float red[T::HZ][T::HY][T::RX];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k = lane % LANES;                        // pair of the row
    const int wrow = warp * T::RPW + lane / LANES;     // tile row, 0 .. TY-1
    for (int item = blockIdx.x, total = tab.prefix[tab.n]; item < total; item += gridDim.x) {
        const int s = find_slot(tab.prefix, tab.n, item);
        if (mg_off(ctl[s], vc)) continue;
        const Lvl L = inst[s].lev[l];
        AF_PTR(const float) AF_RESTRICT ein = view((const float*)(dir ? L.e2 : L.e), lvl_cells(L), DK_PAIR, s);
        AF_PTR(float) AF_RESTRICT eout = view(dir ? L.e : L.e2, lvl_cells(L), DK_PAIR, s);
        AF_PTR(const float) AF_RESTRICT r = view((const float*)L.r, lvl_cells(L), DK_PAIR, s);
        const int nx = L.nx, ny = L.ny, nz = L.nz, nxy = nx * ny;  // a level holds < 2^31 cells
        const unsigned local = (unsigned)(item - tab.prefix[s]);
        int x0, y0, z0;
        if (LANES == 32) {
            const unsigned q1 = L.ftx.div(local), q2 = L.fty[T::FY].div(q1);
            x0 = (int)(local - q1 * L.ftx.d) * T::TX;
            y0 = (int)(q1 - q2 * L.fty[T::FY].d) * T::TY;
            z0 = (int)q2 * T::TZ;
        } else {
            const unsigned q2 = L.fty[T::FY].div(local);
            x0 = L.nxw;
            y0 = (int)(local - q2 * L.fty[T::FY].d) * T::TY;
            z0 = (int)q2 * T::TZ;
        }
        const float inv = 1.0f / (2.0f * (L.wx + L.wy + L.wz));
        // Red cells of the halo tile, a row of lanes per halo row (hy, hz):
        // halo x = x0 - 1 + hx, hx = 2j + ((y + z + 1) & 1); lanes take
        // j < LANES and the rows' last cells (j = LANES) go one per thread
        // afterwards.
        auto red_row = [&](int hy, int hz, int j) {
            const int y = y0 - 1 + hy, z = z0 - 1 + hz;
            const int x = x0 - 1 + 2 * j + ((y + z + 1) & 1);
            float v = 0.0f;
            if ((unsigned)x < (unsigned)nx && (unsigned)y < (unsigned)ny && (unsigned)z < (unsigned)nz) {
                const int i = x + nx * y + nxy * z;
                const int oym = y > 0 ? -nx : 0, oyp = y < ny - 1 ? nx : 0;
                const int ozm = z > 0 ? -nxy : 0, ozp = z < nz - 1 ? nxy : 0;
                const int oxm = x > 0 ? -1 : 0, oxp = x < nx - 1 ? 1 : 0;
                AF_PTR(const float) p = ein + i;
                v = mg_relax(L, p[oxm] + p[oxp], p[oym] + p[oyp], p[ozm] + p[ozp], r[i], inv, p[0]);
            }
            red[hz][hy][j] = v;
        };
        for (int row = wrow; row < T::HY * T::HZ; row += T::TY) red_row(row % T::HY, row / T::HY, k);
        for (int row = tid; row < T::HY * T::HZ; row += T::THREADS)
            red_row(row % T::HY, row / T::HY, LANES);
        __syncthreads();
        // Output pairs: lane k -> x = x0 + 2k + {0, 1}, tile row -> y, loop over z.
        const int y = y0 + wrow, hy = wrow + 1;
        const int xa = x0 + 2 * k;
        if (y < ny && xa < nx) {
            const int zend = min(T::TZ, nz - z0);
            int i0 = xa + nx * y + nxy * z0;
            for (int tz = 0; tz < zend; ++tz, i0 += nxy) {
                const int z = z0 + tz, hz = tz + 1;
                // Of the pair, the red cell is xa + pr and the black one xa + 1 - pr.
                const int pr = (xa + y + z) & 1;
                const int xr = xa + pr, xb = xa + 1 - pr;
                if (xr < nx) eout[i0 + pr] = red[hz][hy][(xr - x0 + 1) >> 1];
                if (xb < nx) {
                    const int h = (xb - x0 + 1) >> 1, hm = (xb - x0) >> 1, hp = (xb - x0 + 2) >> 1;
                    const int ib = i0 + 1 - pr;
                    const float c = ein[ib];
                    const float sx = (xb > 0 ? red[hz][hy][hm] : c) + (xb < nx - 1 ? red[hz][hy][hp] : c);
                    const float sy = (y > 0 ? red[hz][hy - 1][h] : c) + (y < ny - 1 ? red[hz][hy + 1][h] : c);
                    const float sz = (z > 0 ? red[hz - 1][hy][h] : c) + (z < nz - 1 ? red[hz + 1][hy][h] : c);
                    eout[ib] = mg_relax(L, sx, sy, sz, r[ib], inv, c);
                }
            }
        }
        __syncthreads();
    }
}

// --- marching fused pair -----------------------------------------------------
// The red-black pair of kb_smooth_pair with each thread owning a quad (four
// consecutive cells of a row, two red and two black on every plane) and
// marching along z with its column of e, r and red values in registers: a
// plane costs a quad 16-byte loads of e two planes ahead, of r one plane
// ahead and of the two rows beside it, one scalar across the quad's end, and
// one 16-byte store.  Red values of a plane are exchanged with the rows and
// quads beside it through a ring of four planes in shared memory: in the
// iteration that computes the red cells of plane z, a thread computes the black
// ones of plane z - 1, whose neighbours' red cells the barrier of that plane
// published.
//
// A tile is a column of at most kMarchQ quads by March::rows rows; its block
// also computes the red cells of the row on either side, of the quad on
// either side where the level has several columns, and of the plane on
// either side of its z chunk.  Walls cost no selects: a row or plane outside
// the level stands in with the row or plane of the wall cells it faces, and
// its "red" values are their old ones, which is what the black cells beside
// it use.  Operands and their order are those of kb_smooth_pair: the same
// bits.
//
// A plane's operands load into the registers that the plane before has just
// used, between its red and its black cells: no copy waits for a load, and
// the loads have the black cells, the barrier and the other warps to land.
//
// A warp waits for the other warps' red cells of the last plane, not of this
// one, on a barrier that splits arriving from waiting (a block-wide barrier a
// plane left the block idle half the time: 57 us instead of 41 at 256^3).
//
// A level runs it when rows and arrays are 16-byte aligned (nx a multiple
// of 4).  Measured per pair against the best tiles, us: finest levels of
// 512^3 541 -> 323 and 256^3 69 -> 41 (39 of them on the device, 200 MB at
// 5 TB/s, issue 60 % active), 128^3 14.7 -> 12.6, the 256-grid batch 504 ->
// 250.  Block sizes: 1024 threads on 64 quads (one block an SM) for long
// rows, two of 576 on 32 quads for many middling ones, four of 256 for small
// levels; prefetching further planes to L2 gained nothing.
constexpr int kMarchT[3] = {256, 576, 1024}, kMarchQ[3] = {16, 32, 64}, kMarchBlocks[3] = {4, 2, 1};
// Launch shapes the autotuner tries: block size (index into kMarchT) and
// planes of a z chunk.
struct MarchShape {
    int k, zc;
};
constexpr MarchShape kMarchShapes[] = {{0, 4}, {0, 8}, {0, 16}, {1, 8}, {1, 16}, {1, 32}, {2, 16}, {2, 32}};
constexpr int kMarchShapeCount = sizeof kMarchShapes / sizeof kMarchShapes[0];

__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Waits for the block's own warps only: all are resident, wait for nothing
// else and arrive on every plane.  The wait is bounded all the same: `polls`
// here, then, in a function of its own, 2^16 times as many and, as a transfer's
// wait, kWaitLimitNs.  A wait that gives up records it, which makes the call an
// error; the thread goes on, so that its warp still arrives for the others, and
// the work's later waits end after their first polls.  (Looking at the record
// at every launch's start instead is a load in its way: 48x32x64 1.51 -> 1.61
// ms a Step.)
constexpr unsigned kMarchPolls = 64;
__device__ __noinline__ void march_wait_long(unsigned long long* bar, unsigned parity, unsigned polls, unsigned* diag) {
    const unsigned long long t0 = global_ns();
    for (unsigned it = 0; it < polls << 16; ++it) {
        if (mbar_try_wait(bar, parity)) return;
        if ((it & 63u) == 0u && (diag_set(diag) || global_ns() - t0 > kWaitLimitNs)) break;
    }
    atomicOr(diag, 2u);
}
__device__ __forceinline__ void march_wait(unsigned long long* bar, unsigned parity, unsigned polls, unsigned* diag) {
    for (unsigned it = 0; it < polls; ++it)
        if (mbar_try_wait(bar, parity)) return;
    march_wait_long(bar, parity, polls, diag);
}

template <int K>
__global__ void __launch_bounds__(kMarchT[K], kMarchBlocks[K])
    kb_smooth_march(const InstDev* inst, const Ctl* ctl, Tab tab, int l, int dir, int vc, int zc, unsigned polls,
                    unsigned* diag) {
    begin_level(inst, tab, l, 1);
    if (vc_idle(ctl, tab.n, vc)) return;
    constexpr int T = kMarchT[K];
    __shared__ float2 ring[4][T];
    __shared__ __align__(8) unsigned long long bar[2];
    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&bar[0], T / 32);
        mbar_init(&bar[1], T / 32);
    }
    __syncthreads();
    unsigned n = 0;  // planes this block has marched over
    for (int item = blockIdx.x, total = tab.prefix[tab.n]; item < total; item += gridDim.x) {
        const int s = find_slot(tab.prefix, tab.n, item);
        if (mg_off(ctl[s], vc)) continue;
        const Lvl& L = inst[s].lev[l];
        AF_PTR(const float) AF_RESTRICT ein = view((const float*)(dir ? L.e2 : L.e), lvl_cells(L), DK_PAIR, s);
        AF_PTR(float) AF_RESTRICT eout = view(dir ? L.e : L.e2, lvl_cells(L), DK_PAIR, s);
        AF_PTR(const float) AF_RESTRICT r = view((const float*)L.r, lvl_cells(L), DK_PAIR, s);
        const int nx = L.nx, ny = L.ny, nz = L.nz, nxy = nx * ny, mq = L.march[K].q, mw = L.march[K].w;
        const int mrows = L.march[K].rows;
        const MgW W{L.wx, L.wy, L.wz};
        const float inv = 1.0f / (2.0f * (L.wx + L.wy + L.wz));
        const unsigned local = (unsigned)(item - tab.prefix[s]);
        const unsigned t1 = L.march[K].fcol.div(local), t2 = L.march[K].fty.div(t1);
        const int q0 = (int)(local - t1 * L.march[K].fcol.d) * mw;  // first output quad
        const int y0 = (int)(t1 - t2 * L.march[K].fty.d) * mrows;
        const int z0 = (int)t2 * zc, zl = min(z0 + zc, nz);  // output planes z0 .. zl-1
        const int row = (int)L.march[K].fq.div((unsigned)tid), rows = min(mrows, ny - y0);
        const int xq = q0 - (q0 > 0 ? 1 : 0) + tid - row * mq, x = 4 * xq;
        const int y = y0 - 1 + row, yc = min(max(y, 0), ny - 1);
        const bool in_y = y == yc;
        const bool active = row < rows + 2 && x < nx && xq < q0 + mw + 1;
        const bool out = active && row >= 1 && row <= rows && xq >= q0 && xq < q0 + mw;
        const int i0 = x + nx * yc;                    // the quad in its (wall-clamped) row
        const int on = in_y && y > 0 ? -nx : 0, os = in_y && y < ny - 1 ? nx : 0;
        // The cell across the quad's end that a red cell needs: left of it
        // when the red cells are 0 and 2, right when they are 1 and 3 (the
        // quad's own end cell at an x wall).
        const int xl = x > 0 ? -1 : 0, xr = x + 4 < nx ? 4 : 3;
        auto quad = [&](AF_PTR(const float) p) { return AF_VEC(const float4, p, 0, 4); };
        float4 ec{}, ep{}, rc{}, N{}, S{};
        float xs = 0.0f;
        float2 em{}, rb{}, red1{}, red2{};  // e (plane z-1) and r (z-1) at plane z's red positions; red of z-1, z-2
        int pr = (y + z0 - 1) & 1;          // the red cells of plane z are pr and pr + 2
        // The quad at plane z (e) and z + 1 (e), at z (r) and at z - 1 (out);
        // planes outside the level are the wall plane.
        const int zf = max(z0 - 1, 0);
        AF_PTR(const float) pe = ein + (i0 + zf * nxy);
        AF_PTR(const float) pn = ein + (i0 + z0 * nxy);
        AF_PTR(const float) pv = r + (i0 + zf * nxy);
        AF_PTR(float) po = eout + (i0 + z0 * nxy);
        if (active) {
            const float4 e0 = quad(ein + (i0 + max(z0 - 2, 0) * nxy));
            ec = quad(pe);
            ep = quad(pn);
            rc = quad(pv);
            N = quad(pe + on);
            S = quad(pe + os);
            xs = pe[pr ? xr : xl];
            em = pr ? make_float2(e0.y, e0.w) : make_float2(e0.x, e0.z);
        }
        for (int z = z0 - 1; z <= zl; ++z, ++n) {
            float2 red{}, eb{}, rv{};
            if (active) {
                const bool in = in_y && (unsigned)z < (unsigned)nz;
                const float c0 = pr ? ec.y : ec.x, c1 = pr ? ec.w : ec.z;
                const float sx0 = (pr ? ec.x : xs) + (pr ? ec.z : ec.y), sx1 = (pr ? ec.z : ec.y) + (pr ? xs : ec.w);
                const float sy0 = (pr ? N.y : N.x) + (pr ? S.y : S.x), sy1 = (pr ? N.w : N.z) + (pr ? S.w : S.z);
                const float v0 = mg_relax(W, sx0, sy0, em.x + (pr ? ep.y : ep.x), pr ? rc.y : rc.x, inv, c0);
                const float v1 = mg_relax(W, sx1, sy1, em.y + (pr ? ep.w : ep.z), pr ? rc.w : rc.z, inv, c1);
                red = in ? make_float2(v0, v1) : make_float2(c0, c1);
                ring[n & 3u][tid] = red;
                // Plane z + 1's red positions are plane z's black ones.
                eb = em, rv = rb;
                em = pr ? make_float2(ec.x, ec.z) : make_float2(ec.y, ec.w);
                rb = pr ? make_float2(rc.x, rc.z) : make_float2(rc.y, rc.w);
                ec = ep;
                if (z < zl) {  // the next plane's operands
                    pe = pn;
                    if (z >= 0 && z + 1 < nz) pv += nxy;  // r's plane z + 1, e's plane z + 2
                    if (z + 2 < nz) pn += nxy;
                    ep = quad(pn);
                    rc = quad(pv);
                    N = quad(pe + on);
                    S = quad(pe + os);
                    xs = pe[pr ? xl : xr];
                }
            }
            // Publish this plane's red cells; then wait for the last one's.
            // A warp runs at most a plane ahead of the others: its ring slot
            // was last read three planes ago.
            __syncwarp();
            if ((tid & 31) == 0) mbar_arrive(&bar[n & 1u]);
            if (n > 0) march_wait(&bar[(n - 1u) & 1u], ((n - 1u) >> 1) & 1u, polls, diag);
            if (active) {
                if (z > z0) {
                    if (out) {
                        // Black cells of plane z - 1, at plane z's red
                        // positions: their old values are eb, their r rv, the
                        // red cells below and above red2 and red, beside them
                        // red1.
                        const float2* rg = ring[(n - 1u) & 3u];
                        const float2 n = rg[tid - mq], u = rg[tid + mq];
                        // Across the quad's end: the next quad's first red
                        // cell (black 1 and 3) or the previous one's last.
                        float e;
                        if (pr) e = x + 4 < nx ? rg[tid + 1].x : eb.y;
                        else e = x > 0 ? rg[tid - 1].y : eb.x;
                        const float mid = red1.x + red1.y;
                        const float sb0 = pr ? mid : e + red1.x, sb1 = pr ? red1.y + e : mid;
                        const float b0 = mg_relax(W, sb0, n.x + u.x, red2.x + red.x, rv.x, inv, eb.x);
                        const float b1 = mg_relax(W, sb1, n.y + u.y, red2.y + red.y, rv.y, inv, eb.y);
                        AF_VEC(float4, po, 0, 4) =
                            pr ? make_float4(red1.x, b0, red1.y, b1) : make_float4(b0, red1.x, b1, red1.y);
                    }
                    po += nxy;
                }
                red2 = red1, red1 = red;
                pr ^= 1;
            }
        }
    }
}

// --- tail V-cycle: every level from the slot's tail down, in one block -------
// Levels of at most kCoarseMax cells live in shared memory: pre-smoothing and
// restriction down to the coarsest level, its solve (the mean of r removed --
// a Neumann problem is solvable only for zero-mean data -- red-black sweeps
// from zero, the mean of e removed), then prolongation and post-smoothing
// back up.  Sums use a fixed tree.  Replaces one launch per level and sweep.
//
// It is a chain of short phases, so each is kept short.  e carries a ghost
// cell on each side of every axis longer than one cell, which always holds
// the value of the wall cell beside it (the Neumann reflection; an update of
// a wall cell writes its ghosts too), so neighbours sit at fixed offsets
// without tests.  A thread keeps its cells of a level -- index, walls, r and
// its own e -- in registers over all of the level's sweeps.  From the first
// level of at most a cell of a colour a lane (kWarpSlots) on, one warp runs the
// rest of the way down and back up with warp barriers instead of block ones.
// With two to four cells a lane it is slower than the block, above all on
// coarsest levels of odd extents, which take many sweeps: ms a Step at 128, 64
// and 32 slots 20^3 1.36, 0.93, 0.93, 15x15x1 2.94, 0.92, 0.92, 9x9x1 0.78, 0.78,
// 0.45, 12x20x28 1.93, 1.12, 1.12, 48x32x64 1.40, 1.35, 1.35.
// A visit's loops appear once and work on copies of its levels' records, and
// shared memory is indexed as such: the chain otherwise waits on instruction
// fetches and generic loads.  Measured per Step with index decoding, wall
// tests and block barriers in every sweep / so: 16^3 (a tail alone, 14
// V-cycles) 0.72 / 0.59 ms, 48x32x64 1.44 / 1.35 ms, 256^3 10.40 / 10.27 ms.
constexpr int kWarpSlots = 32;  // at most the lanes of a warp
// The most dynamic shared memory a tail takes (plan_tail): ghost cells on
// every side make the thinnest hierarchy, 2 x 2 x 1024 cells, the largest.  The
// limit belongs to the kernel, not to a batch, so every batch sets this one: a
// batch that set its own would take it from another on another thread.
constexpr int kTailSmem = 181344;

// A level's layout in shared memory: strides along the axes (0 along an axis
// of extent 1), offset of cell (0, 0, 0) and floats of e; r is unpadded.
struct SmLvl {
    int nx, ny, nz, hx, dx, dy, dz, o, size;
    SmLvl() = default;
    __host__ __device__ explicit SmLvl(const Lvl& L) : nx(L.nx), ny(L.ny), nz(L.nz), hx((L.nx + 1) / 2) {
        const int px = nx > 1 ? nx + 2 : 1, py = ny > 1 ? ny + 2 : 1, pz = nz > 1 ? nz + 2 : 1;
        dx = nx > 1 ? 1 : 0;
        dy = ny > 1 ? px : 0;
        dz = nz > 1 ? px * py : 0;
        o = dx + dy + dz;
        size = px * py * pz;
    }
    __host__ __device__ int cells() const { return nx * ny * nz; }
    __host__ __device__ int slots() const { return hx * ny * nz; }  // of one colour
    __host__ __device__ bool thin() const { return nx == 2 || ny == 2 || nz == 2; }  // every cell at a wall
};

// What the tail reads of a level, in shared memory: its layout, the places of
// e (cell (0, 0, 0)) and r, weights, dividers, the axes that coarsen.
struct TailLvl {
    SmLvl S;
    MgW W;
    float inv;  // of the relaxation
    int e, e0, r;  // cell (0, 0, 0) and start of e, start of r
    int res;       // residuals of the level being restricted
    int cx, cy, cz;
    FastDiv fnx, fny, fhx;
    // Which walls a cell touches: bit 0 x low, 1 x high, 2 y low, ...
    __device__ __forceinline__ unsigned walls(int x, int y, int z) const {
        unsigned w = 0;
        if (S.nx > 1) w |= (x == 0 ? 1u : 0u) | (x == S.nx - 1 ? 2u : 0u);
        if (S.ny > 1) w |= (y == 0 ? 4u : 0u) | (y == S.ny - 1 ? 8u : 0u);
        if (S.nz > 1) w |= (z == 0 ? 16u : 0u) | (z == S.nz - 1 ? 32u : 0u);
        return w;
    }
    __device__ __forceinline__ int at(int x, int y, int z) const { return e + x * S.dx + y * S.dy + z * S.dz; }
    // Cell of linear index i.
    __device__ __forceinline__ void cell(int i, int* x, int* y, int* z) const {
        const unsigned q = fnx.div((unsigned)i), zz = fny.div(q);
        *x = i - (int)q * S.nx, *y = (int)q - (int)zz * S.ny, *z = (int)zz;
    }
};

// The tail's dynamic shared memory, indexed as such (a pointer handed to a
// function would make every access a generic one); the bounds-checking build
// checks the index.
struct TailMem {
    int n, slot;
    __device__ __forceinline__ float& operator[](int i) const {
        extern __shared__ __align__(128) float tail_smem[];
#if AEROFLUX_DEBUG_BOUNDS
        return view(tail_smem, (long long)n, DK_VTAIL, slot)[i];
#else
        return tail_smem[i];
#endif
    }
};

__device__ __forceinline__ void tail_put(const TailMem& M, const SmLvl& S, int i, unsigned w, float v) {
    M[i] = v;
    if (w) {
        if (w & 1u) M[i - S.dx] = v;
        if (w & 2u) M[i + S.dx] = v;
        if (w & 4u) M[i - S.dy] = v;
        if (w & 8u) M[i + S.dy] = v;
        if (w & 16u) M[i - S.dz] = v;
        if (w & 32u) M[i + S.dz] = v;
    }
}

// The threads that run a level: the block, or its first warp.
template <bool WARP>
struct TailGroup {
    static constexpr int N = WARP ? 32 : kCoarseThreads;
    static __device__ __forceinline__ int id() { return (int)threadIdx.x; }
    static __device__ __forceinline__ void sync() {
        if (WARP) __syncwarp();
        else __syncthreads();
    }
};

// `pairs` red-black pairs of a level, NC cells of a colour a thread at most.
template <bool WARP, int NC>
__device__ __forceinline__ void tail_smooth_n(const TailMem& M, const TailLvl& L, int pairs) {
    using Gr = TailGroup<WARP>;
    const SmLvl S = L.S;
    const MgW W = L.W;
    const float inv = L.inv;
    int at[2][NC];  // walls << 20 | index; -1: none
    float rr[2][NC], own[2][NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const int m = Gr::id() + k * Gr::N;
        const unsigned q = L.fhx.div((unsigned)m), zz = L.fny.div(q);
        const int j = m - (int)q * S.hx, y = (int)q - (int)zz * S.ny, z = (int)zz;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int x = 2 * j + (((y + z) & 1) != c ? 1 : 0);
            at[c][k] = -1;
            rr[c][k] = own[c][k] = 0.0f;
            if (m < S.slots() && x < S.nx) {
                const int i = L.at(x, y, z);
                at[c][k] = (int)(L.walls(x, y, z) << 20) | i;
                rr[c][k] = M[L.r + x + S.nx * (int)q];
                own[c][k] = M[i];
            }
        }
    }
    for (int p = 0; p < pairs; ++p)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int k = 0; k < NC; ++k)
                if (at[c][k] >= 0) {
                    const int i = at[c][k] & 0xFFFFF;
                    const float v = mg_relax(W, M[i - S.dx] + M[i + S.dx], M[i - S.dy] + M[i + S.dy],
                                             M[i - S.dz] + M[i + S.dz], rr[c][k], inv, own[c][k]);
                    own[c][k] = v;
                    tail_put(M, S, i, (unsigned)at[c][k] >> 20, v);
                }
            Gr::sync();
        }
}

// Many pairs (a coarsest level's solve) of a level of at most a cell of a
// colour a thread.  A neighbour across a wall is the cell itself here, by its
// index, and the ghosts, which only the phases around the sweeps read, are
// written by the last pair: on thin levels every cell lies at two to four
// walls.  ms a Step with ghosts in every pair / so: 8x4x194 7.42 / 5.40, 2x2x97
// 31.2 / 22.7, 15x15x1 0.92 / 0.82, 5x7x9 0.55 / 0.49.  For few pairs its set-up
// costs more than it saves, and its presence alone costs the other levels
// registers (16^3 0.613 / 0.656, 48x32x64 with 18 pairs 1.305 / 1.34), so only the
// forms with MANY hold it.
constexpr int kManyPairs = 32;
template <bool WARP>
__device__ __noinline__ void tail_smooth_many(const TailMem M, const TailLvl* lv, int pairs) {
    using Gr = TailGroup<WARP>;
    const TailLvl L = *lv;
    const SmLvl& S = L.S;
    const MgW W = L.W;
    const float inv = L.inv;
    const int m = Gr::id();
    const unsigned q = L.fhx.div((unsigned)m), zz = L.fny.div(q);
    const int j = m - (int)q * S.hx, y = (int)q - (int)zz * S.ny, z = (int)zz;
    int at[2], nb[2][6];
    unsigned walls[2];
    float rr[2], own[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int x = 2 * j + (((y + z) & 1) != c ? 1 : 0);
        at[c] = -1;
        if (m < S.slots() && x < S.nx) {
            const int i = L.at(x, y, z);
            at[c] = i;
            walls[c] = L.walls(x, y, z);
            rr[c] = M[L.r + x + S.nx * (int)q];
            own[c] = M[i];
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const int d = k < 2 ? S.dx : (k < 4 ? S.dy : S.dz);
                nb[c][k] = (walls[c] >> k) & 1u ? i : (k & 1 ? i + d : i - d);
            }
        }
    }
    for (int p = 0; p < pairs; ++p)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (at[c] >= 0) {
                const float v = mg_relax(W, M[nb[c][0]] + M[nb[c][1]], M[nb[c][2]] + M[nb[c][3]],
                                         M[nb[c][4]] + M[nb[c][5]], rr[c], inv, own[c]);
                own[c] = v;
                if (p + 1 < pairs) M[at[c]] = v;
                else tail_put(M, S, at[c], walls[c], v);
            }
            Gr::sync();
        }
}

// The same for levels of more than four slots a thread (rows of few cells waste
// half of theirs) and thin ones of more than one: a coarsest level, its e zero, in
// the space of its padded e but without ghosts, so that a register holds a cell's
// place and walls over all sweeps; then spread over the padded layout.  ms a Step
// decoding in every sweep / with fixed offsets and ghosts / so: 1x63x65 58 / 80 /
// 41, 7x23x25 14.1 / 22.5 / 11.9, 2x45x45 39.5 / 54 / 24, 2x173x7 156 / 192 / 106; fixed
// offsets are better for the others of up to four (5x15x41 26.7 / 20.9).
template <int NC>
__device__ __noinline__ void tail_solve_plain(const TailMem M, const TailLvl* lv, int pairs) {
    const TailLvl L = *lv;
    const SmLvl& S = L.S;
    const int n = S.cells(), nx = S.nx, nxy = S.nx * S.ny, r = L.r - L.e0;
    const MgW W = L.W;
    const float inv = L.inv;
    int at[2][NC];  // walls << 20 | place of e, -1: none
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const int m = (int)threadIdx.x + k * kCoarseThreads;
        const unsigned q = L.fhx.div((unsigned)m), zz = L.fny.div(q);
        const int j = m - (int)q * S.hx, y = (int)q - (int)zz * S.ny, z = (int)zz;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int x = 2 * j + (((y + z) & 1) != c ? 1 : 0);
            unsigned w = (x == 0 ? 1u : 0u) | (x == nx - 1 ? 2u : 0u) | (y == 0 ? 4u : 0u) | (y == S.ny - 1 ? 8u : 0u) |
                         (z == 0 ? 16u : 0u) | (z == S.nz - 1 ? 32u : 0u);
            at[c][k] = m < S.slots() && x < nx ? (int)(w << 20) | (L.e0 + x + nx * (int)q) : -1;
        }
    }
    for (int p = 0; p < pairs; ++p)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int k = 0; k < NC; ++k)
                if (at[c][k] >= 0) {
                    const int e = at[c][k] & 0xFFFFF;
                    const unsigned w = (unsigned)at[c][k] >> 20;
                    const float o = M[e];
                    const float sx = (w & 1u ? o : M[e - 1]) + (w & 2u ? o : M[e + 1]);
                    const float sy = (w & 4u ? o : M[e - nx]) + (w & 8u ? o : M[e + nx]);
                    const float sz = (w & 16u ? o : M[e - nxy]) + (w & 32u ? o : M[e + nxy]);
                    M[e] = mg_relax(W, sx, sy, sz, M[e + r], inv, o);
                }
            __syncthreads();
        }
    float v[kCoarseMax / kCoarseThreads];
#pragma unroll
    for (int k = 0; k < kCoarseMax / kCoarseThreads; ++k) {
        const int i = (int)threadIdx.x + k * kCoarseThreads;
        if (i < n) v[k] = M[L.e0 + i];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kCoarseMax / kCoarseThreads; ++k) {
        const int i = (int)threadIdx.x + k * kCoarseThreads;
        if (i < n) {
            int x, y, z;
            L.cell(i, &x, &y, &z);
            tail_put(M, S, L.at(x, y, z), L.walls(x, y, z), v[k]);
        }
    }
    __syncthreads();
}

// Thin levels of more slots than four a thread (half of a row's slots may be
// of no colour): decoded in every sweep.
__device__ __noinline__ void tail_smooth_thin(const TailMem M, const TailLvl* lv, int pairs) {
    const TailLvl L = *lv;
    const SmLvl& S = L.S;
    for (int p = 0; p < 2 * pairs; ++p) {
        for (int m = (int)threadIdx.x; m < S.slots(); m += kCoarseThreads) {
            const unsigned q = L.fhx.div((unsigned)m), zz = L.fny.div(q);
            const int j = m - (int)q * S.hx, y = (int)q - (int)zz * S.ny, z = (int)zz;
            const int x = 2 * j + (((y + z) & 1) != (p & 1) ? 1 : 0);
            if (x >= S.nx) continue;
            const int i = L.at(x, y, z);
            const float v = mg_relax(L.W, M[i - S.dx] + M[i + S.dx], M[i - S.dy] + M[i + S.dy],
                                     M[i - S.dz] + M[i + S.dz], M[L.r + x + S.nx * (int)q], L.inv, M[i]);
            tail_put(M, S, i, L.walls(x, y, z), v);
        }
        __syncthreads();
    }
}

// Sum over the coarsest level's cells in the fixed order of 512 threads: a
// partial each over cells i, i + 512, ..., a shuffle tree over each warp, one
// over the warps.  One warp forms the same tree where the level has at most
// 64 cells.
template <bool WARP, class F>
__device__ __forceinline__ float tail_sum(int n, float* red, F cell) {
    if (!WARP) {
        float part = 0.0f;
        for (int i = (int)threadIdx.x; i < n; i += kCoarseThreads) part += cell(i);
        return block_sum(part, red);
    }
    const int lane = (int)threadIdx.x;
    float mine = 0.0f;
    for (int w = 0; w * 32 < n; ++w) {
        const int i = w * 32 + lane;
        float v = i < n ? 0.0f + cell(i) : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == w) mine = v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    return __shfl_sync(0xffffffffu, mine, 0);
}

// Levels l0 .. nl - 1 (lv[l]): down, the coarsest solve, and back up to l0.
// One loop over the visits, each part of a visit written once (the chain of
// short phases waits on instruction fetches otherwise); a visit works on a
// copy of its levels' records (stores could alias the table).
template <bool WARP, bool SMALL, bool MANY>
__device__ __noinline__ void tail_levels(const TailMem M, const TailLvl* lv, int l0, int nl, int coarse_sweeps,
                                         float* red, int nu) {
    using Gr = TailGroup<WARP>;
    bool up = false;
    for (int l = l0; l >= l0;) {
        if (!WARP && !up && lv[l].S.slots() <= kWarpSlots) {
            if (threadIdx.x < 32) tail_levels<true, SMALL, MANY>(M, lv, l, nl, coarse_sweeps, red, nu);
            __syncthreads();
            up = true;
            --l;
            continue;
        }
        const TailLvl F = lv[l];
        const bool coarsest = l == nl - 1;
        const int n = F.S.cells();
        if (up) {  // prolongation
            const TailLvl C = lv[l + 1];
            // A thread takes the fine cells 2X and 2X + 1 of a parent column X
            // where x coarsens: they share four coarse values.  The next coarse
            // cell toward the fine one is the parent again across a wall (edge
            // and corner ghosts are unset).
            const float ax = F.cx ? 0.75f : 1.0f, ay = F.cy ? 0.75f : 1.0f, az = F.cz ? 0.75f : 1.0f;
            const int items = C.S.nx * F.S.ny * F.S.nz;
            for (int j = Gr::id(); j < items; j += Gr::N) {
                const unsigned q = C.fnx.div((unsigned)j), zz = F.fny.div(q);
                const int X = j - (int)q * C.S.nx, y = (int)q - (int)zz * F.S.ny, z = (int)zz;
                const int Y = F.cy ? y >> 1 : y, Z = F.cz ? z >> 1 : z;
                auto toward = [](int coarsens, int f, int c, int m, int d) {
                    return !coarsens ? 0 : ((f & 1) ? (c < m - 1 ? d : 0) : (c > 0 ? -d : 0));
                };
                const int k = C.at(X, Y, Z);
                const int oy = toward(F.cy, y, Y, C.S.ny, C.S.dy), oz = toward(F.cz, z, Z, C.S.nz, C.S.dz);
                const float a = M[k], b = M[k + oy], c = M[k + oz], d = M[k + oz + oy];
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    if (o && !F.cx) break;
                    const int x = F.cx ? 2 * X + o : X, ox = toward(F.cx, o, X, C.S.nx, C.S.dx);
                    const float v = mg_interp(ax, ay, az, a, M[k + ox], b, M[k + oy + ox], c, M[k + oz + ox], d,
                                              M[k + oz + oy + ox]);
                    const int i = F.at(x, y, z);
                    tail_put(M, F.S, i, F.walls(x, y, z), __fadd_rn(M[i], v));
                }
            }
            Gr::sync();
        }
        if (coarsest) {
            const float mean_r = tail_sum<WARP>(n, red, [&](int i) { return M[F.r + i]; }) / (float)n;
            for (int i = Gr::id(); i < n; i += Gr::N) M[F.r + i] -= mean_r;
            for (int i = Gr::id(); i < F.S.size; i += Gr::N) M[F.e0 + i] = 0.0f;
            Gr::sync();
        }
        const int pairs = coarsest ? coarse_sweeps : nu;
        // WARP: at most kWarpSlots slots; SMALL: at most kCoarseThreads.
        const bool many = MANY && pairs > kManyPairs;
        if (WARP || SMALL || F.S.slots() <= Gr::N) {
            if (many) tail_smooth_many<WARP>(M, lv + l, pairs);
            else tail_smooth_n<WARP, 1>(M, F, pairs);
        } else if (F.S.slots() <= 4 * Gr::N) {
            if (many && F.S.thin()) tail_solve_plain<4>(M, lv + l, pairs);
            else tail_smooth_n<WARP, 4>(M, F, pairs);
        } else {
            if (many) tail_solve_plain<8>(M, lv + l, pairs);
            else tail_smooth_thin(M, lv + l, pairs);
        }
        if (coarsest) {
            const float mean_e = tail_sum<WARP>(n, red, [&](int i) {
                int x, y, z;
                F.cell(i, &x, &y, &z);
                return M[F.at(x, y, z)];
            }) / (float)n;
            Gr::sync();
            for (int i = Gr::id(); i < n; i += Gr::N) {
                int x, y, z;
                F.cell(i, &x, &y, &z);
                const int k = F.at(x, y, z);
                tail_put(M, F.S, k, F.walls(x, y, z), M[k] - mean_e);
            }
            Gr::sync();
            up = true;
        } else if (!up) {  // restriction
            // Every cell's residual once, then the means of the children in
            // their order.
            const TailLvl C = lv[l + 1];
            const SmLvl& S = F.S;
            for (int j = Gr::id(); j < n; j += Gr::N) {
                int x, y, z;
                F.cell(j, &x, &y, &z);
                const int i = F.at(x, y, z);
                M[F.res + j] = mg_res(F.W, M[i - S.dx] + M[i + S.dx], M[i - S.dy] + M[i + S.dy],
                                      M[i - S.dz] + M[i + S.dz], M[i], M[F.r + j]);
            }
            Gr::sync();
            const int ex = F.cx ? 2 : 1, ey = F.cy ? 2 : 1, ez = F.cz ? 2 : 1;
            const float inv = 1.0f / (float)(ex * ey * ez);
            for (int j = Gr::id(); j < C.S.cells(); j += Gr::N) {
                int X, Y, Z;
                C.cell(j, &X, &Y, &Z);
                const int i = F.res + X * ex + S.nx * (Y * ey + S.ny * (Z * ez));
                float sum = 0.0f;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (((k & 1) == 0 || F.cx) && ((k & 2) == 0 || F.cy) && ((k & 4) == 0 || F.cz))
                        sum += M[i + (k & 1) + ((k >> 1) & 1) * S.nx + (k >> 2) * S.nx * S.ny];
                M[C.r + j] = sum * inv;
            }
            for (int j = Gr::id(); j < C.S.size; j += Gr::N) M[C.e0 + j] = 0.0f;
            Gr::sync();
        }
        l += up ? -1 : 1;
    }
}

// SMALL: a batch of more slots than SMs whose tails' levels have at most a cell
// of a colour a thread (tail_form).  The registers of larger levels' smoothing
// are then not needed and two blocks fit an SM: with one, 256 grids of 5x7x9
// took 1.07 ms a Step and take 0.80 so, 1024 of 8^3 2.15 and 1.79, 256 of 20^3 3.18
// and 2.94; a single 8^3, with nothing to fill the second, 0.333 and 0.345.
// MANY: some slot's coarsest level takes more than kManyPairs pairs.
template <bool SMALL, bool MANY>
__global__ void __launch_bounds__(kCoarseThreads, SMALL ? 2 : 1) kb_vtail(const InstDev* inst, const TailLvl* tables,
                                                                          const Ctl* ctl, Tab tab, int nu, int vc) {
    begin_slot(inst, tab);
    if (vc_idle(ctl, tab.n, vc)) return;
    __shared__ float red[32];
    __shared__ __align__(8) TailLvl lv[kMaxLev];
    for (int item = blockIdx.x, total = tab.prefix[tab.n]; item < total; item += gridDim.x) {
        const int s = find_slot(tab.prefix, tab.n, item);
        if (mg_off(ctl[s], vc)) continue;
        const InstDev& I = inst[s];
        const int t = I.tail, nl = I.nlev, cs = I.coarse_sweeps;
        const TailMem M{I.tail_floats, s};
        AF_PTR(float) te = view(I.lev[t].e, lvl_cells(I.lev[t]), DK_VTAIL, s);
        AF_PTR(const float) tr = view((const float*)I.lev[t].r, lvl_cells(I.lev[t]), DK_VTAIL, s);
        static_assert(sizeof(TailLvl) % 4 == 0, "the table is copied by words");
        for (int k = threadIdx.x; k < (int)sizeof(lv) / 4; k += kCoarseThreads)
            ((unsigned*)lv)[k] = ((const unsigned*)(tables + (size_t)s * kMaxLev))[k];
        __syncthreads();
        const TailLvl T = lv[t];
        const int n = T.S.cells();
        float ve[kCoarseMax / kCoarseThreads], vr[kCoarseMax / kCoarseThreads];
#pragma unroll
        for (int k = 0; k < kCoarseMax / kCoarseThreads; ++k) {
            const int i = (int)threadIdx.x + k * kCoarseThreads;
            if (i < n) ve[k] = te[i], vr[k] = tr[i];
        }
#pragma unroll
        for (int k = 0; k < kCoarseMax / kCoarseThreads; ++k) {
            const int i = (int)threadIdx.x + k * kCoarseThreads;
            if (i < n) {
                int x, y, z;
                T.cell(i, &x, &y, &z);
                tail_put(M, T.S, T.at(x, y, z), T.walls(x, y, z), ve[k]);
                M[T.r + i] = vr[k];
            }
        }
        __syncthreads();
        tail_levels<false, SMALL, MANY>(M, lv, t, nl, cs, red, nu);
        for (int i = threadIdx.x; i < n; i += kCoarseThreads) {
            int x, y, z;
            T.cell(i, &x, &y, &z);
            te[i] = M[T.at(x, y, z)];
        }
        __syncthreads();
    }
}

// --- device-side synthetic initial field ---------------------------------
// The Taylor-Green vortex plus PCG32 noise of af_seed_taylor_green, generated
// in parallel: draw k (two PCG outputs) of the sequential U, V, W; z, y, x
// order comes from jumping the generator ahead 2k steps (F. Brown, "Random
// number generation with arbitrary strides", 1994, the pcg32_advance
// method).  The trigonometric factors use binary32 sinpi/cospi, so the field
// is bit-reproducible on the device but not identical to the host
// generator's libm values.
__device__ __forceinline__ unsigned long long pcg_advance(unsigned long long state, unsigned long long inc,
                                                          unsigned long long delta) {
    unsigned long long cur_mult = 6364136223846793005ull, cur_plus = inc, acc_mult = 1ull, acc_plus = 0ull;
    while (delta > 0) {
        if (delta & 1ull) {
            acc_mult *= cur_mult;
            acc_plus = acc_plus * cur_mult + cur_plus;
        }
        cur_plus = (cur_mult + 1ull) * cur_plus;
        cur_mult *= cur_mult;
        delta >>= 1;
    }
    return acc_mult * state + acc_plus;
}

__device__ __forceinline__ unsigned pcg_output(unsigned long long old) {
    const unsigned xorshifted = (unsigned)(((old >> 18u) ^ old) >> 27u);
    const unsigned rot = (unsigned)(old >> 59u);
    return (xorshifted >> rot) | (xorshifted << ((32u - rot) & 31u));
}

__global__ void k_seed_tg(Geom g, double* u, double* v, double* w, float H, unsigned long long state0,
                          unsigned long long inc, double amp, double noise) {
    const long long cu = (long long)(g.NX + 1) * g.NY * g.NZ, cv = (long long)g.NX * (g.NY + 1) * g.NZ,
                    cw = (long long)g.NX * g.NY * (g.NZ + 1);
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < cu + cv + cw;
         k += (long long)gridDim.x * blockDim.x) {
        const unsigned long long st = pcg_advance(state0, inc, 2ull * (unsigned long long)k);
        const unsigned a = pcg_output(st) >> 5;
        const unsigned b = pcg_output(st * 6364136223846793005ull + inc) >> 6;
        const double uni = ((double)a * 67108864.0 + (double)b) * (1.0 / 9007199254740992.0);
        int comp, ex, ey;
        long long r;
        if (k < cu) { comp = 0; r = k; ex = g.NX + 1; ey = g.NY; }
        else if (k < cu + cv) { comp = 1; r = k - cu; ex = g.NX; ey = g.NY + 1; }
        else { comp = 2; r = k - cu - cv; ex = g.NX; ey = g.NY; }
        const int x = (int)(r % ex), y = (int)((r / ex) % ey), z = (int)(r / ((long long)ex * ey));
        // Staggered face positions: u at (i, j+1/2, k+1/2) H, v at (i+1/2, j, k+1/2) H.
        const float X = ((float)x + (comp == 0 ? 0.0f : 0.5f)) * H;
        const float Y = ((float)y + (comp == 1 ? 0.0f : 0.5f)) * H;
        const float Z = ((float)z + 0.5f) * H;
        float tg = 0.0f;
        if (comp == 0) tg = sinpif(2.0f * X) * cospif(2.0f * Y) * cospif(2.0f * Z);
        else if (comp == 1) tg = -cospif(2.0f * X) * sinpif(2.0f * Y) * cospif(2.0f * Z);
        const double val = amp * (double)tg + noise * (2.0 * uni - 1.0);
        const Dims& d = comp == 0 ? g.u : (comp == 1 ? g.v : g.w);
        AF_PTR(double) f = view(comp == 0 ? u : (comp == 1 ? v : w), d.count, DK_SEED, 0);
        f[(x + g.G) + (long long)(y + g.G) * d.sy + (long long)(z + g.G) * d.sz] = val;
    }
}

inline long long cdivl(long long a, long long b) { return (a + b - 1) / b; }

constexpr int kFwd[3] = {0, 1, 2};  // aeroflux.go:373
constexpr int kRev[3] = {2, 1, 0};  // aeroflux.go:390

// Profile event slots.
constexpr int kEvStart = 0, kEvEnd = 1, kEvSweep = 2 /* 2 per sweep */, kEvProj = 14 /* 2 per projection */;
constexpr int kNumEvents = 18;

// Device memory pool with first-fit placement and coalescing frees.
struct Pool {
    char* base = nullptr;
    size_t size = 0;
    std::map<size_t, size_t> free_;  // offset -> bytes
    bool init(size_t bytes) {
        if (cudaMalloc(&base, bytes) != cudaSuccess) return false;
        size = bytes;
        free_[0] = bytes;
        return true;
    }
    char* alloc(size_t bytes) {
        bytes = (bytes + 255) & ~(size_t)255;
        for (auto it = free_.begin(); it != free_.end(); ++it) {
            if (it->second >= bytes) {
                const size_t off = it->first, rest = it->second - bytes;
                free_.erase(it);
                if (rest) free_[off + bytes] = rest;
                return base + off;
            }
        }
        return nullptr;
    }
    void release(char* p, size_t bytes) {
        bytes = (bytes + 255) & ~(size_t)255;
        size_t off = (size_t)(p - base);
        auto next = free_.lower_bound(off);
        if (next != free_.end() && off + bytes == next->first) {
            bytes += next->second;
            next = free_.erase(next);
        }
        if (next != free_.begin()) {
            auto prev = std::prev(next);
            if (prev->first + prev->second == off) {
                prev->second += bytes;
                return;
            }
        }
        free_[off] = bytes;
    }
};

struct SlotHost {
    bool used = false;
    bool active = false;
    af_config cfg{};
    InstDev d{};
    af_field_desc desc[8]{};
    char* mem = nullptr;   // pool or cudaMalloc block (arena unless external, b, multigrid)
    size_t mem_bytes = 0;
    bool external_arena = false;
};

}  // namespace

struct Batch {
    int cap = 0;
    int sms = 152;
    std::vector<SlotHost> slots;
    Pool pool;
    bool use_pool = false;
    cudaStream_t stream = nullptr;
    cudaStream_t body = nullptr;
    InstDev* d_inst = nullptr;
    TailLvl* d_tails = nullptr;      // kMaxLev per slot: the tail levels' tables
    std::vector<TailLvl> h_tails;
    Status* d_st = nullptr;
    Ctl* d_ctl = nullptr;
    int* d_tab = nullptr;            // S_COUNT prefix arrays of cap+1 ints
    std::vector<int> h_tab;
    Shape shape[S_COUNT];
    int grid_sz[S_COUNT] = {};       // blocks per stage, fixed when the graph is captured
    int graph_levels = 0;            // levels the captured graph runs per-level kernels on
    unsigned graph_big = 0;          // levels whose large-coarsest smoothing the graph carries
    unsigned graph_pair = 0;         // levels with wide fused-pair tiles in the graph
    unsigned graph_pairn = 0;        // levels with narrow fused-pair tiles in the graph
    unsigned graph_march = 0;        // levels with marching pairs in the graph
    unsigned graph_single = 0;       // levels with in-place colour sweeps in the graph
    size_t tail_smem = 0;            // dynamic shared memory of the tail V-cycle
    int tail_form = 0;               // kTailLarge, kTailMany: the tail V-cycle's kernel (kTailKernels)
    int graph_nu = 0;                // smoothing sweeps the captured graph carries
    bool per_level = false;          // multigrid without the tail V-cycle above the coarsest level
    bool pairs = true;               // fused red-black pair smoothing below the tail
    bool cold = false;               // every projection starts from P = 0 (the reference's zeroing)
    cudaGraphExec_t graph = nullptr;
    bool tables_dirty = true;
    // Launches may overlap (launch_maybe_pdl).  Not in a projection captured for
    // one use: the capture of a graph of such launches takes longer than their
    // overlap saves (114x80x36 0.381 / 0.353 ms, 94x114x24 1.05 / 0.96).
    bool overlap = true;
    bool profiling = false;
    cudaEvent_t ev[kNumEvents] = {};
    int64_t launches = 0;
    int nu = 2;
    int vcycles = 4;  // V-cycles per refinement pass at most (measured best of 2, 3, 4, 6, 8)
    double pass_floor = 0.0;  // max|r| reduction one pass can reach (0: not used to cut V-cycles)
    int fixed_passes = 0;
    cudaError_t capture_err = cudaSuccess;
    bool tma_sweep = true;             // staged tile sweep (false: the row kernel)
    CUtensorMap* d_tmaps = nullptr;    // 12 per slot, see InstDev::tmap
    std::vector<CUtensorMap> h_tmaps;
    bool tmaps_dirty = true;
    unsigned march = ~0u;              // levels whose fused pairs march where a slot's level allows it
    int force_pair_var = -1;           // AEROFLUX_PAIR_VARIANT: every fused pair stage's variant (-1: tuned)
    int force_march = -1;              // AEROFLUX_MARCH_SHAPE: every marching pair's shape (-1: tuned)
    bool pair_chosen = false;          // the fused pairs' tile variants are set (tuned or by level size)
    unsigned march_polls = kMarchPolls;  // AEROFLUX_MARCH_POLLS: march_wait's first polls (0: every wait gives up)
    unsigned* d_diag = nullptr;        // nonzero: a kernel gave up a bounded wait; lies behind the statuses
};

namespace {

int max_levels(const Batch* b) {
    int m = 1;
    for (const auto& s : b->slots)
        if (s.used) m = std::max(m, s.d.nlev);
    return m;
}

// Levels some slot smooths and coarsens with per-level kernels.
int slot_levels(const SlotHost& S) { return S.d.tail >= 0 ? S.d.tail : S.d.nlev - 1; }
int kernel_levels(const Batch* b) {
    int m = 0;
    for (const auto& s : b->slots)
        if (s.used) m = std::max(m, slot_levels(s));
    return m;
}

// Levels at which some slot's coarsest grid is too large for the one-block
// solver (smoothed in place instead).
unsigned big_coarse_levels(const Batch* b) {
    unsigned m = 0;
    for (const auto& s : b->slots)
        if (s.used && s.d.tail < 0) m |= 1u << (s.d.nlev - 1);
    return m;
}

// Levels some slot smooths in place (in-place colour sweeps, no second buffer).
unsigned single_levels(const Batch* b) {
    unsigned m = 0;
    for (const auto& s : b->slots) {
        if (!s.used) continue;
        const int lim = slot_levels(s);
        for (int l = 0; l < lim; ++l)
            if (!s.d.lev[l].e2) m |= 1u << l;
    }
    return m;
}

// Whether a slot's fused pairs of level l march.
bool marches(const Batch* b, const SlotHost& S, int l) { return (b->march & (1u << l)) && S.d.lev[l].march[0].w > 0; }

// Levels with marching pairs.
unsigned march_levels(const Batch* b) {
    unsigned m = 0;
    for (const auto& s : b->slots) {
        if (!s.used) continue;
        const int lim = slot_levels(s);
        for (int l = 0; l < lim; ++l)
            if (s.d.lev[l].e2 && marches(b, s, l)) m |= 1u << l;
    }
    return m;
}

// Levels whose fused pairs need the narrow tile column (wide: the others).
unsigned pair_levels(const Batch* b, bool narrow) {
    unsigned m = 0;
    for (const auto& s : b->slots) {
        if (!s.used) continue;
        const int lim = slot_levels(s);
        for (int l = 0; l < lim; ++l) {
            const Lvl& L = s.d.lev[l];
            if (L.e2 && !marches(b, s, l) && (narrow ? L.nxw < L.nx : L.nxw > 0)) m |= 1u << l;
        }
    }
    return m;
}

size_t tail_smem_bytes(const Batch* b) {
    size_t m = 0;
    for (const auto& s : b->slots)
        if (s.used && s.d.tail >= 0) m = std::max(m, (size_t)s.d.tail_floats * sizeof(float));
    return m;
}

// What the tail V-cycle's kernel must hold: a level of more than a cell of a
// colour a thread (the first one is the largest), many pairs at the coarsest.
constexpr int kTailLarge = 1, kTailMany = 2;
void (*const kTailKernels[4])(const InstDev*, const TailLvl*, const Ctl*, Tab, int, int) = {
    kb_vtail<true, false>, kb_vtail<false, false>, kb_vtail<true, true>, kb_vtail<false, true>};
int tail_form(const Batch* b) {
    int f = 0;
    for (const auto& s : b->slots) {
        if (!s.used || s.d.tail < 0) continue;
        if (SmLvl(s.d.lev[s.d.tail]).slots() > kCoarseThreads) f |= kTailLarge;
        if (s.d.coarse_sweeps > kManyPairs) f |= kTailMany;
    }
    return f;
}

// Items of stage `st` for slot `s` under shape sh.
long long stage_items(const Batch* b, const SlotHost& S, int st, const Shape& sh) {
    if (!S.used || !S.active) return 0;
    const InstDev& I = S.d;
    const long long per = (long long)sh.tpb * sh.ept;
    long long n = 0;
    if (st == S_BC) n = bc_count(I.g);
    else if (st == S_SWEEP) n = sweep_box(I.g);
    else if (st == S_GRAD) n = (long long)(I.g.NX + 1) * (I.g.NY + 1) * (I.g.NZ + 1);
    else if (st == S_SHADOW) n = I.shq[3];
    else if (st == S_SWEEPT) return I.sw_tiles;
    else if (st == S_DIV) n = (long long)I.g.p.nx * I.g.p.ny * I.g.p.nz;
    else if (st == S_INT) n = residual_items(I.g, I.res_lg);
    else if (st == S_CORR) n = correct_items(I.g);
    else if (st == S_PBC) n = pbc_count(I.g);
    else if (st == S_COARSE) return I.tail >= 0 ? 1 : 0;
    const int lim = I.tail >= 0 ? I.tail : I.nlev - 1;  // levels smoothed by per-level kernels
    if (st < S_SMOOTH) {
        // n set above
    } else if (st < S_RESTRICT) {
        const int l = st - S_SMOOTH;
        n = (l < lim && !I.lev[l].e2) ? row_box(I.lev[l]) : 0;
    } else if (st >= S_RESTRICT && st < S_PROLONG) {
        const int l = st - S_RESTRICT;
        n = l < lim ? restrict_items(I.lev[l], I.lev[l + 1]) : 0;
    } else if (st >= S_PROLONG && st < S_BIGCOARSE) {
        const int l = st - S_PROLONG;
        n = l < lim ? prolong_box(I.lev[l], I.lev[l + 1]) : 0;
    } else if (st >= S_BIGCOARSE && st < S_PAIR) {
        const int l = st - S_BIGCOARSE;
        n = (l == I.nlev - 1 && I.tail < 0) ? row_box(I.lev[l]) : 0;
    } else if (st >= S_MARCH) {
        const int l = st - S_MARCH;
        if (l >= lim || !I.lev[l].e2 || !marches(b, S, l)) return 0;
        const MarchShape& m = kMarchShapes[sh.var];
        const Lvl::March& M = I.lev[l].march[m.k];
        return (long long)M.fcol.d * M.fty.d * cdivl(I.lev[l].nz, m.zc);
    } else if (st >= S_PAIR) {
        const bool wide = st < S_PAIRN;
        const int l = st - (wide ? S_PAIR : S_PAIRN);
        if (l >= lim || !I.lev[l].e2 || marches(b, S, l)) return 0;
        const Lvl& L = I.lev[l];
        const long long cols = wide ? L.nxw / kPairWideX : (L.nxw < L.nx ? 1 : 0);
        return cols * cdivl(L.ny, kPairVarTY[sh.var]) * cdivl(L.nz, kPairVarTZ[sh.var]);
    }
    return cdivl(n, per);
}

// A stage's prefix of tiles per slot under its present shape.
void fill_tab(Batch* b, int st) {
    int* pre = &b->h_tab[(size_t)st * (b->cap + 1)];
    long long acc = 0;
    for (int s = 0; s < b->cap; ++s) {
        pre[s] = (int)acc;
        acc += stage_items(b, b->slots[s], st, b->shape[st]);
    }
    pre[b->cap] = (int)acc;
}

// One stage's work list alone, when only its shape changed.
cudaError_t upload_stage(Batch* b, int st) {
    const size_t w = (size_t)b->cap + 1;
    fill_tab(b, st);
    return cudaMemcpyAsync(b->d_tab + st * w, &b->h_tab[st * w], w * sizeof(int), cudaMemcpyHostToDevice, b->stream);
}

// Cells a thread of the residual takes: eight where that leaves every slot's
// cells together at least 64 Ki threads, else two.  Measured at one, two, four,
// eight: 48x32x64 10.2, 7.8, 14.7, 19.2 us; 96^3 20.8, 19.3, 19.8, 17.0; 128^3
// 37.2, 34.3, 34.2, 33.2; 256^3 222, 219, -, 184.
int residual_planes_log(const Batch* b) {
    long long cells = 0;
    for (const auto& s : b->slots)
        if (s.used && s.active) cells += (long long)s.d.g.NX * s.d.g.NY * s.d.g.NZ;
    return cells >= (512ll << 10) ? kResMaxLg : 1;
}

cudaError_t upload_tables(Batch* b) {
    const int w = b->cap + 1;
    const int lg = residual_planes_log(b);
    for (auto& s : b->slots) s.d.res_lg = lg;
    b->h_tab.assign((size_t)S_COUNT * w, 0);
    for (int st = 0; st < S_COUNT; ++st) fill_tab(b, st);
    std::vector<InstDev> inst(b->cap);
    for (int s = 0; s < b->cap; ++s) {
        inst[s] = b->slots[s].d;
        inst[s].active = b->slots[s].used && b->slots[s].active ? 1 : 0;
    }
    cudaError_t rc;
    if ((rc = cudaMemcpyAsync(b->d_tab, b->h_tab.data(), b->h_tab.size() * sizeof(int), cudaMemcpyHostToDevice,
                              b->stream)) != cudaSuccess)
        return rc;
    if ((rc = cudaMemcpyAsync(b->d_inst, inst.data(), inst.size() * sizeof(InstDev), cudaMemcpyHostToDevice,
                              b->stream)) != cudaSuccess)
        return rc;
    if (b->tmaps_dirty) {
        if ((rc = cudaMemcpyAsync(b->d_tails, b->h_tails.data(), b->h_tails.size() * sizeof(TailLvl),
                                  cudaMemcpyHostToDevice, b->stream)) != cudaSuccess)
            return rc;
        if ((rc = cudaMemcpyAsync(b->d_tmaps, b->h_tmaps.data(), b->h_tmaps.size() * sizeof(CUtensorMap),
                                  cudaMemcpyHostToDevice, b->stream)) != cudaSuccess)
            return rc;
        b->tmaps_dirty = false;
    }
    b->tables_dirty = false;
    return cudaStreamSynchronize(b->stream);
}

Tab tab(const Batch* b, int st) { return Tab{b->d_tab + (size_t)st * (b->cap + 1), b->cap, b->shape[st].ept}; }
int grid(const Batch* b, int st) { return b->grid_sz[st] > 0 ? b->grid_sz[st] : b->sms * b->shape[st].bpsm; }

// Persistent grid of a stage: up to shape.bpsm blocks per SM, no more blocks
// than tiles at capture time but at least one per SM, so slots assigned
// later still spread over the whole GPU.
void size_grids(Batch* b) {
    const int w = b->cap + 1;
    for (int st = 0; st < S_COUNT; ++st) {
        const int items = b->h_tab[(size_t)st * w + b->cap];
        b->grid_sz[st] = std::max(b->sms, std::min(items, b->sms * b->shape[st].bpsm));
    }
}

#define LAUNCH(b, st, kernel, ...)                                                          \
    do {                                                                                    \
        launch_maybe_pdl(b->overlap, kernel, dim3(grid(b, st)), dim3(b->shape[st].tpb), 0, s, __VA_ARGS__); \
        ++b->launches;                                                                      \
    } while (0)

void rec(Batch* b, int idx, cudaStream_t s) {
    if (b->profiling) cudaEventRecordWithFlags(b->ev[idx], s, cudaEventRecordExternal);
}

void enq_bc(Batch* b, int parity, int gate, cudaStream_t s) { LAUNCH(b, S_BC, kb_bc, b->d_inst, b->d_st, tab(b, S_BC), parity, gate); }

void enq_sweep(Batch* b, int axis, int parity, int phase, cudaStream_t s) {
    LAUNCH(b, S_SHADOW, kb_shadow, b->d_inst, tab(b, S_SHADOW), parity);
    if (b->tma_sweep) {
        const Tab t = tab(b, S_SWEEPT);
        const int g = grid(b, S_SWEEPT);
        const auto k = axis == 0 ? kb_sweep_tma<0> : (axis == 1 ? kb_sweep_tma<1> : kb_sweep_tma<2>);
        launch_maybe_pdl(b->overlap, k, dim3(g), dim3(kSwBlock), kSwSmem, s, b->d_inst, b->d_st, t, parity, phase, b->d_diag);
        ++b->launches;
        return;
    }
    const Tab t = tab(b, S_SWEEP);
    if (axis == 0) LAUNCH(b, S_SWEEP, kb_sweep<0>, b->d_inst, b->d_st, t, parity, phase);
    else if (axis == 1) LAUNCH(b, S_SWEEP, kb_sweep<1>, b->d_inst, b->d_st, t, parity, phase);
    else LAUNCH(b, S_SWEEP, kb_sweep<2>, b->d_inst, b->d_st, t, parity, phase);
}

void enq_smooth(Batch* b, int st, int l, int pairs, int vc, cudaStream_t s) {
    for (int k = 0; k < pairs; ++k) {
        LAUNCH(b, st, kb_smooth, b->d_inst, b->d_ctl, tab(b, st), l, 0, vc);
        LAUNCH(b, st, kb_smooth, b->d_inst, b->d_ctl, tab(b, st), l, 1, vc);
    }
}

// One fused red-black pair of level l with stage st's tile variant (wide
// tiles for S_PAIR + l, the narrow column for S_PAIRN + l).
template <int LANES, int V>
void launch_pair_v(Batch* b, int st, int l, int dir, int vc, cudaStream_t s) {
    launch_maybe_pdl(b->overlap, kb_smooth_pair<LANES, V>, dim3(grid(b, st)), dim3(PairTile<LANES, V>::THREADS), 0, s, b->d_inst, b->d_ctl,
               tab(b, st), l, dir, vc);
    ++b->launches;
}

void launch_pair(Batch* b, int st, int l, int dir, int vc, cudaStream_t s) {
    const bool wide = st < S_PAIRN;
    switch (b->shape[st].var) {
        case 0: wide ? launch_pair_v<32, 0>(b, st, l, dir, vc, s) : launch_pair_v<16, 0>(b, st, l, dir, vc, s); break;
        case 1: wide ? launch_pair_v<32, 1>(b, st, l, dir, vc, s) : launch_pair_v<16, 1>(b, st, l, dir, vc, s); break;
        case 2: wide ? launch_pair_v<32, 2>(b, st, l, dir, vc, s) : launch_pair_v<16, 2>(b, st, l, dir, vc, s); break;
        default: wide ? launch_pair_v<32, 4>(b, st, l, dir, vc, s) : launch_pair_v<16, 4>(b, st, l, dir, vc, s);
    }
}

Shape pair_shape(bool wide, int var) {
    const int threads = kPairVarTY[var] * (wide ? 32 : 16);
    return Shape{threads, 1, (var == 0 || var == 4 ? 2048 : 1536) / threads, var};
}

Shape march_shape(int m) {
    const int t = kMarchT[kMarchShapes[m].k];
    return Shape{t, 1, kMarchBlocks[kMarchShapes[m].k], m};
}

void launch_march(Batch* b, int l, int dir, int vc, cudaStream_t s) {
    const int st = S_MARCH + l, g = grid(b, st);
    const MarchShape m = kMarchShapes[b->shape[st].var];
    const auto k = m.k == 0 ? kb_smooth_march<0> : (m.k == 1 ? kb_smooth_march<1> : kb_smooth_march<2>);
    launch_maybe_pdl(b->overlap, k, dim3(g), dim3(kMarchT[m.k]), 0, s, b->d_inst, b->d_ctl, tab(b, st), l, dir, vc, m.zc, b->march_polls,
               b->d_diag);
    ++b->launches;
}

// Pre- or post-smoothing of level l: fused pairs ping-ponging through e2
// (an even count returns the result to e) for slots that have e2, in-place
// colour sweeps for the others.
void enq_level_smooth(Batch* b, int l, int vc, cudaStream_t s) {
    // A pair reads the previous pair's output across the wide / narrow
    // boundary, so both kinds finish pair k before either starts pair k+1.
    for (int k = 0; k < b->nu; ++k) {
        if (b->graph_pair & (1u << l)) launch_pair(b, S_PAIR + l, l, k & 1, vc, s);
        if (b->graph_pairn & (1u << l)) launch_pair(b, S_PAIRN + l, l, k & 1, vc, s);
        if (b->graph_march & (1u << l)) launch_march(b, l, k & 1, vc, s);
    }
    if (b->graph_single & (1u << l)) enq_smooth(b, S_SMOOTH + l, l, b->nu, vc, s);
}

// V-cycle vc of a refinement pass; slots whose pass runs fewer V-cycles
// skip it.
void enq_vcycle(Batch* b, int vc, cudaStream_t s) {
    const int L = b->graph_levels;
    for (int l = 0; l < L; ++l) {
        enq_level_smooth(b, l, vc, s);
        LAUNCH(b, S_RESTRICT + l, kb_restrict, b->d_inst, b->d_ctl, tab(b, S_RESTRICT + l), l, vc);
    }
    if (b->tail_smem) {
        launch_maybe_pdl(b->overlap, kTailKernels[b->tail_form], dim3(grid(b, S_COARSE)), dim3(kCoarseThreads),
                   b->tail_smem, s, b->d_inst, b->d_tails, b->d_ctl, tab(b, S_COARSE), b->nu, vc);
        ++b->launches;
    }
    for (int l = 0; l < kMaxLev; ++l)
        if (b->graph_big & (1u << l)) enq_smooth(b, S_BIGCOARSE + l, l, 8 * b->nu, vc, s);
    for (int l = L - 1; l >= 0; --l) {
        LAUNCH(b, S_PROLONG + l, kb_prolong, b->d_inst, b->d_ctl, tab(b, S_PROLONG + l), l, vc);
        enq_level_smooth(b, l, vc, s);
    }
}

void enq_pass(Batch* b, cudaStream_t s, cudaGraphConditionalHandle h, int use_cond, int gate) {
    for (int k = 0; k < b->vcycles; ++k) enq_vcycle(b, k, s);
    LAUNCH(b, S_CORR, kb_correct, b->d_inst, b->d_ctl, tab(b, S_CORR));
    LAUNCH(b, S_INT, kb_residual, b->d_inst, b->d_st, b->d_ctl, tab(b, S_INT), gate, 1);
    launch_maybe_pdl(b->overlap, kb_check, dim3(1), dim3(256), 0, s, b->d_inst, b->d_st, b->d_ctl, b->cap, h, use_cond, 1, gate, b->vcycles, b->pass_floor);
    ++b->launches;
}

// project, project.go:12-34, with binary64 refinement; s must be capturing.
void enq_project(Batch* b, int parity, int gate, cudaStream_t s) {
    rec(b, kEvProj + (gate == 3 ? 0 : 2), s);
    enq_bc(b, parity, gate, s);
    LAUNCH(b, S_DIV, kb_div, b->d_inst, b->d_st, tab(b, S_DIV), parity, gate);
    launch_maybe_pdl(b->overlap, kb_init, dim3(1), dim3(256), 0, s, b->d_inst, b->d_ctl, b->cap);
    ++b->launches;
    LAUNCH(b, S_INT, kb_residual, b->d_inst, b->d_st, b->d_ctl, tab(b, S_INT), gate, 0);
    if (b->fixed_passes > 0) {
        launch_maybe_pdl(b->overlap, kb_check, dim3(1), dim3(256), 0, s, b->d_inst, b->d_st, b->d_ctl, b->cap, 0, 0, 0, gate, b->vcycles, b->pass_floor);
        ++b->launches;
        for (int k = 0; k < b->fixed_passes; ++k) enq_pass(b, s, 0, 0, gate);
    } else {
        cudaStreamCaptureStatus cs;
        cudaGraph_t graph = nullptr;
        const cudaGraphNode_t* deps = nullptr;
        size_t ndeps = 0;
        cudaError_t rc = cudaStreamGetCaptureInfo(s, &cs, nullptr, &graph, &deps, nullptr, &ndeps);
        if (rc != cudaSuccess || cs != cudaStreamCaptureStatusActive) {
            b->capture_err = rc != cudaSuccess ? rc : cudaErrorStreamCaptureUnsupported;
            return;
        }
        cudaGraphConditionalHandle h;
        if ((rc = cudaGraphConditionalHandleCreate(&h, graph, 0, cudaGraphCondAssignDefault)) != cudaSuccess) {
            b->capture_err = rc;
            return;
        }
        launch_maybe_pdl(b->overlap, kb_check, dim3(1), dim3(256), 0, s, b->d_inst, b->d_st, b->d_ctl, b->cap, h, 1, 0, gate, b->vcycles,
                   b->pass_floor);
        ++b->launches;
        // Every pass is an iteration of the node, the first two too, which nearly
        // every projection needs: as launches before it they save 1-2.5 % of a
        // Step on small grids and under 1 % from 128^3 on, but a projection that
        // needs none (a fluid at rest, a loose tolerance) walks all their empty
        // launches: 0.32 instead of 0.13 ms a Step at 48x32x64, 0.85 instead of
        // 0.55 at 128^3, and a graph of three passes to capture for one
        // af_project (0.62 instead of 0.25 ms).
        // A launch that the device refused has ended the capture: the graph and
        // its nodes are then no longer ours to use.
        rc = cudaStreamGetCaptureInfo(s, &cs, nullptr, &graph, &deps, nullptr, &ndeps);
        if (rc != cudaSuccess || cs != cudaStreamCaptureStatusActive) {
            b->capture_err = rc != cudaSuccess ? rc : cudaErrorStreamCaptureInvalidated;
            return;
        }
        cudaGraphNodeParams params{cudaGraphNodeTypeConditional};  // the other members value-initialised
        params.conditional.handle = h;
        params.conditional.type = cudaGraphCondTypeWhile;
        params.conditional.size = 1;
        cudaGraphNode_t node;
        if ((rc = cudaGraphAddNode(&node, graph, deps, nullptr, ndeps, &params)) != cudaSuccess) {
            b->capture_err = rc;
            return;
        }
        cudaGraph_t body = params.conditional.phGraph_out[0];
        if ((rc = cudaStreamBeginCaptureToGraph(b->body, body, nullptr, nullptr, 0,
                                                cudaStreamCaptureModeThreadLocal)) != cudaSuccess) {
            b->capture_err = rc;
            return;
        }
        enq_pass(b, b->body, h, 1, gate);
        cudaGraph_t body_out = nullptr;
        if ((rc = cudaStreamEndCapture(b->body, &body_out)) != cudaSuccess) {
            b->capture_err = rc;
            return;
        }
        if ((rc = cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1, cudaStreamSetCaptureDependencies)) !=
            cudaSuccess) {
            b->capture_err = rc;
            return;
        }
    }
    LAUNCH(b, S_PBC, kb_pbc, b->d_inst, b->d_st, tab(b, S_PBC), gate);
    LAUNCH(b, S_GRAD, kb_grad, b->d_inst, b->d_st, tab(b, S_GRAD), parity, gate, 0);
    enq_bc(b, parity, gate, s);
    rec(b, kEvProj + (gate == 3 ? 1 : 3), s);
}

// Step, aeroflux.go:348-409, for every active slot.
void enq_step(Batch* b, cudaStream_t s) {
    rec(b, kEvStart, s);
    for (int k = 0; k < 6; ++k) {
        const int axis = k < 3 ? kFwd[k] : kRev[k - 3];
        enq_bc(b, k & 1, k, s);
        rec(b, kEvSweep + 2 * k, s);
        enq_sweep(b, axis, k & 1, k, s);
        rec(b, kEvSweep + 2 * k + 1, s);
        if (k == 2) enq_project(b, 1, 3, s);
    }
    enq_project(b, 0, 6, s);
    launch_maybe_pdl(b->overlap, kb_tick, dim3(1), dim3(256), 0, s, b->d_inst, b->d_st, b->cap);
    ++b->launches;
    rec(b, kEvEnd, s);
}

template <class F>
cudaError_t capture(Batch* b, F body, cudaGraphExec_t* out) {
    cudaGraph_t graph = nullptr;
    b->capture_err = cudaSuccess;  // an ended capture has left its own
    cudaError_t rc = cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal);
    if (rc != cudaSuccess) return rc;
    body();
    rc = cudaStreamEndCapture(b->stream, &graph);
    if (rc != cudaSuccess) return rc;
    if (b->capture_err != cudaSuccess) {
        rc = b->capture_err;
        b->capture_err = cudaSuccess;
        cudaGraphDestroy(graph);
        return rc;
    }
    rc = cudaGraphInstantiate(out, graph, 0);
    cudaGraphDestroy(graph);
    return rc;
}

// Untuned tile variants and march shapes of the fused pairs, by the largest
// level each pair stage serves: the largest tiles from 4 Mi cells, the middle
// ones from 256 Ki, the smallest below.  Set once, before the first capture
// (the captured kernels and the work lists must agree); the autotuner may
// replace them.
void default_pair_variants(Batch* b) {
    if (b->pair_chosen || b->graph) return;
    if (b->force_pair_var >= 0) b->march = b->force_pair_var == 3 ? ~0u : 0u;
    for (int l = 0; l < kMaxLev; ++l) {
        long long most = 0;
        for (const auto& S : b->slots)
            if (S.used && l < S.d.nlev) most = std::max(most, lvl_cells(S.d.lev[l]));
        int var = most >= (4ll << 20) ? 0 : (most >= (256ll << 10) ? 1 : 2);
        b->shape[S_MARCH + l] = march_shape(b->force_march >= 0 ? b->force_march
                                                                : (most >= (4ll << 20) ? 7 : (most >= (256ll << 10) ? 1 : 0)));
        if (b->force_pair_var >= 0 && b->force_pair_var != 3) var = b->force_pair_var;
        b->shape[S_PAIR + l] = pair_shape(true, var);
        b->shape[S_PAIRN + l] = pair_shape(false, var);
    }
    b->pair_chosen = true;
    b->tables_dirty = true;
}

cudaError_t prepare(Batch* b) {
    cudaError_t rc;
    default_pair_variants(b);
    if (b->tables_dirty && (rc = upload_tables(b)) != cudaSuccess) return rc;
    const int L = kernel_levels(b);
    const unsigned big = big_coarse_levels(b), pair = pair_levels(b, false), pairn = pair_levels(b, true),
                   single = single_levels(b), march = march_levels(b);
    const size_t tsm = tail_smem_bytes(b);
    const int form = tail_form(b);
    if (b->graph && (L > b->graph_levels || (big & ~b->graph_big) || (pair & ~b->graph_pair) ||
                     (pairn & ~b->graph_pairn) || (march & ~b->graph_march) || (single & ~b->graph_single) || tsm > b->tail_smem || (form & ~b->tail_form) ||
                     b->graph_nu != b->nu)) {
        cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    }
    if (!b->graph) {
        b->graph_levels = std::max(L, b->graph_levels);
        b->graph_big |= big;
        b->graph_pair |= pair;
        b->graph_pairn |= pairn;
        b->graph_march |= march;
        b->graph_single |= single;
        b->tail_smem = std::max(b->tail_smem, tsm);
        b->tail_form |= form;
        b->graph_nu = b->nu;
        b->launches = 0;
        size_grids(b);
        if ((rc = capture(b, [&] { enq_step(b, b->stream); }, &b->graph)) != cudaSuccess) {
            b->graph = nullptr;
            return rc;
        }
    }
    return cudaSuccess;
}

// Clears every slot's status (the step counter restarts at 0).  stop_at,
// when given, holds per slot the Steps it performs in the coming call: a slot
// with 0 < stop_at[s] < nsteps is gated from step stop_at[s] on -- its fault
// gate marks the end of that step's last phase, with no fault key -- so every
// later kernel skips it and its state stays that of its last Step.
cudaError_t reset_status(Batch* b, const std::vector<int64_t>* stop_at = nullptr, int64_t nsteps = 0) {
    std::vector<Status> h(b->cap, Status{kNoFault, 0u, kNoKey});
    if (stop_at)
        for (int s = 0; s < b->cap && s < (int)stop_at->size(); ++s)
            if ((*stop_at)[s] > 0 && (*stop_at)[s] < nsteps) h[s].fault_gate = 8u * (unsigned)(*stop_at)[s] - 1u;
    return cudaMemcpyAsync(b->d_st, h.data(), h.size() * sizeof(Status), cudaMemcpyHostToDevice, b->stream);
}

// A recorded gate without a fault key is a planned stop, not a fault.
bool status_faulted(const Status& st) { return st.fault_gate != kNoFault && st.fault_key != kNoKey; }

}  // namespace

std::string fault_message_for(const Geom& g, unsigned gate, unsigned long long key);

namespace {

// cuTensorMapEncodeTiled from the driver, resolved once through the runtime
// (the library links no driver stub); NULL when the driver lacks it.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

// The 12 tensor maps of a slot over its three binary32 shadows: per
// component, the staged boxes of a sweep along x, y and z and the
// axis-velocity box.  Out-of-range box elements load as zeros (never read).
bool encode_slot_maps(const InstDev& I, CUtensorMap* maps) {
    auto enc = tensor_map_encoder();
    if (!enc) return false;
    for (int k = 0; k < 3; ++k) {
        const Dims& d = k == 0 ? I.g.u : (k == 1 ? I.g.v : I.g.w);
        const cuuint64_t dims[3] = {(cuuint64_t)d.nx, (cuuint64_t)d.ny, (cuuint64_t)d.nz};
        const cuuint64_t strides[2] = {(cuuint64_t)I.shp[k] * 4u, (cuuint64_t)I.shp[k] * d.ny * 4u};
        const cuuint32_t estr[3] = {1, 1, 1};
        for (int role = 0; role < 4; ++role) {
            const cuuint32_t box[3] = {(cuuint32_t)sw_bx(role), (cuuint32_t)sw_by(role), (cuuint32_t)sw_bz(role)};
            if (enc(&maps[k * 4 + role], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, I.sh[k], dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return false;
        }
    }
    return true;
}

// The tiles of the marching pair on every level with e2 whose rows and arrays
// are 16-byte aligned.
void plan_march(InstDev& I) {
    for (int l = 0; l < I.nlev; ++l) {
        Lvl& L = I.lev[l];
        auto aligned = [](const void* q) { return ((uintptr_t)q & 15u) == 0; };
        const bool ok = L.e2 && L.nx % 4 == 0 && aligned(L.e) && aligned(L.e2) && aligned(L.r);
        const int quads = L.nx / 4;
        for (int k = 0; k < 3; ++k) {
            Lvl::March& M = L.march[k];
            M = Lvl::March{};
            if (!ok) continue;
            const int cols = (quads + kMarchQ[k] - 1) / kMarchQ[k];
            M.w = (quads + cols - 1) / cols;
            M.q = cols > 1 ? M.w + 2 : M.w;
            const int most = kMarchT[k] / M.q - 2, ty = (L.ny + most - 1) / most;  // most >= 12
            M.rows = (L.ny + ty - 1) / ty;
            M.fq = FastDiv((unsigned)M.q);
            M.fcol = FastDiv((unsigned)((quads + M.w - 1) / M.w));
            M.fty = FastDiv((unsigned)((L.ny + M.rows - 1) / M.rows));
        }
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host API
// ---------------------------------------------------------------------------
Batch* batch_create(int capacity, size_t pool_bytes, std::string* err) {
    Batch* b = new Batch();
    b->cap = capacity;
    b->slots.resize(capacity);
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev);
    if (const char* fp = getenv("AEROFLUX_FIXED_REFINEMENT_PASSES")) b->fixed_passes = std::max(0, atoi(fp));
    // Per-level multigrid kernels only (no tail V-cycle above the coarsest
    // level), and fused red-black pairs on or off: the same bits either way.
    if (const char* pl = getenv("AEROFLUX_MG_PER_LEVEL")) b->per_level = atoi(pl) != 0;
    if (const char* fp = getenv("AEROFLUX_MG_PAIRS")) b->pairs = atoi(fp) != 0;
    // The refinement solves to a tolerance, so it may start from the last
    // projection's pressure instead of zero (project.go:81-83 zeroes it for
    // the fixed sweep count of the red-black solver).
    if (const char* cs = getenv("AEROFLUX_COLD_START")) b->cold = atoi(cs) != 0;
    if (const char* vc = getenv("AEROFLUX_MG_VCYCLES")) b->vcycles = std::min(8, std::max(1, atoi(vc)));
    if (const char* pf = getenv("AEROFLUX_MG_PASS_FLOOR")) b->pass_floor = atoi(pf) < 0 ? ldexp(1.0, atoi(pf)) : 0.0;
    // The row sweep (gathers through L1) instead of the staged tile sweep: the same bits.
    if (const char* sr = getenv("AEROFLUX_SWEEP_ROWS")) b->tma_sweep = atoi(sr) == 0;
    if (b->tma_sweep && !tensor_map_encoder()) b->tma_sweep = false;
    b->shape[S_SWEEPT] = Shape{kSwBlock, 1, 4};  // shared memory holds four blocks' buffers per SM
    cudaFuncSetAttribute(kb_sweep_tma<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSwSmem);
    cudaFuncSetAttribute(kb_sweep_tma<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSwSmem);
    cudaFuncSetAttribute(kb_sweep_tma<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSwSmem);
    for (const auto k : kTailKernels) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem);
    // No more slots than SMs: a second block an SM would have no tail to take.
    b->tail_form = capacity <= b->sms ? kTailLarge : 0;
    // Shapes: the tiny per-slot control and coarse stages keep their own.
    b->shape[S_COARSE] = Shape{kCoarseThreads, 1, 2};
    for (int l = 0; l < kMaxLev; ++l) {
        b->shape[S_PAIR + l] = pair_shape(true, 0);
        b->shape[S_PAIRN + l] = pair_shape(false, 0);
        b->shape[S_MARCH + l] = march_shape(0);
    }
    cudaError_t rc;
    if ((rc = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking)) != cudaSuccess ||
        (rc = cudaStreamCreateWithFlags(&b->body, cudaStreamNonBlocking)) != cudaSuccess ||
        (rc = cudaMalloc(&b->d_inst, sizeof(InstDev) * capacity)) != cudaSuccess ||
        (rc = cudaMalloc(&b->d_tails, sizeof(TailLvl) * kMaxLev * (size_t)capacity)) != cudaSuccess ||
        (rc = cudaMalloc(&b->d_st, sizeof(Status) * (capacity + 1))) != cudaSuccess ||
        (rc = cudaMalloc(&b->d_ctl, sizeof(Ctl) * (capacity + 1))) != cudaSuccess ||
        (rc = cudaMalloc(&b->d_tab, sizeof(int) * (size_t)S_COUNT * (capacity + 1))) != cudaSuccess ||
        (rc = cudaMalloc(&b->d_tmaps, sizeof(CUtensorMap) * 12 * (size_t)capacity)) != cudaSuccess) {
        *err = std::string("aeroflux: batch tables: ") + cudaGetErrorString(rc);
        batch_destroy(b);
        return nullptr;
    }
    b->d_diag = (unsigned*)(b->d_st + capacity);
    cudaMemsetAsync(b->d_ctl, 0, sizeof(Ctl) * (capacity + 1), b->stream);
    cudaMemsetAsync(b->d_diag, 0, sizeof(unsigned), b->stream);
    b->h_tmaps.assign(12 * (size_t)capacity, CUtensorMap{});
    b->h_tails.assign(kMaxLev * (size_t)capacity, TailLvl{});
    // With variant 3, which is not tuned: an index into kMarchShapes, so that
    // small grids run the shapes of large ones.
    if (const char* ms = getenv("AEROFLUX_MARCH_SHAPE"))
        b->force_march = std::min(kMarchShapeCount - 1, std::max(0, atoi(ms)));
    // 0: every wait of the marching pair gives up (how that is reported).
    if (const char* mp = getenv("AEROFLUX_MARCH_POLLS")) b->march_polls = (unsigned)std::min(4096, std::max(0, atoi(mp)));
    // The fused pairs' tile variant for every level (0-2 and 4; 3: marching
    // where a slot's level allows it), instead of the tuned or size-based choice.
    if (const char* pv = getenv("AEROFLUX_PAIR_VARIANT")) b->force_pair_var = std::min(4, std::max(0, atoi(pv)));
    if (pool_bytes) {
        if (!b->pool.init(pool_bytes)) {
            *err = "aeroflux: batch device pool of " + std::to_string(pool_bytes) + " bytes: out of memory";
            batch_destroy(b);
            return nullptr;
        }
        b->use_pool = true;
    }
    if (reset_status(b) != cudaSuccess || upload_tables(b) != cudaSuccess) {
        *err = "aeroflux: batch setup failed";
        batch_destroy(b);
        return nullptr;
    }
    return b;
}

void batch_destroy(Batch* b) {
    if (!b) return;
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->graph) cudaGraphExecDestroy(b->graph);
    for (auto& ev : b->ev)
        if (ev) cudaEventDestroy(ev);
    for (auto& s : b->slots)
        if (s.used && !b->use_pool) cudaFree(s.mem);
    if (b->use_pool) cudaFree(b->pool.base);
    cudaFree(b->d_inst);
    cudaFree(b->d_tails);
    cudaFree(b->d_st);
    cudaFree(b->d_ctl);
    cudaFree(b->d_tab);
    cudaFree(b->d_tmaps);
    if (b->body) cudaStreamDestroy(b->body);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

namespace {

// x extent covered by wide pair tiles: every whole 64 plus a last partial
// one of more than 32 cells; 1..32 remaining cells go to a narrow tile.
int pair_wide_x(int nx) {
    const int w = nx / kPairWideX * kPairWideX;
    return nx - w > kPairWideX / 2 ? w + kPairWideX : w;
}

// Multigrid hierarchy of a grid: coarsen every axis whose extent is even and
// >= 4 until the grid has <= kCoarsestCells cells or no axis halves.  Going
// down to 8 cells instead of 64 measured 0.2-2 % faster (256^3, 512^3, the
// 256-grid batch): the coarsest red-black solve (2 nmax^2 pairs, at least 8)
// is shorter on the smaller grid.
constexpr long long kCoarsestCells = 8;
int plan_levels(int nx, int ny, int nz, Lvl* lev, int* coarse_sweeps) {
    int n = 0;
    float wx = 1.0f, wy = 1.0f, wz = 1.0f;
    while (true) {
        Lvl& L = lev[n++];
        L = Lvl{nx, ny, nz, wx, wy, wz, 0, 0, 0, nullptr, nullptr,
                FastDiv((unsigned)nx), FastDiv((unsigned)ny), FastDiv((unsigned)((nx + 1) / 2)), nullptr,
                FastDiv((unsigned)std::max(1, pair_wide_x(nx) / kPairWideX)),
                {FastDiv((unsigned)((ny + kPairVarTY[0] - 1) / kPairVarTY[0])),
                 FastDiv((unsigned)((ny + kPairVarTY[1] - 1) / kPairVarTY[1])),
                 FastDiv((unsigned)((ny + kPairVarTY[2] - 1) / kPairVarTY[2]))},
                pair_wide_x(nx)};
        // An axis of extent 1 adds nothing to L e (its Neumann neighbours are
        // the cell itself, so its second difference is exactly 0); with its
        // weight kept, the relaxation would count the cell's old value as
        // two neighbours and damp every update on levels whose other axes
        // coarsened (weights 1/4, 1/16, ...).  Its weight is 0 unless every
        // axis has extent 1.
        if (nx > 1 || ny > 1 || nz > 1) {
            if (nx == 1) L.wx = 0.0f;
            if (ny == 1) L.wy = 0.0f;
            if (nz == 1) L.wz = 0.0f;
        }
        const long long c = (long long)nx * ny * nz;
        const int cx = nx % 2 == 0 && nx >= 4, cy = ny % 2 == 0 && ny >= 4, cz = nz % 2 == 0 && nz >= 4;
        if (c <= kCoarsestCells || !(cx || cy || cz) || n == kMaxLev) break;
        L.cx = cx;
        L.cy = cy;
        L.cz = cz;
        if (cx) { nx /= 2; wx *= 0.25f; }
        if (cy) { ny /= 2; wy *= 0.25f; }
        if (cz) { nz /= 2; wz *= 0.25f; }
    }
    const Lvl& last = lev[n - 1];
    const int nmax = std::max(last.nx, std::max(last.ny, last.nz));
    *coarse_sweeps = std::min(1000, std::max(8, 2 * nmax * nmax));
    return n;
}

// First level of the one-block tail V-cycle (every level from it down has at
// most kCoarseMax cells), or -1 when the coarsest level is larger.
int plan_tail(const Lvl* lev, int n, int* floats, bool coarsest_only = false) {
    *floats = 0;
    if (lvl_cells(lev[n - 1]) > kCoarseMax) return -1;
    int t = n - 1;
    while (!coarsest_only && t > 0 && lvl_cells(lev[t - 1]) <= kCoarseMax) --t;
    for (int l = t; l < n; ++l) *floats += SmLvl(lev[l]).size + SmLvl(lev[l]).cells();
    if (t + 1 < n) *floats += SmLvl(lev[t]).cells();  // the residuals of a restriction
    return t;
}

// The tail levels' table: places from 0 on, the residual scratch last.
void plan_tail_table(const InstDev& I, TailLvl* lv) {
    if (I.tail < 0) return;
    int p = 0;
    for (int l = I.tail; l < I.nlev; ++l) {
        const Lvl& L = I.lev[l];
        TailLvl& t = lv[l];
        t.S = SmLvl(L);
        t.W = MgW{L.wx, L.wy, L.wz};
        t.inv = 1.0f / (2.0f * (L.wx + L.wy + L.wz));
        t.e0 = p, t.e = p + t.S.o, t.r = p + t.S.size;
        t.cx = L.cx, t.cy = L.cy, t.cz = L.cz;
        t.fnx = L.fnx, t.fny = L.fny, t.fhx = L.fhx;
        p += t.S.size + t.S.cells();
    }
    for (int l = I.tail; l < I.nlev; ++l) lv[l].res = p;
}

af_field_desc fdesc(int64_t* off, int64_t nx, int64_t ny, int64_t nz) {
    af_field_desc f{*off, nx, ny, nz, nx, nx * ny, nx * ny * nz};
    int64_t sz = f.count * 8;
    if (int64_t r = sz % 128) sz += 128 - r;
    *off += sz;
    return f;
}

Dims dims_of(const af_field_desc& d) {
    return Dims{(int)d.nx, (int)d.ny, (int)d.nz, d.sy, d.sz, d.count};
}

}  // namespace

bool batch_config_fits(const af_config& c, std::string* err) {
    const int64_t g = c.ghost, cx = c.nx + 2 * g, cy = c.ny + 2 * g, cz = c.nz + 2 * g;
    // The kernels decode 32-bit element numbers (FastDiv) and keep the nine
    // velocity-BC write sets' prefix in int (InstDev::bc_off).
    Geom G{};
    G.NX = (int)std::min<int64_t>(c.nx, INT32_MAX);
    G.NY = (int)std::min<int64_t>(c.ny, INT32_MAX);
    G.NZ = (int)std::min<int64_t>(c.nz, INT32_MAX);
    const bool dims_ok = c.nx < (1 << 30) && c.ny < (1 << 30) && c.nz < (1 << 30) && g < (1 << 20);
    const double big = 2147483648.0;  // 2^31, compared in double so no product overflows
    const bool fields_ok = (double)(cx + 1) * cy * cz < big && (double)cx * (cy + 1) * cz < big &&
                           (double)cx * cy * (cz + 1) < big;
    if (!dims_ok || !fields_ok || (double)face_box(G) >= 2.0 * big || (double)bc_count(G) >= big) {
        if (err)
            *err = "aeroflux: grid too large for one batch slot (2^31 elements per field and per velocity-BC "
                   "write set)";
        return false;
    }
    return true;
}

size_t batch_slot_bytes(const af_config& c) {
    int64_t off = 0;
    const int64_t g = c.ghost, cx = c.nx + 2 * g, cy = c.ny + 2 * g, cz = c.nz + 2 * g;
    fdesc(&off, cx, cy, cz);
    fdesc(&off, cx + 1, cy, cz);
    fdesc(&off, cx, cy + 1, cz);
    fdesc(&off, cx, cy, cz + 1);
    fdesc(&off, cx, cy, cz);
    fdesc(&off, cx + 1, cy, cz);
    fdesc(&off, cx, cy + 1, cz);
    fdesc(&off, cx, cy, cz + 1);
    const size_t arena = ((size_t)off + 255) & ~(size_t)255;
    const size_t bb = ((size_t)(cx * cy * cz) * 8 + 255) & ~(size_t)255;
    auto al = [](int64_t n) { return ((size_t)n * 4 + 255) & ~(size_t)255; };
    auto pitch = [](int64_t nx) { return (nx + 3) / 4 * 4; };
    const size_t shb = al(pitch(cx + 1) * cy * cz) + al(pitch(cx) * (cy + 1) * cz) + al(pitch(cx) * cy * (cz + 1));
    Lvl lev[kMaxLev];
    int cs = 0, tf = 0;
    const int nl = plan_levels((int)c.nx, (int)c.ny, (int)c.nz, lev, &cs);
    const int tail = plan_tail(lev, nl, &tf);
    const int lim = tail >= 0 ? tail : nl - 1;
    size_t mg = 0;
    for (int l = 0; l < nl; ++l) mg += ((l < lim && c.inner_sweeps % 2 == 0) ? 3 : 2) * (size_t)lvl_cells(lev[l]) * sizeof(float);
    return arena + bb + shb + ((mg + 255) & ~(size_t)255);
}

int batch_assign(Batch* b, const af_config& c, char* arena, std::string* err) {
    int s = -1;
    for (int i = 0; i < b->cap; ++i)
        if (!b->slots[i].used) {
            s = i;
            break;
        }
    if (s < 0) {
        *err = "aeroflux: batch is full";
        return -1;
    }
    SlotHost& S = b->slots[s];
    S = SlotHost();
    S.cfg = c;
    InstDev& I = S.d;
    // Layout, grid.go:101-134.
    int64_t off = 0;
    const int64_t g = c.ghost, cx = c.nx + 2 * g, cy = c.ny + 2 * g, cz = c.nz + 2 * g;
    S.desc[0] = fdesc(&off, cx, cy, cz);
    S.desc[1] = fdesc(&off, cx + 1, cy, cz);
    S.desc[2] = fdesc(&off, cx, cy + 1, cz);
    S.desc[3] = fdesc(&off, cx, cy, cz + 1);
    S.desc[4] = fdesc(&off, cx, cy, cz);
    S.desc[5] = fdesc(&off, cx + 1, cy, cz);
    S.desc[6] = fdesc(&off, cx, cy + 1, cz);
    S.desc[7] = fdesc(&off, cx, cy, cz + 1);
    I.g.NX = (int)c.nx;
    I.g.NY = (int)c.ny;
    I.g.NZ = (int)c.nz;
    I.g.G = (int)c.ghost;
    I.g.p = dims_of(S.desc[0]);
    I.g.u = dims_of(S.desc[1]);
    I.g.v = dims_of(S.desc[2]);
    I.g.w = dims_of(S.desc[3]);
    if (!batch_config_fits(c, err)) {
        S = SlotHost();
        return -1;
    }
    I.fpx = FastDiv((unsigned)I.g.p.nx);
    I.fpy = FastDiv((unsigned)I.g.p.ny);
    I.ffx = FastDiv((unsigned)(I.g.NX + 1));
    I.ffy = FastDiv((unsigned)(I.g.NY + 1));
    I.ffz = FastDiv((unsigned)(I.g.NZ + 1));
    I.fnx = FastDiv((unsigned)I.g.NX);
    I.fny = FastDiv((unsigned)I.g.NY);
    {
        // bc_set_count of each (component, set), component-major: extents
        // (normal, first tangential, second tangential) per component.
        const long long N[3][3] = {{I.g.NX, I.g.NY, I.g.NZ}, {I.g.NY, I.g.NX, I.g.NZ}, {I.g.NZ, I.g.NX, I.g.NY}};
        long long acc = 0;
        for (int c = 0; c < 3; ++c)
            for (int set = 0; set < 3; ++set) {
                I.bc_off[3 * c + set] = (int)acc;
                const long long Nn = N[c][0], N1 = N[c][1], N2 = N[c][2];
                // Components 1 and 2 (V, W) have their first tangential
                // axis along x, the stride-1 one (bc_t1_first).
                unsigned d1, d2;
                bc_divisors((int)Nn, (int)N1, (int)N2, c != 0 && set == 2, set, &d1, &d2);
                I.bcd[3 * c + set][0] = FastDiv(d1);
                I.bcd[3 * c + set][1] = FastDiv(d2);
                acc += set == 0 ? 2 * N1 * N2 : (set == 1 ? 2 * (Nn + 1) * N2 : 2 * (Nn + 1) * (N1 + 2));
            }
        I.bc_off[9] = (int)acc;
    }
    I.nlev = plan_levels(I.g.NX, I.g.NY, I.g.NZ, I.lev, &I.coarse_sweeps);
    I.tail = plan_tail(I.lev, I.nlev, &I.tail_floats, b->per_level);
    const int lim = I.tail >= 0 ? I.tail : I.nlev - 1;
    // Fused red-black pairs need an even sweep count (the ping-pong returns
    // the result to e) and run on every level below the tail.  The batch's
    // sweep count is the first slot's; a slot joining a batch that sweeps an
    // odd number of times smooths in place.
    bool others = false;
    for (int i = 0; i < b->cap; ++i)
        if (i != s && b->slots[i].used) others = true;
    const int batch_nu = others ? b->nu : (int)c.inner_sweeps;
    const bool fused = c.inner_sweeps % 2 == 0 && batch_nu % 2 == 0 && b->pairs;
    auto pair_level = [&](int l) { return fused && l < lim; };
    const size_t arena_bytes = ((size_t)off + 255) & ~(size_t)255;
    const size_t b_bytes = ((size_t)S.desc[0].count * 8 + 255) & ~(size_t)255;
    size_t sh_bytes[3];
    for (int k = 0; k < 3; ++k) {
        const af_field_desc& d = S.desc[1 + k];
        I.shp[k] = (int)((d.nx + 3) / 4 * 4);
        sh_bytes[k] = ((size_t)I.shp[k] * d.ny * d.nz * 4 + 255) & ~(size_t)255;
    }
    {
        // Shadow conversion: (row, quad) items per component.
        int acc = 0;
        for (int k = 0; k < 3; ++k) {
            const af_field_desc& d = S.desc[1 + k];
            I.shq[k] = acc;
            I.fsq[k] = FastDiv((unsigned)(I.shp[k] / 4));
            acc += (int)(d.ny * d.nz * (I.shp[k] / 4));
        }
        I.shq[3] = acc;
        // Staged sweep tiles: x, y and z tiles from G covering the largest
        // component extent along each axis (a U row's extra face belongs to
        // its last x tile), three components per spatial tile.
        const int ntx = (I.g.NX + kSwTX - 1) / kSwTX;
        const int nty = (I.g.NY + 1 + kSwTY - 1) / kSwTY;
        const int ntz = (I.g.NZ + 1 + kSwTZ - 1) / kSwTZ;
        I.swx = FastDiv((unsigned)ntx);
        I.swy = FastDiv((unsigned)nty);
        I.sw_tiles = 3 * ntx * nty * ntz;
    }
    size_t mg = 0;
    for (int l = 0; l < I.nlev; ++l) mg += (pair_level(l) ? 3 : 2) * (size_t)lvl_cells(I.lev[l]) * sizeof(float);
    mg = (mg + 255) & ~(size_t)255;
    S.external_arena = arena != nullptr;
    S.mem_bytes = (arena ? 0 : arena_bytes) + b_bytes + sh_bytes[0] + sh_bytes[1] + sh_bytes[2] + mg;
    if (b->use_pool) {
        S.mem = b->pool.alloc(S.mem_bytes);
        if (!S.mem) {
            *err = "aeroflux: batch device pool exhausted";
            S = SlotHost();
            return -1;
        }
    } else if (cudaMalloc(&S.mem, S.mem_bytes) != cudaSuccess) {
        cudaGetLastError();
        *err = "aeroflux: batch slot allocation failed";
        S = SlotHost();
        return -1;
    }
    char* p = S.mem;
    char* base = arena;
    if (!arena) {
        base = p;
        p += arena_bytes;
        cudaMemsetAsync(base, 0, arena_bytes, b->stream);  // MAC.Zero, grid.go:158-163
    }
    for (int f = 0; f < 8; ++f) I.slot[f] = (double*)(base + S.desc[f].off);
    I.b = (double*)p;
    p += b_bytes;
    for (int k = 0; k < 3; ++k) {
        I.sh[k] = (float*)p;
        p += sh_bytes[k];
    }
    I.tmap = b->d_tmaps + 12 * (size_t)s;
    b->tmaps_dirty = true;
    if (b->tma_sweep && !encode_slot_maps(I, &b->h_tmaps[12 * (size_t)s])) {
        // No tensor maps for this slot: the whole batch sweeps with the row kernel.
        b->tma_sweep = false;
        if (b->graph) {
            cudaGraphExecDestroy(b->graph);
            b->graph = nullptr;
        }
    }
    float* fp = (float*)p;
    for (int l = 0; l < I.nlev; ++l) {
        const long long n = lvl_cells(I.lev[l]);
        I.lev[l].e = fp;
        I.lev[l].r = fp + n;
        fp += 2 * n;
        I.lev[l].e2 = nullptr;
        if (pair_level(l)) {
            I.lev[l].e2 = fp;
            fp += n;
        }
    }
    cudaMemsetAsync(p, 0, mg, b->stream);
    for (int l = 0; l + 1 < I.nlev; ++l) {
        Lvl &F = I.lev[l], &C = I.lev[l + 1];
        auto aligned = [](const float* q) { return ((uintptr_t)q & 15) == 0; };
        F.v4 = restrict_pairs(F) && F.nx % 4 == 0 && aligned(F.e) && aligned(F.r) && aligned(C.e) && aligned(C.r);
    }
    plan_march(I);
    plan_tail_table(I, &b->h_tails[kMaxLev * (size_t)s]);
    const double half = c.dt * 0.5;  // aeroflux.go:353
    const double invH = 1.0 / c.h;
    I.dt_invh = (float)(half * invH);
    I.lam = (float)(c.viscosity * half * invH * invH);  // stencil.go:73
    I.div_scale = exact::mul_const(c.density / (c.dt * c.h));   // project.go:49
    I.h2 = exact::mul_const(c.h * c.h);                         // project.go:107
    I.grad_scale = exact::mul_const(c.dt / (c.density * c.h));  // project.go:179
    I.res_scale = c.dt / (c.density * c.h * c.h);
    I.thresh = 0.5 * c.div_tol;
    I.max_refine = (unsigned)c.max_refine;
    I.parity = 0;
    I.warm = b->cold ? 0 : 1;
    cudaMemsetAsync(b->d_ctl + s, 0, sizeof(Ctl), b->stream);  // no measured V-cycle factor yet
    // Smoothing sweeps per level are a property of the batch's step graph:
    // the first slot of an empty batch sets them.
    b->nu = batch_nu;
    S.used = true;
    S.active = true;
    b->tables_dirty = true;
    return s;
}

void batch_release(Batch* b, int s) {
    SlotHost& S = b->slots[s];
    if (!S.used) return;
    cudaStreamSynchronize(b->stream);
    if (b->use_pool) b->pool.release(S.mem, S.mem_bytes);
    else cudaFree(S.mem);
    S = SlotHost();
    b->tables_dirty = true;
}

void batch_set_active(Batch* b, int s, bool active) {
    if (b->slots[s].active != active) {
        b->slots[s].active = active;
        b->tables_dirty = true;
    }
}

af_field_desc batch_field(const Batch* b, int s, int field, double** dev) {
    const SlotHost& S = b->slots[s];
    int f = field;
    if (S.d.parity && field != 0 && field != 4) f = field <= 3 ? field + 4 : field - 4;
    if (dev) *dev = S.d.slot[f];
    return S.desc[f];
}

const Geom& batch_geom(const Batch* b, int s) { return b->slots[s].d.g; }
cudaStream_t batch_stream(Batch* b) { return b->stream; }

cudaError_t batch_step(Batch* b, int64_t nsteps, std::string* err, const std::vector<int64_t>* stop_at) {
    cudaError_t rc;
    if ((rc = prepare(b)) != cudaSuccess) {
        *err = std::string("aeroflux: cuda: preparing the batched step: ") + cudaGetErrorString(rc);
        return rc;
    }
    if ((rc = reset_status(b, stop_at, nsteps)) != cudaSuccess) return rc;
    for (int64_t i = 0; i < nsteps; ++i)
        if ((rc = cudaGraphLaunch(b->graph, b->stream)) != cudaSuccess) {
            *err = std::string("aeroflux: cuda: cudaGraphLaunch: ") + cudaGetErrorString(rc);
            return rc;
        }
    return cudaSuccess;
}

cudaError_t batch_prepare_capture(Batch* b) {
    cudaError_t rc;
    b->capture_err = cudaSuccess;
    default_pair_variants(b);
    if (b->tables_dirty && (rc = upload_tables(b)) != cudaSuccess) return rc;
    if (kernel_levels(b) > b->graph_levels && b->graph) {
        cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    }
    b->graph_levels = std::max(b->graph_levels, kernel_levels(b));
    b->graph_big |= big_coarse_levels(b);
    b->graph_pair |= pair_levels(b, false);
    b->graph_pairn |= pair_levels(b, true);
    b->graph_march |= march_levels(b);
    b->graph_single |= single_levels(b);
    b->tail_smem = std::max(b->tail_smem, tail_smem_bytes(b));
    b->tail_form |= tail_form(b);
    size_grids(b);
    return cudaSuccess;
}

int64_t batch_enqueue_project(Batch* b, int parity, int gate, cudaStream_t s, bool once) {
    const int64_t before = b->launches;
    const bool prof = b->profiling;
    b->profiling = false;
    b->overlap = !once;
    enq_project(b, parity, gate, s);
    b->overlap = true;
    b->profiling = prof;
    return b->launches - before;
}

cudaError_t batch_capture_error(Batch* b) {
    const cudaError_t rc = b->capture_err;
    b->capture_err = cudaSuccess;
    return rc;
}

Status* batch_status(Batch* b, int slot) { return b->d_st + slot; }

cudaError_t batch_project(Batch* b, std::string* err) {
    cudaError_t rc;
    if ((rc = batch_prepare_capture(b)) != cudaSuccess) return rc;
    if ((rc = reset_status(b)) != cudaSuccess) return rc;
    cudaGraphExec_t g = nullptr;
    const bool prof = b->profiling;
    b->profiling = false;
    b->overlap = false;
    rc = capture(b, [&] { enq_project(b, 0, 0, b->stream); }, &g);
    b->overlap = true;
    b->profiling = prof;
    if (rc != cudaSuccess) {
        *err = std::string("aeroflux: cuda: capturing the projection: ") + cudaGetErrorString(rc);
        return rc;
    }
    rc = cudaGraphLaunch(g, b->stream);
    cudaStreamSynchronize(b->stream);
    cudaGraphExecDestroy(g);
    return rc;
}

cudaError_t batch_velocity_bc(Batch* b) {
    cudaError_t rc;
    if (b->tables_dirty && (rc = upload_tables(b)) != cudaSuccess) return rc;
    if ((rc = reset_status(b)) != cudaSuccess) return rc;
    cudaStream_t s = b->stream;
    enq_bc(b, 0, 0, s);
    return cudaGetLastError();
}

cudaError_t batch_sweep(Batch* b, int axis, double dt) {
    cudaError_t rc;
    // A sweep at a caller-chosen dt: the per-slot sweep constants change for
    // this launch only.
    std::vector<std::pair<float, float>> keep;
    for (auto& S : b->slots) {
        keep.emplace_back(S.d.dt_invh, S.d.lam);
        if (!S.used) continue;
        const double invH = 1.0 / S.cfg.h;
        S.d.dt_invh = (float)(dt * invH);
        S.d.lam = (float)(S.cfg.viscosity * dt * invH * invH);
    }
    if ((rc = upload_tables(b)) != cudaSuccess) return rc;
    if ((rc = reset_status(b)) != cudaSuccess) return rc;
    cudaStream_t s = b->stream;
    enq_sweep(b, axis, 0, 0, s);
    rc = cudaGetLastError();
    for (int i = 0; i < b->cap; ++i) {
        b->slots[i].d.dt_invh = keep[i].first;
        b->slots[i].d.lam = keep[i].second;
    }
    b->tables_dirty = true;
    if (rc != cudaSuccess) return rc;
    if ((rc = cudaStreamSynchronize(s)) != cudaSuccess) return rc;
    std::vector<Status> st(b->cap);
    cudaMemcpy(st.data(), b->d_st, sizeof(Status) * b->cap, cudaMemcpyDeviceToHost);
    for (int i = 0; i < b->cap; ++i)
        if (b->slots[i].used && b->slots[i].active && st[i].fault_gate == kNoFault) b->slots[i].d.parity ^= 1;
    b->tables_dirty = true;
    return cudaSuccess;
}

cudaError_t batch_seed(Batch* b, int s, double amp, double noise, uint64_t seed, uint64_t stream) {
    SlotHost& S = b->slots[s];
    if (!S.used) return cudaErrorInvalidValue;
    // The fields start from zero (as after New), then the write ranges are set.
    for (int f = 1; f <= 3; ++f) cudaMemsetAsync(S.d.slot[f], 0, (size_t)S.desc[f].count * 8, b->stream);
    for (int f = 5; f <= 7; ++f) cudaMemsetAsync(S.d.slot[f], 0, (size_t)S.desc[f].count * 8, b->stream);
    S.d.parity = 0;
    b->tables_dirty = true;
    return seed_tg_fields(S.d.g, S.d.slot[1], S.d.slot[2], S.d.slot[3], S.cfg.h, amp, noise, seed, stream, b->stream);
}

cudaError_t seed_tg_fields(const Geom& g, double* u, double* v, double* w, double h, double amp, double noise,
                           uint64_t seed, uint64_t stream, cudaStream_t s) {
    // pcg32_srandom_r(seed, stream): state 0, one step, add the seed, one step.
    const unsigned long long inc = (stream << 1u) | 1u;
    unsigned long long st = inc;
    st += seed;
    st = st * 6364136223846793005ull + inc;
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    k_seed_tg<<<sms * 4, 256, 0, s>>>(g, u, v, w, (float)h, st, inc, amp, noise);
    return cudaGetLastError();
}

int batch_collect_faults(Batch* b, std::string* msg, int* first_slot) {
    std::vector<Status> st(b->cap);
    cudaStreamSynchronize(b->stream);
    cudaMemcpy(st.data(), b->d_st, sizeof(Status) * b->cap, cudaMemcpyDeviceToHost);
    int n = 0;
    *first_slot = -1;
    for (int s = 0; s < b->cap; ++s) {
        SlotHost& S = b->slots[s];
        if (!S.used || !status_faulted(st[s])) continue;
        if (n++ == 0) {
            *first_slot = s;
            *msg = fault_message_for(S.d.g, st[s].fault_gate, st[s].fault_key);
        }
        // The faulting step returned before commitVelocity of the faulting
        // sweep: `phase` commits happened in it.
        S.d.parity ^= (int)((st[s].fault_gate % 8u) & 1u);
        b->tables_dirty = true;
    }
    return n;
}

bool batch_debug_bounds(unsigned long long* first, unsigned* count, bool reset) {
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

bool batch_device_error(Batch* b, std::string* msg) {
    unsigned v = 0;
    cudaStreamSynchronize(b->stream);
    cudaMemcpy(&v, b->d_diag, sizeof v, cudaMemcpyDeviceToHost);
    if (!v) return false;
    cudaMemset(b->d_diag, 0, sizeof v);
    *msg = (v & 4u)   ? "aeroflux: cuda: a staged kernel's shared-memory buffers are not 128-byte aligned; the step's "
                        "results are invalid"
           : (v & 2u) ? "aeroflux: cuda: a smoothing kernel gave up waiting for its block; the step's results are "
                        "invalid"
                      : "aeroflux: cuda: a staged kernel gave up waiting for its tile transfer; the step's results "
                        "are invalid";
    return true;
}

bool batch_slot_faulted(const Batch* b, int s, std::string* msg) {
    Status st;
    cudaMemcpy(&st, b->d_st + s, sizeof st, cudaMemcpyDeviceToHost);
    if (!status_faulted(st)) return false;
    *msg = fault_message_for(b->slots[s].d.g, st.fault_gate, st.fault_key);
    return true;
}

void batch_slot_projection(Batch* b, int s, int64_t* passes, double* max_div, int64_t* vcycles) {
    Ctl c;
    cudaStreamSynchronize(b->stream);
    cudaMemcpy(&c, b->d_ctl + s, sizeof c, cudaMemcpyDeviceToHost);
    *passes = c.passes;
    *max_div = c.last_div;
    if (vcycles) *vcycles = c.vtotal;
}

cudaError_t batch_profile(Batch* b, bool on) {
    if (on == b->profiling) return cudaSuccess;
    cudaStreamSynchronize(b->stream);
    if (on)
        for (auto& ev : b->ev)
            if (!ev) {
                cudaError_t rc = cudaEventCreate(&ev);
                if (rc != cudaSuccess) return rc;
            }
    b->profiling = on;
    if (b->graph) {
        cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    }
    return cudaSuccess;
}

cudaError_t batch_last_profile(Batch* b, double* step_ms, double* sweep_ms, double* proj_ms, int64_t* launches) {
    if (!b->profiling) return cudaErrorInvalidValue;
    cudaError_t rc = cudaStreamSynchronize(b->stream);
    if (rc != cudaSuccess) return rc;
    auto ms = [&](int a, int c) {
        float t = 0;
        rc = cudaEventElapsedTime(&t, b->ev[a], b->ev[c]);
        return (double)t;
    };
    *step_ms = ms(kEvStart, kEvEnd);
    *sweep_ms = 0;
    for (int k = 0; k < 6; ++k) *sweep_ms += ms(kEvSweep + 2 * k, kEvSweep + 2 * k + 1);
    *proj_ms = ms(kEvProj, kEvProj + 1) + ms(kEvProj + 2, kEvProj + 3);
    *launches = b->launches;
    return rc;
}

// ---------------------------------------------------------------------------
// Autotuner: for every stage that has work, time each candidate shape on the
// current slots (each launch is idempotent or acts on scratch that the next
// projection reinitialises; run it before uploading fields, or between
// steps) and keep the fastest.
// ---------------------------------------------------------------------------
std::string batch_tune(Batch* b, int reps) {
    const Shape cands[] = {{128, 1, 8}, {256, 1, 8}, {512, 1, 4}, {256, 2, 8}, {256, 4, 8},
                           {128, 4, 16}, {256, 1, 16}, {512, 2, 4}, {1024, 1, 2}};
    std::string report = "{";
    for (int& gz : b->grid_sz) gz = 0;
    reps = std::max(1, reps);
    std::vector<cudaEvent_t> rev(2 * (size_t)reps);
    for (auto& ev : rev) cudaEventCreate(&ev);
    cudaStream_t s = b->stream;
    // The control records must see the slots as they are now (a slot
    // assigned since the last upload would read as inactive, and every
    // multigrid stage would be timed as a no-op).
    if (b->tables_dirty) upload_tables(b);
    kb_init<<<1, 256, 0, s>>>(b->d_inst, b->d_ctl, b->cap);
    reset_status(b);
    const int L = max_levels(b);
    auto run = [&](int st) {
        const Tab t = tab(b, st);
        const int gsz = grid(b, st), tpb = b->shape[st].tpb;
        if (st == S_BC) kb_bc<<<gsz, tpb, 0, s>>>(b->d_inst, b->d_st, t, 0, 0);
        else if (st == S_SWEEP) kb_sweep<0><<<gsz, tpb, 0, s>>>(b->d_inst, b->d_st, t, 0, 0);
        else if (st == S_SHADOW) kb_shadow<<<gsz, tpb, 0, s>>>(b->d_inst, t, 0);
        else if (st == S_DIV) kb_div<<<gsz, tpb, 0, s>>>(b->d_inst, b->d_st, t, 0, 0);
        else if (st == S_INT) kb_residual<<<gsz, tpb, 0, s>>>(b->d_inst, b->d_st, b->d_ctl, t, 0, 0);
        else if (st == S_PBC) kb_pbc<<<gsz, tpb, 0, s>>>(b->d_inst, b->d_st, t, 0);
        else if (st == S_GRAD) kb_grad<<<gsz, tpb, 0, s>>>(b->d_inst, b->d_st, t, 0, 0, 1);
        else if (st >= S_SMOOTH && st < S_RESTRICT) kb_smooth<<<gsz, tpb, 0, s>>>(b->d_inst, b->d_ctl, t, st - S_SMOOTH, 0, 0);
        else if (st >= S_RESTRICT && st < S_PROLONG)
            kb_restrict<<<gsz, tpb, 0, s>>>(b->d_inst, b->d_ctl, t, st - S_RESTRICT, 0);
        else if (st >= S_PROLONG && st < S_BIGCOARSE)
            kb_prolong<<<gsz, tpb, 0, s>>>(b->d_inst, b->d_ctl, t, st - S_PROLONG, 0);
        else if (st >= S_PAIR && st < S_PAIRN) launch_pair(b, st, st - S_PAIR, 0, 0, s);
        else if (st >= S_PAIRN && st < S_PAIRN + kMaxLev) launch_pair(b, st, st - S_PAIRN, 0, 0, s);
        else if (st >= S_MARCH) launch_march(b, st - S_MARCH, 0, 0, s);
    };
    std::vector<int> stages = {S_BC, S_SHADOW, S_DIV, S_INT, S_PBC, S_GRAD};
    if (!b->tma_sweep) stages.push_back(S_SWEEP);  // the staged sweep keeps its fixed tile shape
    for (int l = 0; l + 1 < L; ++l) {
        stages.push_back(S_SMOOTH + l);
        stages.push_back(S_RESTRICT + l);
        stages.push_back(S_PROLONG + l);
    }
    default_pair_variants(b);
    b->pair_chosen = true;
    // Per-launch median of stage st under its present shape, microseconds (each
    // repetition timed on its own: one disturbed launch does not decide);
    // negative when a launch failed.  Events resolve about 2 us, so a
    // repetition of a short stage is two or four launches (decided by the first
    // candidate's warm-up, *launches = 0).
    auto timed = [&](int st, int* launches) {
        upload_stage(b, st);
        if (*launches == 0) cudaEventRecord(rev[0], s);
        run(st);  // warm-up
        if (*launches == 0) {
            cudaEventRecord(rev[1], s);
            cudaEventSynchronize(rev[1]);
            float once = 0.0f;
            cudaEventElapsedTime(&once, rev[0], rev[1]);
            *launches = once < 0.015f ? 4 : (once < 0.03f ? 2 : 1);
        }
        for (int r = 0; r < reps; ++r) {
            cudaEventRecord(rev[2 * r], s);
            for (int k = 0; k < *launches; ++k) run(st);
            cudaEventRecord(rev[2 * r + 1], s);
        }
        cudaEventSynchronize(rev[2 * reps - 1]);
        std::vector<float> t(reps);
        for (int r = 0; r < reps; ++r) cudaEventElapsedTime(&t[r], rev[2 * r], rev[2 * r + 1]);
        std::nth_element(t.begin(), t.begin() + reps / 2, t.end());
        return cudaGetLastError() == cudaSuccess ? 1e3f * t[reps / 2] / *launches : -1.0f;
    };
    auto has_items = [&](int st) {
        for (auto& S : b->slots)
            if (stage_items(b, S, st, b->shape[st])) return true;
        return false;
    };
    auto report_stage = [&](int st, const Shape& sh, int var, float us, const std::string& variants) {
        char buf[160];
        snprintf(buf, sizeof buf,
                 "%s\"stage_%d\": {\"tpb\": %d, \"ept\": %d, \"blocks_per_sm\": %d, \"variant\": %d, \"us\": %.2f",
                 report.size() > 1 ? ", " : "", st, sh.tpb, sh.ept, sh.bpsm, var, us);
        report += buf;
        if (!variants.empty()) report += ", \"variants_us\": {" + variants + "}";
        report += "}";
    };
    // Gives a stage the fastest of the candidate shapes: of the first `brief`
    // only when the first one takes less than 10 us, most of it the launch.
    auto fastest = [&](int st, const std::vector<Shape>& cs, std::vector<float>* times, size_t brief) {
        Shape best = b->shape[st];
        float best_us = 1e30f, first_us = 1e30f;
        int launches = 0;
        for (size_t i = 0; i < cs.size() && (i < brief || first_us >= 10.0f); ++i) {
            const Shape& c = cs[i];
            b->shape[st] = c;
            const float us = timed(st, &launches);
            if (i == 0) first_us = us;
            if (times) times->push_back(us);
            if (us >= 0.0f && us < best_us) best_us = us, best = c;
        }
        b->shape[st] = best;
        return best_us;
    };
    for (int st : stages) {
        if (!has_items(st)) continue;
        const float us = fastest(st, std::vector<Shape>(cands, cands + sizeof cands / sizeof cands[0]), nullptr, 3);
        report_stage(st, b->shape[st], b->shape[st].var, us, "");
    }
    // Fused pairs, per level: the tile variants of both tile columns with no
    // slot marching, then the march shapes; a level marches (variant 3 of its
    // first pair stage) when that and what cannot march take less time than
    // the tiles do.
    for (int l = 0; l < L && b->force_pair_var < 0; ++l) {
        const unsigned bit = 1u << l;
        b->march &= ~bit;
        const int stages2[2] = {S_PAIR + l, S_PAIRN + l};
        std::vector<float> t[2];
        float tile_us[2] = {0.0f, 0.0f};
        bool has[2];
        for (int w = 0; w < 2; ++w) {
            has[w] = has_items(stages2[w]);
            if (!has[w]) continue;
            std::vector<Shape> cs;
            for (int v : kPairTileVars) cs.push_back(pair_shape(w == 0, v));
            tile_us[w] = fastest(stages2[w], cs, &t[w], cs.size());
        }
        if (!has[0] && !has[1]) continue;
        const float tiles = tile_us[0] + tile_us[1];
        float march_us = -1.0f;
        b->march |= bit;
        if (has_items(S_MARCH + l)) {
            std::vector<Shape> cs;
            long long most = 0;  // the largest level's cells: small ones have no use for long chunks of large blocks
            for (auto& S : b->slots)
                if (S.used && S.active && l < S.d.nlev) most = std::max(most, lvl_cells(S.d.lev[l]));
            for (int m = 0; m < kMarchShapeCount; ++m)
                if (most >= (1ll << 20) ? kMarchShapes[m].zc >= 8 : kMarchShapes[m].k == 0)
                    cs.push_back(march_shape(m));
            march_us = fastest(S_MARCH + l, cs, nullptr, cs.size());
            for (int st : stages2)
                if (has_items(st)) {  // slots that cannot march
                    int launches = 0;
                    march_us += std::max(0.0f, timed(st, &launches));
                }
        }
        const bool march = march_us >= 0.0f && march_us < tiles;
        if (!march) b->march &= ~bit;
        const int lead = has[0] ? 0 : 1;  // the stage whose report carries the level's choice
        for (int w = 0; w < 2; ++w) {
            if (!has[w]) continue;
            const float other = w == lead ? tiles - tile_us[w] : 0.0f;
            std::string variants;
            char buf[64];
            for (size_t v = 0; v < t[w].size(); ++v) {
                snprintf(buf, sizeof buf, "%s\"%d\": %.2f", v ? ", " : "", kPairTileVars[v],
                         t[w][v] < 0.0f ? -1.0f : t[w][v] + other);
                variants += buf;
            }
            if (w == lead && march_us >= 0.0f) {
                snprintf(buf, sizeof buf, ", \"3\": %.2f", march_us);
                variants += buf;
            }
            const bool m = w == lead && march;
            report_stage(stages2[w], m ? b->shape[S_MARCH + l] : b->shape[stages2[w]],
                         m ? 3 : b->shape[stages2[w]].var, m ? march_us : tile_us[w] + other, variants);
        }
    }
    report += "}";
    for (auto& ev : rev) cudaEventDestroy(ev);
    upload_tables(b);
    kb_init<<<1, 256, 0, s>>>(b->d_inst, b->d_ctl, b->cap);
    if (b->graph) {
        cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    }
    cudaStreamSynchronize(s);
    return report;
}

// Contained-fault text of the reference (arena.go:230-243 around Go's
// bounds-check panic) for a NaN backtrace at fault key `key` in sweep phase
// gate%8: the tap indices follow from the face, component, axis and strides.
std::string fault_message_for(const Geom& g, unsigned gate, unsigned long long key) {
    const int phase = (int)(gate % 8u);
    const int axis = phase < 3 ? kFwd[phase] : kRev[phase - 3];
    const int comp = (int)(key >> 60);
    const unsigned long long z = (key >> 40) & 0xFFFFF, y = (key >> 20) & 0xFFFFF, x = key & 0xFFFFF;
    const Dims& d = comp == 0 ? g.u : (comp == 1 ? g.v : g.w);
    unsigned long long x0 = x, y0 = y, z0 = z;
    const unsigned long long nan_int = 0x8000000000000000ull;
    if (axis == 0) x0 = nan_int;
    if (axis == 1) y0 = nan_int;
    if (axis == 2) z0 = nan_int;
    const unsigned long long sy = (unsigned long long)d.sy, sz = (unsigned long long)d.sz;
    const unsigned long long i000 = x0 + y0 * sy + z0 * sz;
    const unsigned long long taps[8] = {i000, i000 + 1, i000 + sy, i000 + sy + 1,
                                        i000 + sz, i000 + sz + 1, i000 + sz + sy, i000 + sz + sy + 1};
    char buf[200];
    for (unsigned long long t : taps) {
        const long long idx = (long long)t;
        if (idx < 0) {
            snprintf(buf, sizeof buf, "aeroflux: guard-page fault contained: runtime error: index out of range [%lld]", idx);
            return buf;
        }
        if (idx >= d.count) {
            snprintf(buf, sizeof buf,
                     "aeroflux: guard-page fault contained: runtime error: index out of range [%lld] with length %lld",
                     idx, (long long)d.count);
            return buf;
        }
    }
    return "aeroflux: guard-page fault contained: runtime error: index out of range";
}

}  // namespace af
