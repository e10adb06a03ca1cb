// af_internal.h -- types shared by the engine (af_engine.cu) and the kernels
// (af_fp64.cu, af_batch.cu).  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <string>

namespace af {

// Field geometry on the device: padded extents and strides of grid.go:12-21.
// A field holds fewer than 2^31 elements (af_create and batch_config_fits
// refuse larger grids), so most kernels index it in int.
struct Dims {
    int nx, ny, nz;
    long long sy, sz, count;
};

// Grid geometry shared by every stage.
struct Geom {
    int NX, NY, NZ, G;   // interior extents and ghost thickness
    Dims p, u, v, w;     // P (= Div shape), U (= Tmp0), V (= Tmp1), W (= Tmp2)
};

// Unsigned 32-bit division by an invariant divisor with one multiply-high
// (Granlund & Montgomery, "Division by invariant integers using
// multiplication", 1994): l = ceil(log2 d), m = ceil(2^(32+l)/d) - 2^32,
// n/d = (umulhi(n, m) + n) >> l for every n < 2^32.
struct FastDiv {
    unsigned d = 1, m = 0, l = 0;
    FastDiv() = default;
    __host__ explicit FastDiv(unsigned div) : d(div) {
        while ((1ull << l) < d) ++l;
        m = (unsigned)((((1ull << (32 + l)) + d - 1) / d) - (1ull << 32));
    }
    __device__ __forceinline__ unsigned div(unsigned n) const {
        return (unsigned)(((unsigned long long)__umulhi(n, m) + n) >> l);
    }
};

// Scratch of the red-black solver: P and B = h^2 Div split by colour, so a
// colour's update reads and writes contiguous cells and touches no cell it
// does not need.  Colour c holds the interior cells (x, y, z) with
// x + y + z + G = c (mod 2), at half index x >> 1.  P rows carry one ghost
// cell on every side (pitch px = hx + 2, NY + 2 rows, NZ + 2 planes per
// colour); a wall cell's ghost lies in the other colour's array, where its
// update writes its new value too (applyPressureBC, project.go:139-163:
// before a cell is updated its face ghosts hold the cell's own value).
// B holds the interior only (pitch hx).
struct Split {
    int NX, NY, NZ, G;
    int hx, px, plane;      // (NX+1)/2, hx + 2, px * (NY + 2)
    long long pn, bn;       // elements per colour of p and b
    double* p;
    double* b;
    FastDiv fhx;
    static Split of(const Geom& g) {
        Split s{};
        s.NX = g.NX, s.NY = g.NY, s.NZ = g.NZ, s.G = g.G;
        s.hx = (g.NX + 1) / 2;
        s.px = s.hx + 2;
        s.plane = s.px * (g.NY + 2);
        s.pn = (long long)s.plane * (g.NZ + 2);
        s.bn = (long long)s.hx * g.NY * g.NZ;
        s.fhx = FastDiv((unsigned)s.hx);
        return s;
    }
    size_t bytes() const { return (size_t)(2 * pn + 2 * bn) * sizeof(double); }
    void place(void* mem) {
        p = (double*)mem;
        b = p + 2 * pn;
    }
};

// Device status block of one engine.
//  fault_gate: step*8 + sweep phase (0..5) of the first contained fault,
//              0xFFFFFFFF when none.  Every kernel of a later phase returns at
//              entry, so the state freezes where the reference's Step returns.
//  step:       device step counter, bumped at the end of each captured step.
//  fault_key:  min over the faults of that phase of (component, z, y, x),
//              the order the reference's single-worker loop meets them.
struct Status {
    unsigned int fault_gate;
    unsigned int step;
    unsigned long long fault_key;
};

constexpr unsigned int kNoFault = 0xFFFFFFFFu;
constexpr unsigned long long kNoKey = ~0ull;

__host__ __device__ inline unsigned long long fault_key(int comp, int x, int y, int z) {
    return ((unsigned long long)comp << 60) | ((unsigned long long)(unsigned)z << 40) |
           ((unsigned long long)(unsigned)y << 20) | (unsigned long long)(unsigned)x;
}

// Pointers of the eight arena fields (current descriptor slots).
struct Fields {
    double* p;
    double* u;
    double* v;
    double* w;
    double* div;
    double* t0;
    double* t1;
    double* t2;
};

// Launches a kernel that may be scheduled while its predecessor in the stream
// still runs (programmatic dependent launch): the kernel waits for it with
// pdl_wait() before it touches anything an earlier kernel wrote or reads.
// Every kernel launched so calls pdl_wait() in every block that does work;
// then a kernel that follows finds all earlier ones finished too.  Measured
// for the red-black sweeps, us per launch: 16^3 2.01 -> 1.76, 64^3 3.26 ->
// 2.79, 128^3 11.5 -> 11.0, 256^3 79.1 -> 77.8; with the trigger at the
// kernel's start, where the early blocks take residency from the running
// ones, 64^3 3.54.
// overlap = false launches it in the usual way.
template <class... P, class... A>
void launch_maybe_pdl(bool overlap, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    launch_maybe_pdl(true, kernel, grid, block, smem, s, args...);
}
#if defined(__CUDACC__)
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

// --- FP64 plain-form stage launchers (af_fp64.cu) ---------------------------
// `gate` is the step-relative phase index a kernel belongs to: it returns at
// entry when a fault was recorded at an earlier (step, phase).
void launch_velocity_bc(const Geom& g, double* u, double* v, double* w, Status* st, int gate, cudaStream_t s);
void launch_sweep_fp64(const Geom& g, int axis, const Fields& f, double dt, double invH, double lam,
                       Status* st, int phase, cudaStream_t s);
// MacCormack form of the same sweep: forward semi-Lagrangian step into
// fwd.t0..t2 (fwd.u/v/w = f.u/v/w), then the limited correction plus the
// directional diffusion into f.t0..t2.  Two launches.
void launch_maccormack_fp64(const Geom& g, int axis, const Fields& f, const Fields& fwd, double dt, double invH,
                            double lam, Status* st, int phase, cudaStream_t s);
// computeDivergence into Div (project.go:42-62); with split, also B into it
// and its P zeroed for the red-black sweeps (project.go:81-83).
void launch_divergence_fp64(const Geom& g, const Fields& f, const Split* split, double scale, double h2, Status* st,
                            int gate, cudaStream_t s);
// B and zero P of the red-black sweeps from a Div supplied directly.
void launch_split_from_div(const Geom& g, const double* div, const Split& split, double h2, cudaStream_t s);
// One colour sweep over the split arrays (scratch only: not gated).
void launch_rbgs_fp64(const Split& split, int color, cudaStream_t s);
// Every sweep of a solve (`pairs` red-black pairs) from zero P in one launch,
// for grids small enough for it; false, nothing launched, for the others and
// where the device refuses the launch.
bool launch_rbgs_all_fp64(const Split& split, long long pairs, cudaStream_t s);
// The split P back into P, with applyPressureBC's ghosts; cells no one
// writes (ghost layers past the first) are zero.
void launch_join_fp64(const Geom& g, const Split& split, double* p, Status* st, int gate, cudaStream_t s);
void launch_pressure_bc_fp64(const Geom& g, double* p, Status* st, int gate, cudaStream_t s);
void launch_gradient_fp64(const Geom& g, const Fields& f, double scale, Status* st, int gate, cudaStream_t s);
void launch_step_tick(Status* st, cudaStream_t s);

// Diagnostics (af_fp64.cu).  `out` receives the bit pattern of a
// non-negative double (max; of max |du + dv + dw|, to be multiplied by 1/h,
// for the divergence) or the fixed-order sum; `partials` holds
// kinetic_energy_partials(g) doubles for the sum.
void launch_max_divergence(const Geom& g, const double* u, const double* v, const double* w, unsigned long long* out,
                           cudaStream_t s);
void launch_max_abs3(const double* u, long long nu, const double* v, long long nv, const double* w, long long nw,
                     unsigned long long* out, cudaStream_t s);
// MaxDivergence from launch_max_divergence's word.  A product that is not a
// number (1/h infinite and nothing to scale, or the reverse) counts for
// nothing, as in the reference's comparison.
inline double max_divergence_of(unsigned long long bits, double h) {
    double m;
    memcpy(&m, &bits, sizeof m);
    const double d = (1.0 / h) * m;
    return d == d ? d : 0.0;
}
int kinetic_energy_partials(const Geom& g);
void launch_kinetic_energy(const Geom& g, const double* u, const double* v, const double* w, double* partials,
                           double* out, cudaStream_t s);

// The reference's contained-fault text for a NaN backtrace recorded with
// fault gate `gate` (step*8 + sweep phase) and fault key `key`.
std::string fault_message_for(const Geom& g, unsigned gate, unsigned long long key);

// Writes the seeded Taylor-Green + PCG32 noise initial field into the write
// ranges of u, v, w (device, af_batch.cu).
cudaError_t seed_tg_fields(const Geom& g, double* u, double* v, double* w, double h, double amp, double noise,
                           uint64_t seed, uint64_t stream, cudaStream_t s);

// Compares both exact /6 forms with IEEE division on n random bit patterns
// (af_fp64.cu); false on a CUDA error.
bool selftest_div6(unsigned long long n, unsigned long long seed, unsigned long long* mismatches);
// Compares the integer-pipe binary64 add and subtract with the native ones.
bool selftest_dadd(unsigned long long n, unsigned long long seed, unsigned long long* mismatches);

// Debug build (AEROFLUX_DEBUG_BOUNDS): the first out-of-buffer access each
// kernel unit recorded -- (kernel << 56) | (slot << 40) | offset, ~0 when
// none -- and how many there were; reset clears them.  Product build: none.
bool fp64_debug_bounds(unsigned long long* first, unsigned* count, bool reset);
bool batch_debug_bounds(unsigned long long* first, unsigned* count, bool reset);
// Both units together; true with *msg set when the debug build recorded a
// violation (the record is then cleared).
bool debug_bounds_error(std::string* msg);

// Binary64 FMA issue rate of the current device (independent chains, timed
// with events); false on a CUDA error.
bool measure_fp64_rate(double* fma_per_s);

}  // namespace af
