// Device helpers shared by the sm_100a eigensolver kernels: complex FP64
// arithmetic on double2, warp / column-group reductions, the total order used
// to rank eigenvalues, and the fast FP64 reciprocal.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#ifdef SGEIG_PHASE_TIMERS
#include <vector>
#endif

namespace sgeig {

// A kernel launch; `started` (may be NULL) is recorded when the last of its CTAs
// has begun.
template <class... Args>
inline cudaError_t launch_with_event(void (*kernel)(Args...), unsigned grid, int threads, size_t smem,
                                     cudaStream_t stream, cudaEvent_t started, const Args&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeLaunchCompletionEvent;
    at.val.launchCompletionEvent.event = started;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    c.attrs = &at;
    c.numAttrs = started ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, args...);
}

// ---------------------------------------------------------------- complex FP64
__device__ __forceinline__ double2 c2(double re, double im) { return make_double2(re, im); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return c2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return c2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return c2(a.x * s, a.y * s); }
__device__ __forceinline__ double2 cconj(double2 a) { return c2(a.x, -a.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return c2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// acc + a*b
__device__ __forceinline__ double2 cfma(double2 acc, double2 a, double2 b) {
    acc.x = fma(a.x, b.x, acc.x); acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y); acc.y = fma(a.y, b.x, acc.y);
    return acc;
}
// acc - a*b
__device__ __forceinline__ double2 cfms(double2 acc, double2 a, double2 b) {
    acc.x = fma(-a.x, b.x, acc.x); acc.x = fma(a.y, b.y, acc.x);
    acc.y = fma(-a.x, b.y, acc.y); acc.y = fma(-a.y, b.x, acc.y);
    return acc;
}
// acc + conj(a)*b
__device__ __forceinline__ double2 cfmac(double2 acc, double2 a, double2 b) {
    acc.x = fma(a.x, b.x, acc.x); acc.x = fma(a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y); acc.y = fma(-a.y, b.x, acc.y);
    return acc;
}
// acc - conj(a)*b
__device__ __forceinline__ double2 cfmsc(double2 acc, double2 a, double2 b) {
    acc.x = fma(-a.x, b.x, acc.x); acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(-a.x, b.y, acc.y); acc.y = fma(a.y, b.x, acc.y);
    return acc;
}
// acc - a*conj(b)
__device__ __forceinline__ double2 cfms_bc(double2 acc, double2 a, double2 b) {
    acc.x = fma(-a.x, b.x, acc.x); acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y); acc.y = fma(-a.y, b.x, acc.y);
    return acc;
}

// ---------------------------------------------------------------- reductions
// One FP64 tensor-core step D += A B on an 8x8x4 tile (mma.m8n8k4.f64).
// Fragments: lane l holds A(l/4, l%4), B(l%4, l/4) and D(l/4, 2(l%4)+{0,1}).
__device__ __forceinline__ void mma884(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}
// Sum over the warp's lanes, the same value in every lane, as two tensor-core
// steps with A = 1: the first sums each B column (four lanes), leaving columns
// 2q and 2q + 1 in the lanes l%4 == q; their sum as the second step's B adds
// the four pairs. Two dependent steps and an add (60 cycles, 3 instructions)
// where five shuffle-and-add rounds take 175 cycles and 15 instructions.
__device__ __forceinline__ double warp_sum(double v) {
    double c[2] = {0.0, 0.0}, t[2] = {0.0, 0.0};
    mma884(c, 1.0, v);
    mma884(t, 1.0, c[0] + c[1]);
    return t[0];
}
__device__ __forceinline__ double2 warp_sum2(double2 v) { return c2(warp_sum(v.x), warp_sum(v.y)); }
// Sum over the G consecutive lanes of one column group (G a power of two).
template <int G>
__device__ __forceinline__ double2 group_sum2(unsigned mask, double2 v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(mask, v.x, o, G);
        v.y += __shfl_xor_sync(mask, v.y, o, G);
    }
    return v;
}
template <int G>
__device__ __forceinline__ double2 group_bcast2(unsigned mask, double2 v, int src) {
    v.x = __shfl_sync(mask, v.x, src, G);
    v.y = __shfl_sync(mask, v.y, src, G);
    return v;
}

// First index i >= start with i % G == q.
template <int G>
__device__ __forceinline__ int first_in_class(int start, int q) {
    int d = q - (start % G);
    if (d < 0) d += G;
    return start + d;
}

// Total-order sort key for eigenvalues: NaN sorts after +inf, so that ranks
// computed as #{t : key_t < key_j or (key_t == key_j and t < j)} always form
// a permutation (they are used as indices).
__host__ __device__ __forceinline__ double order_key(double x) {
    return (x != x) ? __builtin_inf() : x;
}

// Reciprocal without a divide: the hardware's approximate FP64 reciprocal
// (PTX rcp.approx.ftz.f64) refined by two Newton-Raphson steps
// r <- r + r (1 - x r), each of which doubles the number of correct bits.
// Branch-free, so independent reciprocals pipeline, unlike IEEE division.
// Accuracy (checked against 1/x on the GPU by the self-test entry point):
// within 1 ulp for normal x; x = 0 or +-inf give NaN (callers never pass them).
__host__ __device__ __forceinline__ double fast_rcp(double x) {
#ifdef __CUDA_ARCH__
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    double e = fma(-x, r, 1.0);
    r = fma(r, e, r);
    e = fma(-x, r, 1.0);
    return fma(r, e, r);
#else
    return 1.0 / x;
#endif
}

// ---------------------------------------------------------------- teams
// The NT threads that solve one pencil in a CTA of BLOCK threads: the whole
// CTA when BLOCK == NT, else one of its BLOCK / NT teams of consecutive whole
// warps (several pencils per CTA). team_sync is the team's barrier:
// __syncwarp for a team of one warp, __syncthreads for a whole-CTA team,
// named barrier 1 + team otherwise (barrier 0 stays the CTA's own).
template <int NT, int BLOCK>
__device__ __forceinline__ unsigned team_tid() {
    if constexpr (BLOCK == NT) return threadIdx.x;
    else return threadIdx.x % NT;
}
template <int NT, int BLOCK>
__device__ __forceinline__ void team_sync() {
    static_assert(NT % 32 == 0 && BLOCK % NT == 0 && BLOCK / NT <= 15, "team shape");
    if constexpr (NT == 32) __syncwarp();
    else if constexpr (BLOCK == NT) __syncthreads();
    else asm volatile("bar.sync %0, %1;" :: "r"(1 + (int)(threadIdx.x / NT)), "n"(NT) : "memory");
}

// Makes the compiler forget what it knows of x, so that address arithmetic
// derived from x is redone where it is used instead of being kept (or
// spilled) across the phases of a long kernel.
__device__ __forceinline__ void forget(int& x) { asm volatile("" : "+r"(x)); }

// ---------------------------------------------------------------- reflectors
// Householder's elementary reflector I - tau v v^H, v = (1, scal x), that takes
// (alpha, x) to (beta, 0) with beta real (zlarfg), from rest = ||x||^2 +
// Im(alpha)^2 and nn = rest + Re(alpha)^2.
struct Reflector {
    double2 tau, scal;
    double beta;
};
// True where the squares neither underflow nor overflow and rest is not zero
// (rest at least 2^-927, nn below 2^929, about 1e-279 and 1e+279; compares on the
// exponents, false for NaN): reflector() holds.
__device__ __forceinline__ bool squares_safe(double rest, double nn) {
    return __double2hiint(rest) >= 0x06000000 && __double2hiint(nn) < 0x7a000000;
}
__device__ __forceinline__ Reflector reflector(double2 alpha, double nn) {
    Reflector h;
    const double rn = rsqrt(nn);                         // 1 / beta comes with the root
    h.beta = -copysign(nn * rn, alpha.x);
    const double rbeta = -copysign(rn, alpha.x);
    h.tau = c2((h.beta - alpha.x) * rbeta, -alpha.y * rbeta);
    const double2 z = c2(alpha.x - h.beta, alpha.y);
    const double inv = fast_rcp(fma(z.x, z.x, z.y * z.y));
    h.scal = c2(z.x * inv, -z.y * inv);
    return h;
}
// Otherwise the same from the column times f = column_scale(nn) (as = f alpha,
// rest its sum): columns of zeros, those that the rounding residues of a low-rank
// matrix leave (1e-16, 1e-32, 1e-48, ... of its norm), and matrices of extreme
// scale. A column below 2^-1000 is zero, and so is one whose x underflows beside an
// alpha above 2^-200.
__device__ __forceinline__ double column_scale(double nn) { return nn < 0x1p-400 ? 0x1p700 : 0x1p-700; }
__device__ __forceinline__ Reflector reflector_scaled(double2 alpha, double2 as, double rest, double f) {
    const double nn = fma(as.x, as.x, rest);
    Reflector h;
    h.tau = h.scal = c2(0.0, 0.0);
    h.beta = alpha.x;
    if (!(rest == 0.0 || (f > 1.0 && nn < 0x1p-600))) {
        h = reflector(as, nn);
        h.beta *= f > 1.0 ? 0x1p-700 : 0x1p700;
        h.scal = cscale(h.scal, f);                      // scal is applied to x itself
    }
    return h;
}

// ---------------------------------------------------------------- constants
// LAPACK dlamch convention: eps = 2^-53 (relative machine precision).
constexpr double kEps    = 1.1102230246251565e-16;

// ---------------------------------------------------------------- failure codes
// Internal marker of a failed tridiagonal eigensolve (non-finite values):
// distinct from every info code (0, 1..n, n+1..2n).
constexpr int kEigFailCode = -1;
// The info such a pencil reports, LAPACK zhegv's for the same input: its
// tridiagonal QR counts the n - 1 off-diagonal elements that did not
// converge, and for n <= 2 it returns 0 with NaN eigenvalues (W and U are
// NaN-filled here in every case).
__host__ __device__ __forceinline__ int eig_fail_info(int n) { return n >= 3 ? n - 1 : 0; }

// ---------------------------------------------------------------- phase timers
// Profiling builds only (-DSGEIG_PHASE_TIMERS, built as a separate library by
// build.py --phase-timers): thread 0 of every CTA adds the clock64 cycles
// since its previous mark to the counter of the phase that just ended. Marks
// sit right after CTA barriers, so a counter divided by the number of solves
// is the CTA time per solve spent in that phase (with the SM shared by the
// other resident CTAs, as in a normal run). The product library compiles
// every mark to nothing.
constexpr int kPhaseSlots = 32;
#ifdef SGEIG_PHASE_TIMERS
static __device__ unsigned long long g_phase_cycles[kPhaseSlots];
__device__ __forceinline__ long long& phase_prev() {
    __shared__ long long t;
    return t;
}
__device__ __forceinline__ unsigned& phase_level();
__device__ __forceinline__ void phase_start() {
    if (threadIdx.x == 0) { phase_prev() = clock64(); phase_level() = 0; }
}
__device__ __forceinline__ void phase_mark(int slot) {
    if (threadIdx.x == 0) {
        const long long t = clock64();
        atomicAdd(&g_phase_cycles[slot], (unsigned long long)(t - phase_prev()));
        phase_prev() = t;
    }
}
// Event counters in the same array (profiling builds): phase_count adds v
// to a slot; phase_level_max keeps the largest v seen since the last
// phase_level_flush, which (thread 0, after a barrier) adds it to a slot.
__device__ __forceinline__ unsigned& phase_level() {
    __shared__ unsigned m;
    return m;
}
__device__ __forceinline__ void phase_count(int slot, unsigned long long v) { atomicAdd(&g_phase_cycles[slot], v); }
__device__ __forceinline__ void phase_level_max(unsigned v) { atomicMax(&phase_level(), v); }
__device__ __forceinline__ void phase_level_flush(int slot) {
    if (threadIdx.x == 0) {
        atomicAdd(&g_phase_cycles[slot], (unsigned long long)phase_level());
        phase_level() = 0;
    }
}
// Adds this translation unit's counters to `out` (and clears them). Each unit
// that includes this header puts its own into phase_readers().
static inline cudaError_t add_phase_cycles(unsigned long long* out, int count, bool reset) {
    unsigned long long mine[kPhaseSlots] = {};
    cudaError_t e = cudaMemcpyFromSymbol(mine, g_phase_cycles, sizeof(mine));
    for (int i = 0; e == cudaSuccess && i < count && i < kPhaseSlots; ++i) out[i] += mine[i];
    if (e == cudaSuccess && reset) {
        static const unsigned long long zeros[kPhaseSlots] = {};
        e = cudaMemcpyToSymbol(g_phase_cycles, zeros, sizeof(zeros));
    }
    return e;
}
using PhaseReader = cudaError_t (*)(unsigned long long* out, int count, bool reset);
inline std::vector<PhaseReader>& phase_readers() {
    static std::vector<PhaseReader> r;
    return r;
}
static const bool g_phase_registered = (phase_readers().push_back(add_phase_cycles), true);
#else
__device__ __forceinline__ void phase_start() {}
__device__ __forceinline__ void phase_mark(int) {}
__device__ __forceinline__ void phase_count(int, unsigned long long) {}
__device__ __forceinline__ void phase_level_max(unsigned) {}
__device__ __forceinline__ void phase_level_flush(int) {}
#endif

}  // namespace sgeig
