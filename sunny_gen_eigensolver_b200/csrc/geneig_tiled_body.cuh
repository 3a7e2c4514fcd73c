// Per-pencil body of the tiled (l2-slot) solver, shared by its own kernel
// (geneig_tiled.cu) and the persistent uneven-size kernel (geneig_uneven.cu).
// The stage chain is described in geneig_tiled.cu.
#pragma once

// How the per-pencil body is compiled into its callers: inlined into the
// size's own kernel; a caller that dispatches several bodies (the persistent
// uneven-size kernel) may define it as __noinline__ before including, so
// that each body keeps its own register allocation.
#ifndef SGEIG_TILED_BODY_INLINE
#define SGEIG_TILED_BODY_INLINE __forceinline__
#endif

#include "geneig_common.cuh"
#include "geneig_dc.cuh"
#include "geneig_kernels.h"
namespace sgeig {
namespace tiled {

// Threads per CTA: 256, two CTAs per SM, as long as two work areas fit one; 512
// and one CTA above, where the steps want the loads of one pencil in flight and
// the slots stay closer to the L2's size. ms, 256 / 512 threads: N=111 (1184
// pencils) 8.15 / 10.11, N=128 10.5 / 12.7, N=162 (888) 15.4 / 17.5, N=200 (592)
// 16.6 / 17.7, N=216 19.7 / 20.6 in full waves but no gain in ragged ones,
// N=232 (444; one CTA per SM fits) 22.1 / 17.9.
constexpr int kTiledWide = 512, kTiledNarrow = 256, kNarrowMaxN = 200;
__host__ __device__ constexpr int tiled_threads(int n) { return n > kNarrowMaxN ? kTiledWide : kTiledNarrow; }

struct TiledArgs {
    const double2* __restrict__ H;
    const double2* __restrict__ S;
    double*  W;
    double2* U;
    int*     info;
    double2* scratch;
    long long batch;
    int n, ld, stage;
    int sigma;      // H = diag(I_{n/2}, -I_{n/2}), not read from memory
    int refine_max; // mixed: refinement steps before the FP64 fallback
    int defer;      // mixed: leave the fallback to the shared-memory kernel (info = kRetryInfo)
    // (arguments rather than functions of n in the kernel: n = 216 2.5 % faster)
    int work;       // the launch's shared memory has the work area (not tiled_rows)
    int keep32;     // mixed: it has the FP32 copy of C (tiled_keep32)
};

// Ogita-Aishima refinement of the mixed form: it stops as soon as the current
// estimate V is orthonormal and diagonalises C to rounding level
// (||I - V^H V||_F and ||V^H C V - diag(lam)||_F / max|lam| both <= 16 eps n,
// checked directly: the correction alone can look converged while vectors
// of a tight pair stay mixed), after at most TiledArgs::refine_max
// corrections (default kRefineMaxIters). Widely spread spectra (cond(S) =
// 1e5 makes C's small eigenvalues nearly clustered against ||C||) need more
// steps from the FP32 start; a pencil that has not converged by then is
// solved again in FP64.

// ---------------------------------------------------------------- complex FP32
__device__ __forceinline__ float2 f2(float re, float im) { return make_float2(re, im); }
__device__ __forceinline__ float2 fcmul(float2 a, float2 b) {
    return f2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// acc + conj(a) * b
__device__ __forceinline__ float2 fcfmac(float2 acc, float2 a, float2 b) {
    acc.x = fmaf(a.x, b.x, acc.x); acc.x = fmaf(a.y, b.y, acc.x);
    acc.y = fmaf(a.x, b.y, acc.y); acc.y = fmaf(-a.y, b.x, acc.y);
    return acc;
}
// acc + a * b
__device__ __forceinline__ float2 fcfma(float2 acc, float2 a, float2 b) {
    acc.x = fmaf(a.x, b.x, acc.x); acc.x = fmaf(-a.y, b.y, acc.x);
    acc.y = fmaf(a.x, b.y, acc.y); acc.y = fmaf(a.y, b.x, acc.y);
    return acc;
}
// acc - a * conj(b)
__device__ __forceinline__ float2 fcfms_bc(float2 acc, float2 a, float2 b) {
    acc.x = fmaf(-a.x, b.x, acc.x); acc.x = fmaf(-a.y, b.y, acc.x);
    acc.y = fmaf(a.x, b.y, acc.y); acc.y = fmaf(-a.y, b.x, acc.y);
    return acc;
}
__device__ __forceinline__ float warp_sumf(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float2 warp_sum2f(float2 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}
__device__ __forceinline__ double2 f2d(float2 a) { return c2((double)a.x, (double)a.y); }

// Shared-memory vectors of one CTA.
struct TVec {
    double2* tau;   // n    Householder scalars
    double2* vb;    // n    current Householder vector (v[k+1] = 1)
    double2* pb;    // n    tau * A22 * v
    double2* red;   // 32   reduction scratch
    double2* tb;    // 256  T factor of the current WY block (16 x 16, column-major)
    double2* part;  // threads/32 x kMvRows: per-warp partials of y = A v
    double2* ring;  // tiled_ring_elems(n): elements of A on their way
    double2* gb;    // 512  Y^H Y of the current WY block: two partial sums, then their sum
    double*  d;     // n    tridiagonal diagonal
    double*  e;     // n    tridiagonal off-diagonal
    double*  rdg;   // n    1 / L_kk
    double*  dcd;   // divide-and-conquer doubles (dc_vec_doubles(n)); eigenvalues first
    int*     rank;  // n    ascending position of eigenvalue j
    int*     ctl;   // 8    control words
    int*     dci;   // divide-and-conquer ints (dc_vec_ints(n))
};

// y = A v of the Householder steps: rows per warp, and the columns whose
// elements a lane has on their way to shared memory.
constexpr int kMvRows = 128, kMvDepth = 3;
__host__ __device__ inline size_t tiled_part_elems(int n) { return (size_t)(tiled_threads(n) / 32) * kMvRows; }
__host__ __device__ inline size_t tiled_ring_elems(int n) { return (size_t)kMvDepth * (kMvRows / 32) * tiled_threads(n); }
// The work area of the blocked FP64 reduction (tiled_house), last in shared
// memory. Small sizes are reduced by house_rows and go without it, which leaves
// the SM's L1 to the matrices. ms, two slots per SM, house_rows / tiled_house:
// N=16 (4096 pencils) 1.36 / 1.82, N=54 (1024) 1.68 / 2.39, N=80 (592) 2.08 / 2.26,
// N=90 2.75 / 2.87, N=96 3.16 / 3.09, N=108 4.15 / 3.90. The mixed form needs the
// FP64 reduction for few pencils and keeps to house_rows up to kResidentMaxN
// (U over H, 592 pencils of N=108: 6.48 / 7.20).
__host__ __device__ constexpr bool tiled_rows(int n, bool mixed) { return n <= (mixed ? kResidentMaxN : 95); }
__host__ __device__ inline size_t tiled_work_elems(int n) { return tiled_part_elems(n) + tiled_ring_elems(n); }

__host__ __device__ inline size_t tiled_base_bytes(int n) {
    const size_t b = (size_t)n * 16 * 3 + 32 * 16 + 3 * 256 * 16 + (size_t)n * 8 * 3 + (size_t)dc_vec_doubles(n) * 8 +
                     (size_t)n * 4 + 8 * 4 + (size_t)dc_vec_ints(n) * 4;
    return (b + 15) & ~(size_t)15;
}

// The mixed form's FP32 copy of C in the same place, as long as two CTAs fit an
// SM (up to N = 103). N=54: the reduction takes 333 K cycles on a copy in global
// memory, 191 K here.
__host__ __device__ inline size_t tiled_c32_bytes(int n) { return ((size_t)n * (n | 1) * 8 + 15) & ~(size_t)15; }
__host__ __device__ inline bool tiled_keep32(int n) {
    return n <= kResidentMaxN && tiled_base_bytes(n) + tiled_c32_bytes(n) <= 112 * 1024;
}

__device__ inline TVec tcarve(unsigned char* p, int n) {
    TVec v;
    v.tau = reinterpret_cast<double2*>(p);
    v.vb  = v.tau + n;
    v.pb  = v.vb + n;
    v.red = v.pb + n;
    v.tb  = v.red + 32;
    v.gb  = v.tb + 256;
    v.d   = reinterpret_cast<double*>(v.gb + 512);
    v.e   = v.d + n;
    v.rdg = v.e + n;
    v.dcd = v.rdg + n;
    v.rank = reinterpret_cast<int*>(v.dcd + dc_vec_doubles(n));
    v.ctl  = v.rank + n;
    v.dci  = v.ctl + 8;
    v.part = reinterpret_cast<double2*>(p + tiled_base_bytes(n));
    v.ring = v.part + tiled_part_elems(n);
    return v;
}

__device__ __forceinline__ double2 cneg(double2 a) { return c2(-a.x, -a.y); }

// ---------------------------------------------------------------- 16x16 complex MMA tiles
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) { mma884(d, a, b); }

// A warp's 16 x 16 complex accumulator: 2 x 2 subtiles of 8 x 8, real and
// imaginary parts apart. Element [h][g][e] is row i0 + 8h + lane/4, column
// j0 + 8g + 2(lane%4) + e.
struct Z16 {
    double re[2][2][2];
    double im[2][2][2];
};

__device__ __forceinline__ void z16_zero(Z16& c) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int e = 0; e < 2; ++e) c.re[h][g][e] = c.im[h][g][e] = 0.0;
}

// f(i, j) -> double2 for every element of the tile at (i0, j0)
template <class F>
__device__ __forceinline__ void z16_load(Z16& c, int i0, int j0, F f) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const double2 x = f(i0 + 8 * h + (lane >> 2), j0 + 8 * g + 2 * (lane & 3) + e);
                c.re[h][g][e] = x.x;
                c.im[h][g][e] = x.y;
            }
}

// f(i, j, value) for every element of the tile at (i0, j0)
template <class F>
__device__ __forceinline__ void z16_store(const Z16& c, int i0, int j0, F f) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                f(i0 + 8 * h + (lane >> 2), j0 + 8 * g + 2 * (lane & 3) + e, c2(c.re[h][g][e], c.im[h][g][e]));
}

// One k step of 4: a = A fragments of rows r, r + 8, b = B fragments of columns r, r + 8.
__device__ __forceinline__ void z16_step(Z16& c, const double2 (&a)[2], const double2 (&b)[2]) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            dmma(c.re[h][g], a[h].x, b[g].x);
            dmma(c.re[h][g], -a[h].y, b[g].y);
            dmma(c.im[h][g], a[h].x, b[g].y);
            dmma(c.im[h][g], a[h].y, b[g].x);
        }
}

// c += A(i0:i0+16, k0:k1) B(k0:k1, j0:j0+16), A(i, k) at pa[i si + k sk], B(k, j)
// at pb[k tk + j tj], conjugated where CA / CB say so, A negated for NA. Rows and
// columns past ni, nj repeat the last one (they reach discarded results only);
// k blocks are unmasked but for the last, whose A is zeroed past k1.
template <bool CA, bool NA, bool CB>
__device__ __forceinline__ void z16_gemm(Z16& c, int i0, int j0, int k0, int k1, const double2* pa, int si, int sk, int ni,
                                         const double2* pb, int tk, int tj, int nj) {
    const int lane = threadIdx.x & 31;
    const int r = lane >> 2, kq = lane & 3;
    const double2* a0 = pa + (size_t)min(i0 + r, ni - 1) * si;
    const double2* a1 = pa + (size_t)min(i0 + r + 8, ni - 1) * si;
    const double2* b0 = pb + (size_t)min(j0 + r, nj - 1) * tj;
    const double2* b1 = pb + (size_t)min(j0 + r + 8, nj - 1) * tj;
    auto fix_a = [](double2 x) { return c2(NA ? -x.x : x.x, NA != CA ? -x.y : x.y); };
    auto fix_b = [](double2 x) { return c2(x.x, CB ? -x.y : x.y); };
    int k = k0;
#pragma unroll 4
    for (; k + 4 <= k1; k += 4) {
        const size_t ka = (size_t)(k + kq) * sk, kb = (size_t)(k + kq) * tk;
        const double2 a[2] = {fix_a(a0[ka]), fix_a(a1[ka])}, b[2] = {fix_b(b0[kb]), fix_b(b1[kb])};
        z16_step(c, a, b);
    }
    if (k < k1) {
        const bool in = k + kq < k1;
        const size_t ka = (size_t)min(k + kq, k1 - 1) * sk, kb = (size_t)min(k + kq, k1 - 1) * tk;
        double2 a[2] = {fix_a(a0[ka]), fix_a(a1[ka])};
        const double2 b[2] = {fix_b(b0[kb]), fix_b(b1[kb])};
        if (!in) a[0] = a[1] = c2(0.0, 0.0);
        z16_step(c, a, b);
    }
}

// Work order of tm x tn tiles: 4 x 4 blocks of tiles after one another, so that
// the warps of a CTA share 4 + 4 operand strips at a time. Returns false for a
// number past the edge (numbers run to tile_blocks(tm, tn)).
__device__ __forceinline__ int tile_blocks(int tm, int tn) { return ((tm + 3) >> 2) * ((tn + 3) >> 2) * 16; }
__device__ __forceinline__ bool tile_at(int t, int tm, int tn, int& ti, int& tj) {
    const int bn = (tn + 3) >> 2, blk = t >> 4, bi = blk / bn, bj = blk - bi * bn;
    ti = 4 * bi + ((t >> 2) & 3);
    tj = 4 * bj + (t & 3);
    return ti < tm && tj < tn;
}

// t -> (ti, tj) with ti >= tj, enumerating the lower triangle row by row.
__device__ __forceinline__ void tri_tile(int t, int& ti, int& tj) {
    int r = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((r + 1) * (r + 2) / 2 <= t) ++r;
    while (r * (r + 1) / 2 > t) --r;
    ti = r;
    tj = t - r * (r + 1) / 2;
}

// ---------------------------------------------------------------- back-transform
// Complex 8 x 8 x 4 step with four real ones.
__device__ __forceinline__ void z8_step(double (&re)[2], double (&im)[2], double2 a, double2 b) {
    dmma(re, a.x, b.x);
    dmma(re, -a.y, b.y);
    dmma(im, a.x, b.y);
    dmma(im, a.y, b.x);
}

// T factor of the compact WY form I - Y T Y^H of w reflectors (Y: rows k0 .. n,
// ones and zeros in place), forward column-wise: T(j, j) = tau_j, T(0:j, j) =
// -tau_j T(0:j, 0:j) (Y^H Y)(0:j, j). 16 x 16, zero past w, by one warp.
__device__ __forceinline__ void wy_factor(double2* tf, const double2* Y, int ld, int k0, int n, int w, const double2* tau) {
    const int lane = threadIdx.x & 31;
    Z16 acc;
    z16_zero(acc);
    z16_gemm<true, false, false>(acc, 0, 0, k0, n, Y, ld, 1, w, Y, 1, ld, w);
    z16_store(acc, 0, 0, [&](int i, int j, double2 x) { tf[i + 16 * j] = i < j && j < w ? x : c2(0.0, 0.0); });
    __syncwarp();
#pragma unroll 1
    for (int j = 0; j < w; ++j) {
        const double2 tj = tau[j];
        const double2 y = lane < j ? cneg(cmul(tj, tf[lane + 16 * j])) : c2(0.0, 0.0);
        double2 s = c2(0.0, 0.0);
#pragma unroll 2
        for (int l = 0; l < j; ++l) {
            const double2 yl = c2(__shfl_sync(0xffffffffu, y.x, l), __shfl_sync(0xffffffffu, y.y, l));
            if (lane <= l) s = cfma(s, tf[lane + 16 * l], yl);
        }
        if (lane < j) tf[lane + 16 * j] = s;
        if (lane == j) tf[j + 16 * j] = tj;
        __syncwarp();
    }
}

// V <- (I - Y1 T1 Y1^H) (I - Y2 T2 Y2^H) V on columns j0 .. j0 + 7 of V, by one
// warp; Y1: reflectors k0 .. k0 + 15, Y2: the next 16 (two: they exist).
// Worked on transposed, W^H = V^H Y, so that every accumulator is the next
// product's A fragment (in each k block of 8 the MMA's slot q of step s is
// index 2 q + s) and W stays in registers: nothing is shared, and the warps run
// through all blocks without a barrier. Two blocks at a time, because a strip
// of V is read twice and written once for each visit:
//   W2 = T2 Y2^H V, W1 = T1 (Y1^H V - (Y1^H Y2) W2), V -= Y1 W1 + Y2 W2.
// t1, t2: T factors, g12 = Y1^H Y2. Columns of Y past nref repeat the last one
// (finite, and T is zero there); rows above a reflector are zero in Y.
// Bound by the loads of V and Y from L2. N=216, the whole back-transform:
// 2.06 M cycles block by block over all of V with five barriers each, 1.65 M
// here; strips of 16 columns spill and are slower (N=384: 5 % of the solve).
__device__ __forceinline__ void wy_strip(double2* V, int n, int j0, const double2* Y, int ld, int k0, int nref, bool two,
                                         const double2* t1, const double2* t2, const double2* g12) {
    const int lane = threadIdx.x & 31, fr = lane >> 2, fq = lane & 3;
    double wr[2][2][2], wi[2][2][2];               // W^H of both blocks: column tiles of 8
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int h = 0; h < 2; ++h) wr[b][h][0] = wr[b][h][1] = wi[b][h][0] = wi[b][h][1] = 0.0;
    const bool col = j0 + fr < n;
    double2* vj = V + (size_t)min(j0 + fr, n - 1) * n;
    const double2* yc[4];                          // columns of Y as right-hand operands
#pragma unroll
    for (int h = 0; h < 4; ++h) yc[h] = Y + (size_t)min(k0 + 8 * h + fr, nref - 1) * ld;
#pragma unroll 1
    for (int i0 = k0; i0 < n; i0 += 8) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int i = i0 + 2 * fq + s, ic = min(i, n - 1);
            double2 a = cconj(vj[ic]), y[4];
            if (i >= n) a = c2(0.0, 0.0);
#pragma unroll
            for (int h = 0; h < 4; ++h) if (h < 2 || two) y[h] = yc[h][ic];
#pragma unroll
            for (int h = 0; h < 4; ++h) if (h < 2 || two) z8_step(wr[h >> 1][h & 1], wi[h >> 1][h & 1], a, y[h]);
        }
    }
    // out += sgn w m^H, m a 16 x 16 matrix (upper triangular if tri)
    auto times = [&](double (&outr)[2][2], double (&outi)[2][2], const double (&r)[2][2], const double (&im)[2][2],
                     const double2* m, double sgn, bool tri) {
#pragma unroll
        for (int h = 0; h < 2; ++h)                // k block (column of m)
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int g = 0; g < 2; ++g) {      // column tile (row of m)
                    if (tri && g > h) continue;
                    const double2 bv = cconj(m[8 * g + fr + 16 * (8 * h + 2 * fq + s)]);
                    z8_step(outr[g], outi[g], c2(sgn * r[h][s], sgn * im[h][s]), bv);
                }
    };
    auto apply_t = [&](double (&r)[2][2], double (&im)[2][2], const double2* m) {
        double nr[2][2] = {}, ni[2][2] = {};
        times(nr, ni, r, im, m, 1.0, true);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                r[h][e] = nr[h][e];
                im[h][e] = ni[h][e];
            }
    };
    if (two) {
        apply_t(wr[1], wi[1], t2);
        times(wr[0], wi[0], wr[1], wi[1], g12, -1.0, false);
    }
    apply_t(wr[0], wi[0], t1);
    const int ce = nref - 1 - k0;                  // last column of Y, from k0
#pragma unroll 1
    for (int i0 = k0; i0 < n; i0 += 8) {
        double vr[2], vi[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const double2 x = vj[min(i0 + 2 * fq + e, n - 1)];
            vr[e] = x.x;
            vi[e] = x.y;
        }
        const double2* yi = Y + (size_t)k0 * ld + min(i0 + fr, n - 1);
#pragma unroll
        for (int h = 0; h < 4; ++h)
            if (h < 2 || two)
#pragma unroll
                for (int s = 0; s < 2; ++s)
                    z8_step(vr, vi, c2(-wr[h >> 1][h & 1][s], wi[h >> 1][h & 1][s]),
                            yi[(size_t)min(8 * h + 2 * fq + s, ce) * ld]);
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (col && i0 + 2 * fq + e < n) vj[i0 + 2 * fq + e] = c2(vr[e], vi[e]);
    }
    __syncwarp();
}

// V <- Q V, Q the product of the nref reflectors in Y. tf: room for the T
// factors and, of each pair of blocks, Y1^H Y2, 256 elements each.
template <int kNT>
__device__ __forceinline__ void wy_apply(double2* V, int n, const double2* Y, int ld, int nref, const double2* tau,
                                             double2* tf) {
    constexpr int kNW = kNT / 32;
    const int warp = threadIdx.x >> 5;
    const int nblk = (nref + 15) >> 4, npair = (nblk + 1) >> 1;
    double2* g12 = tf + 256 * nblk;
#pragma unroll 1
    for (int t = warp; t < nblk + (nblk >> 1); t += kNW) {
        if (t < nblk) {
            wy_factor(tf + 256 * t, Y + (size_t)16 * t * ld, ld, 16 * t + 1, n, min(16, nref - 16 * t), tau + 16 * t);
        } else {
            const int p = t - nblk, kb = 32 * p + 16, w = min(16, nref - kb);
            Z16 acc;
            z16_zero(acc);
            z16_gemm<true, false, false>(acc, 0, 0, kb + 1, n, Y + (size_t)(kb - 16) * ld, ld, 1, 16,
                                         Y + (size_t)kb * ld, 1, ld, w);
            z16_store(acc, 0, 0, [&](int i, int j, double2 x) { g12[256 * p + i + 16 * j] = x; });
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int j0 = 8 * warp; j0 < n; j0 += 8 * kNW)
#pragma unroll 1
        for (int p = npair - 1; p >= 0; --p) {
            const double2 *t1 = tf + 512 * p, *t2 = t1 + 256, *g = g12 + 256 * p;
            const bool two = 2 * p + 1 < nblk;
            wy_strip(V, n, j0, Y, ld, 32 * p, nref, two, t1, t2, g);
        }
}

// The divide and conquer with a register allocation of its own: inlined, it
// made the tile products around it spill (n = 216: 4 % slower).
template <int kNT>
static __device__ __noinline__ void tiled_dc(int n, DCShared dc) { tridiag_dc<kNT, 0>(n, dc); }

// How y = A v over rows and columns lo .. n-1 is dealt to the warps: blocks of
// kMvRows rows, counted from the last row up, each with a share of the warps
// in proportion to its elements (first[q] .. first[q + 1] - 1 for block q).
struct MatvecSplit {
    int first[5];
};
template <int NW>
__device__ __forceinline__ MatvecSplit matvec_split(int n, int lo) {
    const int m = n - lo, nq = (m + kMvRows - 1) / kMvRows;
    MatvecSplit s;
    float total = 0.0f, sum = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) if (q < nq) total += (float)(m - kMvRows * q);
    s.first[0] = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q < nq) sum += (float)(m - kMvRows * q);
        // at least one warp for each block
        const int f = (int)(NW * sum / total + 0.5f);
        s.first[q + 1] = q + 1 >= nq ? NW : min(max(f, s.first[q] + 1), NW - (nq - 1 - q));
    }
    return s;
}

// y = A v for the Hermitian trailing matrix A kept in its lower triangle, v zero
// below lo. A warp has a block of rows, four per lane, and every G-th column j
// of it, and gets from each element both halves of the product: y_i += A(i, j)
// v_j for i > j (in registers, to part at the end) and y_j = sum_{i >= j}
// conj(A(i, j)) v_i (each block's share to ydot[block]). The elements come
// through shared memory by asynchronous copies, kMvDepth columns ahead; a lane
// reads what it copied itself, so nothing but its own copies is waited for.
// N=216, cycles per column: 18.4 K for the full matrix column by column with
// two pencils per SM, 17.6 K with one column ahead in registers (one pencil of
// 512 threads): the loads' latency, with some 30 KB in flight per SM.
template <int kNT>
__device__ __forceinline__ void sym_matvec(const double2* A, int ld, int n, int lo, const double2* vb, double2* part,
                                           double2* const (&ydot)[4], double2* ring) {
    constexpr int NW = kNT / 32, RB = kMvRows / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const MatvecSplit ms = matvec_split<NW>(n, lo);
    int q = 0;
#pragma unroll
    for (int u = 1; u < 4; ++u) if (warp >= ms.first[u]) q = u;
    int f = 0, G = 0;
    double2* yd = nullptr;
#pragma unroll
    for (int u = 0; u < 4; ++u) if (q == u) { f = ms.first[u]; G = ms.first[u + 1] - f; yd = ydot[u]; }
    const int r1 = n - kMvRows * q, r0 = max(lo, r1 - kMvRows), g = warp - f;
    double2 v[RB], y[RB];
#pragma unroll
    for (int t = 0; t < RB; ++t) {
        const int i = r0 + lane + 32 * t;
        v[t] = i < r1 ? vb[i] : c2(0.0, 0.0);
        y[t] = c2(0.0, 0.0);
    }
    const unsigned dst = (unsigned)__cvta_generic_to_shared(ring + threadIdx.x);
    auto fetch = [&](int j, int stage) {
        if (j < r1) {
            const double2* cj = A + (size_t)j * ld + r0 + lane;
#pragma unroll
            for (int t = 0; t < RB; ++t) {
                const int i = r0 + lane + 32 * t;
                if (i >= j && i < r1)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                 :: "r"(dst + (unsigned)((stage * RB + t) * kNT * 16)), "l"(cj + 32 * t) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int u = 0; u < kMvDepth - 1; ++u) fetch(lo + g + u * G, u);
    int stage = 0;
#pragma unroll 1
    for (int j = lo + g; j < r1; j += G) {
        fetch(j + (kMvDepth - 1) * G, stage == 0 ? kMvDepth - 1 : stage - 1);
        asm volatile("cp.async.wait_group %0;" :: "n"(kMvDepth - 1) : "memory");
        const double2* x = ring + stage * RB * kNT + threadIdx.x;
        const double2 vj = vb[j];
        double2 dot = c2(0.0, 0.0);
#pragma unroll
        for (int t = 0; t < RB; ++t) {
            const int i = r0 + lane + 32 * t;
            if (r0 + 32 * t + 31 < j || r0 + 32 * t >= r1) continue;
            const double2 e = x[t * kNT];
            const bool in = i >= j && i < r1;
            const double2 z = c2(in ? e.x : 0.0, in ? e.y : 0.0);
            dot = cfmac(dot, z, v[t]);
            if (i != j) y[t] = cfma(y[t], z, vj);                    // the diagonal belongs to the dot
        }
        dot = warp_sum2(dot);
        if (lane == 0) yd[j] = dot;
        stage = stage == kMvDepth - 1 ? 0 : stage + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int t = 0; t < RB; ++t) part[warp * kMvRows + lane + 32 * t] = y[t];
}

// Element i of that product, after a barrier.
template <int kNT>
__device__ __forceinline__ double2 sym_matvec_row(int n, int lo, int i, const double2* part, double2* const (&ydot)[4]) {
    const MatvecSplit ms = matvec_split<kNT / 32>(n, lo);
    const int q = (n - 1 - i) / kMvRows, r0 = max(lo, n - kMvRows * (q + 1));
    double2 y = c2(0.0, 0.0);
    int f = 0, e = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (u <= q) y = cadd(y, ydot[u][i]);     // this block and those below it
        if (u == q) { f = ms.first[u]; e = ms.first[u + 1]; }
    }
#pragma unroll 4
    for (int w = f; w < e; ++w) y = cadd(y, part[w * kMvRows + i - r0]);
    return y;
}

// Sum over the CTA: every thread gets the value; red holds threads/32 entries
// that no other sum since the last barrier has used.
template <int kNT>
__device__ __forceinline__ double cta_sum(double x, double* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    x = warp_sum(x);
    if (lane == 0) red[warp] = x;
    __syncthreads();
    return warp_sum(lane < kNT / 32 ? red[lane] : 0.0);
}

// X = L^-1 -> M1, block row r0..re at a time; zeros above its diagonal, so that
// the products need no masks.
template <int kNT>
__device__ __forceinline__ void tiled_inverse(int n, int ld, const double2* M0, double2* M1, const double* rdg) {
    constexpr int kNW = kNT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double2 zero = c2(0.0, 0.0);
    for (int j = warp; j < n; j += kNW)
        for (int i = lane; i < j; i += 32) M1[i + (size_t)j * ld] = zero;
    for (int r0 = 0; r0 < n; r0 += 16) {
        const int re = min(r0 + 16, n);
        for (int t = warp; t < (r0 >> 4); t += kNW) {
            const int j0 = 16 * t;
            Z16 acc;
            z16_zero(acc);
            z16_gemm<false, false, false>(acc, r0, j0, j0, r0, M0, 1, ld, n, M1, 1, ld, n);
            z16_store(acc, r0, j0, [&](int i, int j, double2 x) { if (i < n) M1[i + (size_t)j * ld] = x; });
        }
        __syncthreads();
        for (int c = tid; c < re; c += kNT) {
            double2 x[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int i = r0 + r;
                x[r] = (i < re) ? ((c < r0) ? cneg(M1[i + (size_t)c * ld]) : c2(i == c ? 1.0 : 0.0, 0.0))
                                : zero;
            }
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int i = r0 + r;
                if (i < re) {
                    double2 s = x[r];
#pragma unroll
                    for (int q = 0; q < r; ++q) s = cfms(s, M0[i + (size_t)(r0 + q) * ld], x[q]);
                    x[r] = cscale(s, rdg[i]);
                }
            }
#pragma unroll
            for (int r = 0; r < 16; ++r)
                if (r0 + r < re) M1[r0 + r + (size_t)c * ld] = x[r];
        }
        __syncthreads();
    }
}

// T = H X^H -> M2, T(i, j) = sum_{k <= j} H(i, k) conj(X(j, k)), then C = X T -> M0.
template <int kNT>
__device__ __forceinline__ void tiled_form_c(int n, int ld, int sigma, const double2* Hb, double2* M0, const double2* M1,
                                                 double2* M2) {
    constexpr int kNW = kNT / 32;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int tn = (n + 15) >> 4;
    const size_t nn = (size_t)n * n;
    const double2 zero = c2(0.0, 0.0);
    if (sigma) {
        const int m = n >> 1;
        for (int idx = tid; idx < (int)nn; idx += kNT) {
            const int j = idx / n, i = idx - j * n;
            const double2 x = (i <= j) ? cconj(M1[j + (size_t)i * ld]) : zero;
            M2[i + (size_t)j * ld] = (i < m) ? x : cneg(x);
        }
    } else {
        for (int t = warp; t < tile_blocks(tn, tn); t += kNW) {
            int ti, tj;
            if (!tile_at(t, tn, tn, ti, tj)) continue;
            const int i0 = 16 * ti, j0 = 16 * tj;
            Z16 acc;
            z16_zero(acc);
            z16_gemm<false, false, true>(acc, i0, j0, 0, min(n, j0 + 16), Hb, 1, n, n, M1, ld, 1, n);
            z16_store(acc, i0, j0, [&](int i, int j, double2 x) {
                if (i < n && j < n) M2[i + (size_t)j * ld] = x;
            });
        }
    }
    __syncthreads();
    // C = X T, lower tiles; each lower element is written with its
    // mirror so that C is exactly Hermitian. L in M0 is dead by now.
    for (int t = warp; t < tile_blocks(tn, tn); t += kNW) {
        int ti, tj;
        if (!tile_at(t, tn, tn, ti, tj) || ti < tj) continue;
        const int i0 = 16 * ti, j0 = 16 * tj;
        Z16 acc;
        z16_zero(acc);
        z16_gemm<false, false, false>(acc, i0, j0, 0, min(n, i0 + 16), M1, 1, ld, n, M2, 1, ld, n);
        z16_store(acc, i0, j0, [&](int i, int j, double2 x) {
            if (i < n && j < n && i >= j) {
                if (i == j) x.y = 0.0;
                M0[i + (size_t)j * ld] = x;
                M0[j + (size_t)i * ld] = cconj(x);
            }
        });
    }
    __syncthreads();
}

// A reflector whose squares leave the range, from the column's elements x[lo .. n)
// in shared memory, by every warp for itself; out of line to keep the caller's
// registers (n = 216: 1 % of the solve).
static __device__ __noinline__ Reflector column_out_of_range(const double2* x, int lo, int n, double2 alpha, double nn) {
    const double f = column_scale(nn);
    double ss = 0.0;
    for (int i = lo + (int)(threadIdx.x & 31); i < n; i += 32) {
        const double2 y = cscale(x[i], f);
        ss = fma(y.x, y.x, fma(y.y, y.y, ss));
    }
    const double2 as = cscale(alpha, f);
    return reflector_scaled(alpha, as, fma(as.y, as.y, warp_sum(ss)), f);
}

// The FP64 reduction of C (lower, M0) to tridiagonal form, reflectors in its
// columns, (d, e, tau) to shared memory.
template <int kNT>
__device__ __forceinline__ void tiled_house(int n, int ld, double2* M0, double2* M2, unsigned char* smem_raw) {
    constexpr int kNW = kNT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double2 zero = c2(0.0, 0.0);
    const TVec v = tcarve(smem_raw, n);
    // thread i owns row i of the vectors and of the panel (kNT >= n)
    // V and W of the panel: columns Vp + c ld, Wp + c ld
    double2* Wp = M2;
    const int i = tid;
    const bool row = i < n;
    double* red = reinterpret_cast<double*>(v.red);   // 32 doubles for each of two sums
    double2* t12 = v.tb;                               // W^H v at [0, c), V^H v at [16, 16 + c)
    // (the divide and conquer's scratch is free until then: 2 n complex of its 7 n + 1 doubles)
    double2* yx = reinterpret_cast<double2*>(v.dcd + (n & 1));
    double2* const ydot[4] = {v.pb, v.gb, yx, yx + n};
    for (int p = 0; p < n - 1; p += 16) {
        const int w = min(16, n - 1 - p);
        double2* Vp = M0 + (size_t)p * ld;
        for (int c = 0; c < w; ++c) {
            const int k = p + c;
            // (1) column k of the current matrix:
            // a_k -= V(:, 0:c) W(k, 0:c)^H + W(:, 0:c) V(k, 0:c)^H
            // (rows k .. n-1 of V are stored whole)
            double2 x = zero;
            if (row && i >= k) {
                x = M0[i + (size_t)k * ld];
#pragma unroll 4
                for (int cc = 0; cc < c; ++cc) {
                    x = cfms_bc(x, Vp[i + cc * ld], Wp[k + cc * ld]);
                    x = cfms_bc(x, Wp[i + cc * ld], Vp[k + cc * ld]);
                }
            }
            if (i == k) { v.d[k] = x.x; M0[k + (size_t)k * ld] = x; }
            if (i == k + 1) v.gb[0] = x;
            // (2) reflector from a_k(k+1:n)
            const double ss = cta_sum<kNT>((row && i > k + 1) ? fma(x.x, x.x, x.y * x.y) : 0.0, red);
            const double2 alpha = v.gb[0];
            const double rest = fma(alpha.y, alpha.y, ss), nn = fma(alpha.x, alpha.x, rest);
            Reflector refl;                                // the same in every thread
            if (squares_safe(rest, nn)) {
                refl = reflector(alpha, nn);
            } else {
                if (row) v.vb[i] = x;
                __syncthreads();
                refl = column_out_of_range(v.vb, k + 2, n, alpha, nn);
                __syncthreads();
            }
            const double2 taui = refl.tau;
            double2 vi = zero;
            if (row && i > k) {
                vi = i == k + 1 ? c2(1.0, 0.0) : cmul(x, refl.scal);
                v.vb[i] = vi;
                M0[i + (size_t)k * ld] = vi;
            }
            if (tid == 0) { v.tau[k] = taui; v.e[k] = refl.beta; }
            __syncthreads();
            // (3) y = A v (A: panel-start trailing matrix, lower
            // triangle), t1 = W^H v, t2 = V^H v
            sym_matvec<kNT>(M0, ld, n, k + 1, v.vb, v.part, ydot, v.ring);
            for (int it = warp; it < 2 * c; it += kNW) {
                const int cc = it >> 1;
                double2 acc = zero;
                const double2* col = (it & 1 ? Vp : Wp) + cc * ld;
#pragma unroll 4
                for (int j = k + 1 + lane; j < n; j += 32) acc = cfmac(acc, col[j], v.vb[j]);
                acc = warp_sum2(acc);
                if (lane == 0) t12[16 * (it & 1) + cc] = acc;
            }
            __syncthreads();
            // (4) w = tau (y - V t1 - W t2) + alpha2 v on rows k+1..n (the
            // current matrix is A - V W^H - W V^H), alpha2 =
            // -tau/2 (w^H v) = -|tau|^2/2 v^H A v; zero above
            double2 y = zero;
            if (row && i > k) {
                y = sym_matvec_row<kNT>(n, k + 1, i, v.part, ydot);
#pragma unroll 4
                for (int cc = 0; cc < c; ++cc) {
                    y = cfms(y, Vp[i + cc * ld], t12[cc]);
                    y = cfms(y, Wp[i + cc * ld], t12[16 + cc]);
                }
            }
            const double h = -0.5 * fma(taui.x, taui.x, taui.y * taui.y) *
                             cta_sum<kNT>(fma(y.x, vi.x, y.y * vi.y), red + 32);
            if (row) {
                const double2 wt = cmul(taui, y);
                Wp[i + c * ld] = c2(fma(h, vi.x, wt.x), fma(h, vi.y, wt.y));
            }
            __syncthreads();
        }
        // trailing update, lower tiles: A(q:n, q:n) -= V W^H + W V^H, q = p + w
        const int q = p + w, mq = n - q;
        if (mq > 0) {
            const int tq = (mq + 15) >> 4;
            for (int t = warp; t < tile_blocks(tq, tq); t += kNW) {
                int ti, tj;
                if (!tile_at(t, tq, tq, ti, tj) || ti < tj) continue;
                const int i0 = q + 16 * ti, j0 = q + 16 * tj;
                Z16 acc;
                z16_load(acc, i0, j0, [&](int r, int j) { return (r < n && j < n) ? M0[r + (size_t)j * ld] : zero; });
                z16_gemm<false, true, true>(acc, i0, j0, 0, w, Vp, 1, ld, n, Wp, ld, 1, n);
                z16_gemm<false, true, true>(acc, i0, j0, 0, w, Wp, 1, ld, n, Vp, ld, 1, n);
                z16_store(acc, i0, j0, [&](int r, int j, double2 x) {
                    if (r < n && j < n && r >= j) M0[r + (size_t)j * ld] = x;
                });
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        v.d[n - 1] = M0[(n - 1) + (size_t)(n - 1) * ld].x;
        if (n == 1) v.tau[0] = zero;
    }
    __syncthreads();
}

// The same names for both precisions.
__device__ __forceinline__ float2 xmul(float2 a, float2 b) { return fcmul(a, b); }
__device__ __forceinline__ double2 xmul(double2 a, double2 b) { return cmul(a, b); }
__device__ __forceinline__ float2 xfma(float2 acc, float2 a, float2 b) { return fcfma(acc, a, b); }
__device__ __forceinline__ double2 xfma(double2 acc, double2 a, double2 b) { return cfma(acc, a, b); }
__device__ __forceinline__ float2 xfms_bc(float2 acc, float2 a, float2 b) { return fcfms_bc(acc, a, b); }
__device__ __forceinline__ double2 xfms_bc(double2 acc, double2 a, double2 b) { return cfms_bc(acc, a, b); }
__device__ __forceinline__ float xfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double xfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float xsum(float v) { return warp_sumf(v); }
__device__ __forceinline__ double xsum(double v) { return warp_sum(v); }
__device__ __forceinline__ double2 widen(float2 a) { return f2d(a); }
__device__ __forceinline__ double2 widen(double2 a) { return a; }
template <class T2> __device__ __forceinline__ T2 xshfl(T2 v, int src) {
    v.x = __shfl_sync(0xffffffffu, v.x, src);
    v.y = __shfl_sync(0xffffffffu, v.y, src);
    return v;
}

// Reflector from a column (alpha, x) whose elements, x from row lo on, the lanes
// hold and `column` has room for; ss = ||x||^2.
__device__ __forceinline__ void column_reflector(float2 alpha, float ss, float2& tau, float2& scal, float& beta) {
    tau = scal = f2(0.0f, 0.0f);
    beta = alpha.x;
    if (!(ss == 0.0f && alpha.y == 0.0f)) {
        beta = -copysignf(sqrtf(alpha.x * alpha.x + alpha.y * alpha.y + ss), alpha.x);
        tau = f2((beta - alpha.x) / beta, -alpha.y / beta);
        const float2 z = f2(alpha.x - beta, alpha.y);
        const float inv = 1.0f / (z.x * z.x + z.y * z.y);
        scal = f2(z.x * inv, -z.y * inv);
    }
}
template <class Store>
__device__ __forceinline__ void column_reflector(double2 alpha, double ss, double2& tau, double2& scal, double& beta,
                                                 const double2* column, int lo, int n, Store store) {
    const double rest = fma(alpha.y, alpha.y, ss), nn = fma(alpha.x, alpha.x, rest);
    Reflector h;
    if (squares_safe(rest, nn)) {
        h = reflector(alpha, nn);
    } else {
        store();
        __syncwarp();
        h = column_out_of_range(column, lo, n, alpha, nn);
        __syncwarp();
    }
    tau = h.tau;
    scal = h.scal;
    beta = h.beta;
}

// The reduction of a small C to tridiagonal form (n <= 128) by the smem-cta
// kernel's scheme: per step one warp forms w and the next reflector from the
// partial products, then every warp, over its block of 32 rows and its class of
// columns, applies A -= v w^H + w v^H and multiplies the updated elements by the
// new reflector in the same pass. Two barriers a step. The mixed form runs it on
// the FP32 copy of C (in shared memory), the FP64 form on C in the slot
// (tiled_rows). Reflectors stay in A's columns; tau, d, e in FP64. part: 32 values
// per warp, vb: 2 n, wb: n.
template <int kNT, class T2>
__device__ __forceinline__ void house_rows(int n, int ld, T2* A, T2* part, T2* vb, T2* wb, double2* tauv, double* dv,
                                           double* ev) {
    using T = decltype(T2::x);
    constexpr int NW = kNT / 32, R = 4;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int last = n - 1 - lane;                 // row of block t: last - 32 t
    const T2 zero{0, 0}, one{1, 0};
    for (int i = tid; i < n; i += kNT) vb[n + i] = wb[i] = zero;
    __syncthreads();
    int rb = 0, G = 0, myt = 0, myg = 0;
    T2 tau = zero;                                 // of reflector c - 1
#pragma unroll 1
    for (int c = 0; c < n; ++c) {
        const T2* vk = vb + ((c + 1) & 1) * n;
        T2* vc = vb + (c & 1) * n;
        if (warp == 0) {
            T2 x[R], w[R];
            T2* mc = A + c * ld;
            const int ic = n - 1 - c;              // slot of row c
#pragma unroll
            for (int t = 0; t < R; ++t) x[t] = mc[max(last - 32 * t, 0)];
            if (c > 0) {
                T2 v[R];
                T s = 0;
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    v[t] = vk[max(last - 32 * t, 0)];
                    w[t] = zero;
                }
                const T2* pt = part + lane;
#pragma unroll 2
                for (int g = 0; g < G; ++g, pt += 32 * rb)
#pragma unroll
                    for (int t = 0; t < R; ++t)
                        if (t < rb) { w[t].x += pt[32 * t].x; w[t].y += pt[32 * t].y; }
#pragma unroll
                for (int t = 0; t < R; ++t) s = xfma(w[t].x, v[t].x, xfma(w[t].y, v[t].y, s));
                const T h = T(-0.5) * xfma(tau.x, tau.x, tau.y * tau.y) * xsum(s);
                T2 wc = zero;
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    w[t] = xmul(tau, w[t]);
                    w[t].x = xfma(h, v[t].x, w[t].x);
                    w[t].y = xfma(h, v[t].y, w[t].y);
                    if (last - 32 * t >= 0) wb[last - 32 * t] = w[t];
                    if ((ic >> 5) == t) wc = w[t];
                }
                wc = xshfl(wc, ic & 31);
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    x[t] = xfms_bc(x[t], v[t], wc);
                    x[t].x -= w[t].x;                                    // v(c) = 1
                    x[t].y -= w[t].y;
                }
            }
            T2 xc = x[0], alpha = x[0];
#pragma unroll
            for (int t = 1; t < R; ++t) {
                if ((ic >> 5) == t) xc = x[t];
                if (((ic - 1) >> 5) == t) alpha = x[t];
            }
            T beta = 0;
            if (c < n - 1) {
                alpha = xshfl(alpha, (ic - 1) & 31);
                T ss = 0;
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    if (last - 32 * t <= c + 1) x[t] = zero;
                    ss = xfma(x[t].x, x[t].x, xfma(x[t].y, x[t].y, ss));
                }
                ss = xsum(ss);
                T2 scal;
                if constexpr (sizeof(T) == 8) {
                    column_reflector(alpha, ss, tau, scal, beta, vc, c + 2, n, [&]() {
#pragma unroll
                        for (int t = 0; t < R; ++t) if (last - 32 * t >= 0) vc[last - 32 * t] = x[t];
                    });
                } else {
                    column_reflector(alpha, ss, tau, scal, beta);
                }
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    const int i = last - 32 * t;
                    x[t] = xmul(x[t], scal);
                    if (i >= 0) vc[i] = i == c + 1 ? one : x[t];
                    if (i > c + 1) mc[i] = x[t];
                }
                if (lane == 0) tauv[c] = widen(tau);
            }
            if (lane == (ic & 31)) {
                dv[c] = (double)xc.x;
                if (c < n - 1) ev[c] = (double)beta;
            }
        }
        if (c >= n - 1) break;
        __syncthreads();
        if (const int r = (n - 1 - c + 31) >> 5; r != rb) {
            rb = r;
            G = NW / rb;
            myg = warp / rb;
            myt = warp - myg * rb;
        }
        if (myg < G) {
            const int i = last - 32 * myt, o = max(i, 0);
            const T2 vi = vk[o], wi = wb[o];
            T2 y = zero;
#pragma unroll 4
            for (int j = c + 1 + myg; j < n; j += G) {
                T2* q = A + o + j * ld;
                const T2 z = xfms_bc(xfms_bc(*q, vi, wb[j]), wi, vk[j]);
                if (i >= 0) *q = z;
                y = xfma(y, z, vc[j]);
            }
            part[32 * (myg * rb + myt) + lane] = y;
        }
        __syncthreads();
    }
    if (n == 1 && tid == 0) tauv[0] = c2(0.0, 0.0);
    __syncthreads();
}

// One pencil b, solved end to end by the whole CTA in its global-memory
// slot `slot` (tiled_slot_elems(n, mixed) complex entries) with the
// launch's dynamic shared memory as the vector area. kNT >= n.
// MIXED: FP32 Householder reduction + FP64 refinement, an instance of its own
// so that the FP64 form does not carry its pointers (n = 216: 1.6 %).
// ROWS: tiled_rows(n, MIXED), the FP64 reduction is house_rows.
template <int kNT, bool MIXED, bool ROWS>
__device__ SGEIG_TILED_BODY_INLINE void tiled_solve(const TiledArgs& a, long long b, double2* slot,
                                            unsigned char* smem_raw) {
    constexpr int kNW = kNT / 32;
    const int n = a.n, ld = a.ld;
    const size_t mat = (size_t)n * ld;
    constexpr bool mixed = MIXED;
    double2* M0 = slot;
    double2* M1 = M0 + mat;
    double2* M2 = M1 + mat;
    double2* M3 = mixed ? M2 + mat : nullptr;       // mixed only
    double2* zob = mixed ? M3 + mat : M2 + mat;
    double*  Zo = reinterpret_cast<double*>(zob);
    // mixed only: FP32 copy of C after Zo; after the back-transform Zo and
    // it together hold one more n x ld complex matrix (M4)
    double2* M4 = zob;
    TVec v = tcarve(smem_raw, n);
    float2*  C32s = reinterpret_cast<float2*>(v.part);             // a.keep32
    float2*  C32 = reinterpret_cast<float2*>(zob + tiled_zo_elems(n));

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tn = (n + 15) >> 4;
    const size_t nn = (size_t)n * n;
    const double2 zero = c2(0.0, 0.0);
    const double2* Hb = a.H + (size_t)b * nn;
    const double2* Sb = a.S + (size_t)b * nn;
    double*  Wb = a.W + (size_t)b * n;
    double2* Ub = a.U + (size_t)b * nn;

    __syncthreads();  // previous pencil fully consumed
    phase_mark(24);
    // ---- a1: S (lower triangle and diagonal) -> M0
    for (int idx = tid; idx < (int)nn; idx += kNT) {
        const int j = idx / n, i = idx - j * n;
        if (i >= j) M0[i + (size_t)j * ld] = __ldg(Sb + idx);
    }
    if (tid < 8) v.ctl[tid] = 0;
    __syncthreads();
    phase_mark(16);

    // ---- a2: blocked Cholesky (lower). The pivot test is the same as
    // potrf's (not > 0, NaN included), taken in column order.
    int fail = 0;
    for (int p = 0; p < n && !fail; p += 16) {
        const int pe = min(p + 16, n);
        for (int c = p; c < pe; ++c) {
            const double piv = M0[c + (size_t)c * ld].x;
            if (!(piv > 0.0)) { fail = c + 1; break; }
            const double lc = sqrt(piv), r = 1.0 / lc;
            double2* lcol = M0 + (size_t)c * ld;
            for (int i = c + 1 + tid; i < n; i += kNT) lcol[i] = cscale(lcol[i], r);
            __syncthreads();
            if (tid == 0) { lcol[c] = c2(lc, 0.0); v.rdg[c] = r; }
            // rank-1 update of the panel columns right of c
            const int wc = pe - c - 1, rows = n - c - 1;
            for (int idx = tid; idx < rows * wc; idx += kNT) {
                const int cc = c + 1 + idx / rows, i = c + 1 + idx % rows;
                if (i >= cc) {
                    double2* x = M0 + i + (size_t)cc * ld;
                    *x = cfms_bc(*x, lcol[i], lcol[cc]);
                }
            }
            __syncthreads();
        }
        if (fail) break;
        // trailing lower tiles: C -= L_p L_p^H over columns [p, pe)
        const int m2 = n - pe;
        if (m2 > 0) {
            const int tm = (m2 + 15) >> 4, T = tm * (tm + 1) / 2;
            for (int t = warp; t < T; t += kNW) {
                int ti, tj;
                tri_tile(t, ti, tj);
                const int i0 = pe + 16 * ti, j0 = pe + 16 * tj;
                Z16 acc;
                z16_load(acc, i0, j0, [&](int i, int j) { return (i < n && j < n) ? M0[i + (size_t)j * ld] : zero; });
                z16_gemm<false, true, true>(acc, i0, j0, p, pe, M0, 1, ld, n, M0, ld, 1, n);
                z16_store(acc, i0, j0, [&](int i, int j, double2 x) {
                    if (i < n && j < n && i >= j) M0[i + (size_t)j * ld] = x;
                });
            }
        }
        __syncthreads();
    }
    int code = fail ? n + fail : 0;   // zhegv: info = n + order of the failing minor
    phase_mark(17);

    if (!code && a.stage >= 2) {
        // ---- a3: X = L^-1 -> M1
        tiled_inverse<kNT>(n, ld, M0, M1, v.rdg);
        phase_mark(18);
    }

    if (!code && a.stage == 1) {
        for (int idx = tid; idx < (int)nn; idx += kNT) {
            const int j = idx / n, i = idx - j * n;
            Ub[idx] = (i >= j) ? M0[i + (size_t)j * ld] : zero;
        }
        if (tid == 0) a.info[b] = 0;
        return;
    }

    if (!code) {
        // ---- a4: C = X H X^H -> M0
        tiled_form_c<kNT>(n, ld, a.sigma, Hb, M0, M1, M2);
        phase_mark(19);
    }

    if (!code && a.stage == 2) {
        for (int idx = tid; idx < (int)nn; idx += kNT) {
            const int j = idx / n, i = idx - j * n;
            Ub[idx] = M0[i + (size_t)j * ld];
        }
        if (tid == 0) a.info[b] = 0;
        return;
    }

    // The mixed form tries the FP32 reduction first; a pencil whose
    // refinement does not converge goes round once more in FP64.
    bool use32 = mixed;
    for (;;) {
        if (!code) {
            // ---- a5a: Householder tridiagonalisation of C (lower). Reflector
            // k: I - tau_k v v^H on rows k+1.., v[k+1] = 1, stored in column k
            // of M0 from row k+1 on. Blocked as LAPACK's zhetrd/zlatrd: panels
            // of up to 16 columns reduced against the panel-start trailing
            // matrix A with the corrections of the panel's earlier columns
            // (V = reflectors, W = their update vectors, W kept in M2 whose
            // product T is dead by now), then A -= V W^H + W V^H on
            // tensor-core tiles. Only the lower triangle is read and written.
            if (use32) {
                // Mixed form: the unblocked reduction in FP32 on a
                // single-precision copy of C (reflectors kept in its columns;
                // tau, d, e widened to FP64). C itself stays in M0 for the
                // refinement. The vectors live in pb's storage as float2.
                for (int j = warp; j < n; j += kNW)
                    for (int i = lane; i < n; i += 32) {
                        const double2 x = M0[i + (size_t)j * ld];
                        const float2 f = f2((float)x.x, (float)x.y);
                        if (a.keep32) C32s[i + j * ld] = f;
                        else C32[i + (size_t)j * ld] = f;
                    }
                if (a.keep32) {
                    __syncthreads();
                    house_rows<kNT>(n, ld, C32s, reinterpret_cast<float2*>(v.gb), reinterpret_cast<float2*>(v.vb),
                                 reinterpret_cast<float2*>(v.pb), v.tau, v.d, v.e);
                } else {
                float2* vbf = reinterpret_cast<float2*>(v.pb);
                float2* pbf = vbf + n;
                const float2 fz = f2(0.0f, 0.0f);
                __syncthreads();
                for (int k = 0; k < n - 1; ++k) {
                    float2* ck = C32 + (size_t)k * ld;
                    if (warp == 0) {
                        float ss = 0.0f;
                        for (int i = k + 2 + lane; i < n; i += 32) { const float2 x = ck[i]; ss = fmaf(x.x, x.x, fmaf(x.y, x.y, ss)); }
                        ss = warp_sumf(ss);
                        const float2 alpha = ck[k + 1];
                        float2 taui = fz, scal = fz;
                        float beta;
                        if (ss == 0.0f && alpha.y == 0.0f) {
                            beta = alpha.x;
                        } else {
                            beta = -copysignf(sqrtf(alpha.x * alpha.x + alpha.y * alpha.y + ss), alpha.x);
                            taui = f2((beta - alpha.x) / beta, -alpha.y / beta);
                            const float2 z = f2(alpha.x - beta, alpha.y);
                            const float inv = 1.0f / (z.x * z.x + z.y * z.y);
                            scal = f2(z.x * inv, -z.y * inv);
                        }
                        for (int i = k + 2 + lane; i < n; i += 32) {
                            const float2 vi = fcmul(ck[i], scal);
                            vbf[i] = vi;
                            ck[i] = vi;
                        }
                        if (lane == 0) {
                            vbf[k + 1] = f2(1.0f, 0.0f);
                            v.tau[k] = f2d(taui);
                            v.d[k] = (double)ck[k].x;
                            v.e[k] = (double)beta;
                        }
                    }
                    __syncthreads();
                    const float2 taui = f2((float)v.tau[k].x, (float)v.tau[k].y);
                    if (taui.x == 0.0f && taui.y == 0.0f) continue;
                    for (int i = k + 1 + warp; i < n; i += kNW) {
                        const float2* ci = C32 + (size_t)i * ld;
                        float2 acc = fz;
#pragma unroll 4
                        for (int j = k + 1 + lane; j < n; j += 32) acc = fcfmac(acc, ci[j], vbf[j]);
                        acc = warp_sum2f(acc);
                        if (lane == 0) pbf[i] = fcmul(taui, acc);
                    }
                    __syncthreads();
                    if (warp == 0) {
                        float2 dot = fz;
                        for (int i = k + 1 + lane; i < n; i += 32) dot = fcfmac(dot, pbf[i], vbf[i]);
                        dot = warp_sum2f(dot);
                        if (lane == 0) { const float2 t = fcmul(taui, dot); v.red[0] = c2(-0.5 * t.x, -0.5 * t.y); }
                    }
                    __syncthreads();
                    const float2 alpha2 = f2((float)v.red[0].x, (float)v.red[0].y);
                    for (int j = k + 1 + warp; j < n; j += kNW) {
                        float2* cj = C32 + (size_t)j * ld;
                        // w = p + alpha2 v
                        const float2 vj = vbf[j], wj = fcfma(pbf[j], alpha2, vj);
#pragma unroll 4
                        for (int i = k + 1 + lane; i < n; i += 32) {
                            const float2 vi = vbf[i], wi = fcfma(pbf[i], alpha2, vi);
                            float2 x = cj[i];
                            x = fcfms_bc(x, vi, wj);
                            x = fcfms_bc(x, wi, vj);
                            cj[i] = x;
                        }
                    }
                    __syncthreads();
                }
                if (tid == 0) {
                    v.d[n - 1] = (double)C32[(n - 1) + (size_t)(n - 1) * ld].x;
                    if (n == 1) v.tau[0] = zero;
                }
                __syncthreads();
                }
            } else if constexpr (ROWS) {
                house_rows<kNT>(n, ld, M0, v.gb, v.vb, reinterpret_cast<double2*>(v.dcd + (n & 1)), v.tau, v.d, v.e);
            } else {
                tiled_house<kNT>(n, ld, M0, M2, smem_raw);
            }
            phase_mark(20);

            // ---- a5b: divide and conquer on T: Z in M2 (real), its merge
            // workspace after it, merge products through Zo
            DCShared dc;
            dc.Z = reinterpret_cast<double*>(M2); dc.ldz = ld;
            dc.U = dc.Z + mat;                    dc.ldu = ld;
            dc.Zo = Zo;
            // the work area is free here, else tb and gb are
            dc.leaf = reinterpret_cast<double*>(a.work ? v.part : v.tb);
            dc.leaf_lanes = (int)((a.work ? tiled_work_elems(n) : 768) * 2 / (kLeafStride * kLeaf)) * kLeaf;
            dc.d = v.d; dc.ds = 1; dc.e = v.e; dc.es = 1;
            dc_carve(dc, v.dcd, v.dci, n);
            tiled_dc<kNT>(n, dc);
            // a failed eigensolve shows as a non-finite value (every warp looks
            // at all of them: the verdict is uniform without a barrier)
            bool bad = false;
            for (int i = lane; i < n; i += 32) bad |= !isfinite(dc.w[i]);
            code = __any_sync(0xffffffffu, bad) ? kEigFailCode : 0;
            for (int t = tid; t < n; t += kNT) v.rank[dc.ord[t]] = t;
            __syncthreads();
            phase_mark(21);
        }

        if (use32 && code) {
            // FP32 overflowed or underflowed (or the input is not finite): FP64 decides
            code = 0;
            if (a.defer) {
                if (tid == 0) a.info[b] = kRetryInfo;
                return;
            }
            use32 = false;
            continue;
        }
        if (code) break;

        // ---- a5c: V = Q Z in the output, columns in ascending eigenvalue order
        {
            const double* Z = reinterpret_cast<const double*>(M2);
            for (int idx = tid; idx < (int)nn; idx += kNT) {
                const int j = idx / n, i = idx - j * n;
                Ub[i + (size_t)v.rank[j] * n] = c2(Z[i + (size_t)j * ld], 0.0);
            }
            for (int j = tid; j < n; j += kNT) Wb[v.rank[j]] = v.dcd[j];
        }
        __syncthreads();
        const int nref = n - 1;
        {
            // Y with its ones and zeros in place, so that the products need
            // no masks: over the reduced C, or, for the mixed form, which
            // still needs C, widened from the FP32 reduction into M3
            double2* Y = use32 ? M3 : M0;
            for (int k = warp; k < nref; k += kNW)
                for (int i = lane; i < n; i += 32)
                    if (use32 || i <= k + 1)
                        Y[i + (size_t)k * ld] = i <= k ? zero : i == k + 1 ? c2(1.0, 0.0)
                                              : f2d(a.keep32 ? C32s[i + k * ld] : C32[i + (size_t)k * ld]);
            __syncthreads();
            // (M2 is free: Z is in the output; it holds the factors' 24 n from
            // n = 34 on, tb and gb three of them)
            wy_apply<kNT>(Ub, n, Y, ld, nref, v.tau, nref > 32 ? M2 : v.tb);
            __syncthreads();
        }
        if (use32) phase_mark(22);

        if (use32) {
            // ---- a5d: Ogita-Aishima refinement in FP64 of the eigenpairs of
            // C (M0) from the estimate V (columns in the output):
            //   R = I - V^H V, P = C V, Sm = V^H P, lam_i = Sm_ii / (1 - R_ii),
            //   delta = 2 (||Sm - diag(lam)||_F + max|lam| ||R||_F),
            //   E_ij = (Sm_ij + lam_j R_ij) / (lam_j - lam_i) if |lam_j - lam_i| > delta,
            //          R_ij / 2 otherwise (and on the diagonal),
            //   V <- V + V E,
            // until V passes the convergence test above. R / E in M2, P in
            // the next-estimate buffer, Sm in M4.
            double* lam = v.dcd + n;
            double2* Vh = Ub;  int ldh = n;
            double2* Vn = M3;  int ldn = ld;
            const int tl = tn * (tn + 1) / 2;
            bool conv = false;
            for (int it = 0;; ++it) {
                for (int t = warp; t < tl + tn * tn; t += kNW) {
                    Z16 acc;
                    z16_zero(acc);
                    if (t < tl) {
                        int ti, tj;
                        tri_tile(t, ti, tj);
                        const int i0 = 16 * ti, j0 = 16 * tj;
                        z16_gemm<true, false, false>(acc, i0, j0, 0, n, Vh, ldh, 1, n, Vh, 1, ldh, n);
                        z16_store(acc, i0, j0, [&](int i, int j, double2 x) {
                            if (i < n && j < n && i >= j) {
                                x = c2((i == j ? 1.0 : 0.0) - x.x, i == j ? 0.0 : -x.y);
                                M2[i + (size_t)j * ld] = x;
                                M2[j + (size_t)i * ld] = cconj(x);
                            }
                        });
                    } else {
                        const int t2 = t - tl, ti = t2 / tn, tj = t2 - ti * tn, i0 = 16 * ti, j0 = 16 * tj;
                        z16_gemm<false, false, false>(acc, i0, j0, 0, n, M0, 1, ld, n, Vh, 1, ldh, n);
                        z16_store(acc, i0, j0, [&](int i, int j, double2 x) { if (i < n && j < n) Vn[i + (size_t)j * ldn] = x; });
                    }
                }
                __syncthreads();
                for (int t = warp; t < tl; t += kNW) {
                    int ti, tj;
                    tri_tile(t, ti, tj);
                    const int i0 = 16 * ti, j0 = 16 * tj;
                    Z16 acc;
                    z16_zero(acc);
                    z16_gemm<true, false, false>(acc, i0, j0, 0, n, Vh, ldh, 1, n, Vn, 1, ldn, n);
                    z16_store(acc, i0, j0, [&](int i, int j, double2 x) {
                        if (i < n && j < n && i >= j) {
                            if (i == j) x.y = 0.0;
                            M4[i + (size_t)j * ld] = x;
                            M4[j + (size_t)i * ld] = cconj(x);
                        }
                    });
                }
                __syncthreads();
                for (int i = tid; i < n; i += kNT) lam[i] = M4[i + (size_t)i * ld].x / (1.0 - M2[i + (size_t)i * ld].x);
                __syncthreads();
                {
                    double sS = 0.0, sR = 0.0, lmax = 0.0;
                    for (int idx = tid; idx < (int)nn; idx += kNT) {
                        const int j = idx / n, i = idx - j * n;
                        double2 x = M4[i + (size_t)j * ld];
                        if (i == j) x.x -= lam[i];
                        sS = fma(x.x, x.x, fma(x.y, x.y, sS));
                        const double2 r = M2[i + (size_t)j * ld];
                        sR = fma(r.x, r.x, fma(r.y, r.y, sR));
                    }
                    for (int i = tid; i < n; i += kNT) lmax = fmax(lmax, fabs(lam[i]));
                    sS = warp_sum(sS);
                    sR = warp_sum(sR);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
                    if (lane == 0) { v.red[warp] = c2(sS, sR); v.gb[warp] = c2(lmax, 0.0); }
                    __syncthreads();
                    if (tid == 0) {
                        double a1 = 0.0, a2 = 0.0, mx = 0.0;
                        for (int w8 = 0; w8 < kNW; ++w8) { a1 += v.red[w8].x; a2 += v.red[w8].y; mx = fmax(mx, v.gb[w8].x); }
                        v.gb[16] = c2(2.0 * (sqrt(a1) + mx * sqrt(a2)), 0.0);
                        // converged: V orthonormal and C V = V diag(lam) to rounding level
                        const double tol = 16.0 * kEps * n;
                        v.gb[17] = c2((sqrt(a2) <= tol && sqrt(a1) <= tol * mx) ? 1.0 : 0.0, 0.0);
                    }
                    __syncthreads();
                }
                if (v.gb[17].x != 0.0) { conv = true; break; }
                if (it == a.refine_max) break;
                const double delta = v.gb[16].x;
                for (int idx = tid; idx < (int)nn; idx += kNT) {
                    const int j = idx / n, i = idx - j * n;
                    const double2 r = M2[i + (size_t)j * ld];
                    double2 e = cscale(r, 0.5);
                    if (i != j) {
                        const double g = lam[j] - lam[i];
                        if (fabs(g) > delta) e = cscale(cadd(M4[i + (size_t)j * ld], cscale(r, lam[j])), 1.0 / g);
                    }
                    M2[i + (size_t)j * ld] = e;
                }
                __syncthreads();
                for (int t = warp; t < tn * tn; t += kNW) {
                    const int ti = t / tn, tj = t - ti * tn, i0 = 16 * ti, j0 = 16 * tj;
                    Z16 acc;
                    z16_load(acc, i0, j0, [&](int i, int j) { return (i < n && j < n) ? Vh[i + (size_t)j * ldh] : zero; });
                    z16_gemm<false, false, false>(acc, i0, j0, 0, n, Vh, 1, ldh, n, M2, 1, ld, n);
                    z16_store(acc, i0, j0, [&](int i, int j, double2 x) { if (i < n && j < n) Vn[i + (size_t)j * ldn] = x; });
                }
                __syncthreads();
                double2* tp = Vh; Vh = Vn; Vn = tp;
                const int tld = ldh; ldh = ldn; ldn = tld;
            }
            if (!conv) {
                // no convergence from the FP32 start (possible when C's
                // spectrum is spread over many orders of magnitude): redo
                // this pencil's eigensolve in FP64 from C, still intact in M0
                if (a.defer) {
                    if (tid == 0) a.info[b] = kRetryInfo;
                    return;
                }
                use32 = false;
                continue;
            }
            if (Vh != Ub) {   // an odd number of steps left the estimate in M3
                for (int idx = tid; idx < (int)nn; idx += kNT) {
                    const int j = idx / n, i = idx - j * n;
                    Ub[idx] = Vh[i + (size_t)j * ldh];
                }
                __syncthreads();
            }
            // new ascending order of the refined eigenvalues
            for (int j = tid; j < n; j += kNT) {
                const double dj = order_key(lam[j]);
                int r = 0;
                for (int k2 = 0; k2 < n; ++k2) {
                    const double dk = order_key(lam[k2]);
                    r += (dk < dj) || (dk == dj && k2 < j);
                }
                v.rank[j] = r;
            }
            __syncthreads();
            for (int j = tid; j < n; j += kNT) Wb[v.rank[j]] = lam[j];
            if (a.stage == 3) {
                for (int idx = tid; idx < (int)nn; idx += kNT) {
                    const int j = idx / n, i = idx - j * n;
                    M2[i + (size_t)v.rank[j] * ld] = Ub[idx];
                }
                __syncthreads();
                for (int idx = tid; idx < (int)nn; idx += kNT) {
                    const int j = idx / n, i = idx - j * n;
                    Ub[idx] = M2[i + (size_t)j * ld];
                }
            }
        }

        break;
    }
    phase_mark(use32 ? 25 : 22);
    if (code) {
        const double qnan = __longlong_as_double(0x7ff8000000000000LL);
        for (int idx = tid; idx < (int)nn; idx += kNT) Ub[idx] = c2(qnan, qnan);
        if (a.stage >= 3) for (int i = tid; i < n; i += kNT) Wb[i] = qnan;
        if (tid == 0) a.info[b] = code == kEigFailCode ? eig_fail_info(n) : code;
        return;
    }

    if (tid == 0) a.info[b] = 0;
    if (a.stage == 3) return;

    // ---- a6: U = X^H V -> M2, U(i, j) = sum_{k >= i} conj(X(k, i)) V(k, j); then to the output
    for (int t = warp; t < tile_blocks(tn, tn); t += kNW) {
        int ti, tj;
        if (!tile_at(t, tn, tn, ti, tj)) continue;
        const int i0 = 16 * ti, j0 = 16 * tj;
        Z16 acc;
        z16_zero(acc);
        z16_gemm<true, false, false>(acc, i0, j0, i0, n, M1, ld, 1, n, Ub, 1, n, n);
        z16_store(acc, i0, j0, [&](int i, int j, double2 x) { if (i < n && j < n) M2[i + (size_t)j * ld] = x; });
    }
    __syncthreads();
    phase_mark(23);
    for (int idx = tid; idx < (int)nn; idx += kNT) {
        const int j = idx / n, i = idx - j * n;
        Ub[i + (size_t)(use32 ? v.rank[j] : j) * n] = M2[i + (size_t)j * ld];
    }
}

}  // namespace tiled
}  // namespace sgeig
