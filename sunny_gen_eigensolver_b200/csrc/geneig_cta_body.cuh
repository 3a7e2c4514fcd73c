// Per-pencil body of the shared-memory (smem-cta) solver, shared by its own
// kernel (geneig_cta.cu) and the persistent uneven-size kernel
// (geneig_uneven.cu). The stage chain is described in geneig_cta.cu.
#pragma once

// How the per-pencil body is compiled into its callers: inlined into the
// size's own kernel; a caller that dispatches several bodies (the persistent
// uneven-size kernel) may define it as __noinline__ before including, so
// that each body keeps its own register allocation.
#ifndef SGEIG_CTA_BODY_INLINE
#define SGEIG_CTA_BODY_INLINE __forceinline__
#endif

#include "geneig_common.cuh"
#include "geneig_dc.cuh"
#include "geneig_kernels.h"

#include <cmath>
namespace sgeig {
namespace cta {

struct CtaArgs {
    const double2* __restrict__ H;
    const double2* __restrict__ S;
    double*  W;
    double2* U;
    int*     info;
    long long batch;
    int n, ld, stage;
    int sigma;      // H = diag(I_{n/2}, -I_{n/2}), not read from memory
    // intensity form (SPEC): spin-wave intensities in place of U
    const double2* O;        // 3 x n observable matrix per problem (column-major)
    const double*  qhat;     // 3 per problem
    const double*  energies; // ne
    double*        spec;     // ne per problem
    int            ne;
    double         gnorm;    // Gaussian normalisation 1 / (sigma sqrt(2 pi))
    double         ginv2;    // 1 / (2 sigma^2)
    int            retry;    // only the pencils whose info is kRetryInfo
};

// S assembled on the device instead of loaded (the FS form of cta_solve):
// S(q)_e = sum_{t in [start[e], start[e+1])} coef[t] exp(2 pi i q . disp[3t..3t+2])
// for the lower-triangle entries e = row + n col (row >= col), q = q[3b..3b+2].
struct CtaFourier {
    const int*     start;   // n*n + 1
    const double2* coef;
    const double*  disp;
    const double*  q;
    int            nterms;  // terms are read only from [0, nterms)
};

// Threads that solve one pencil, by row bound. One matrix per pencil is kept
// in shared memory, so the pencils per SM are bounded by registers for small
// n and by shared memory above; narrow teams keep many pencils, whose steps
// are chains of dependent operations, in flight.
constexpr int cta_team_threads(int nmax) {
    return nmax <= 16 ? 32 : nmax <= 32 ? 64 : nmax <= 64 ? 128 : nmax <= 80 ? 256 : 512;
}

// Rows of a pencil's matrix in shared memory: the intensity form appends the
// three rows of P = O X^H, which the Householder updates turn into P Q.
constexpr int kSpecRows = 3;
__host__ __device__ inline int cta_rows(int n, bool spec) { return spec ? n + kSpecRows : n; }
// Leading dimension: odd, so that walks along a row and the fragment accesses
// below (rows lane/4, columns 2 (lane%4) + s) are free of bank conflicts.
__host__ __device__ inline int cta_ld(int n, bool spec) { return cta_rows(n, spec) | 1; }

// Shared memory of one pencil's team after its n x ld matrix:
//   work   phase by phase: the 8-column panel of the Cholesky and reduction,
//          the Householder partial products and vectors, the divide and
//          conquer scratch with the WY factors after it
//   de     (d_k, e_k) of the tridiagonal, when the matrix has no padding row
//          to hold them
//   rank   ascending position of each eigenvalue
__host__ __device__ inline size_t cta_dc_bytes(int n, bool spec) {   // (d, e) first, then the scratch
    const size_t b = (size_t)n * 16 + (size_t)dc_vec_doubles(n) * 8 + (size_t)(spec ? kRowsTracked * n : 0) * 8 +
                     (size_t)dc_vec_ints(n) * 4;
    return (b + 15) & ~(size_t)15;
}
// The reduction's panel is two blocks wide where one pencil has the SM (its
// shared memory) to itself anyway. N=108: 235 K cycles for one, 141 K for two.
__host__ __device__ constexpr bool cta_two_panels(int nw) { return nw >= 16; }
constexpr int kDElems = 72;       // an 8 x 8 tile with leading dimension 9
__host__ __device__ inline size_t cta_work_bytes(int n, int nw, bool spec) {
    const size_t one = (size_t)8 * (n | 1);
    const size_t panel = (cta_two_panels(nw) ? 2 * one : one + 2 * kDElems) * 16;
    const size_t hh = ((size_t)32 * nw + 3 * cta_rows(n, spec)) * 16;
    const size_t dc = cta_dc_bytes(n, spec) + (spec ? 0 : (size_t)((n + 7) / 8) * 36 * 16);
    const size_t m = panel > hh ? panel : hh;
    return m > dc ? m : dc;
}
// Complex entries of the matrix area (the leaves of the divide and conquer
// keep their rows there too, which for tiny n take more than n x ld).
__host__ __device__ inline size_t cta_mat_elems(int n, bool spec) {
    const size_t mat = (size_t)n * cta_ld(n, spec), leaf = ((size_t)dc_leaf_doubles(n) + 1) / 2;
    return mat > leaf ? mat : leaf;
}
__host__ __device__ inline bool cta_pad_row(int n, bool spec) { return cta_ld(n, spec) > cta_rows(n, spec); }
__host__ __device__ inline size_t cta_bytes(int n, int nw, bool spec) {
    const size_t b = cta_mat_elems(n, spec) * 16 + cta_work_bytes(n, nw, spec) +
                     (cta_pad_row(n, spec) ? 0 : (size_t)n * 16) + (size_t)n * 4;
    return (b + 15) & ~(size_t)15;
}

// Complex step: D += A B with four real ones.
__device__ __forceinline__ void zmma(double (&re)[2], double (&im)[2], double2 a, double2 b) {
    mma884(re, a.x, b.x);
    mma884(re, -a.y, b.y);
    mma884(im, a.x, b.y);
    mma884(im, a.y, b.x);
}

template <int V> struct IntC { static constexpr int value = V; };

__device__ __forceinline__ double2 shfl2(double2 v, int src) {
    return c2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// One pencil b, solved end to end by a team of NT threads (every thread of
// the team calls this with the same b and the team's shared memory): the
// whole CTA when BLOCK == NT, else one of the BLOCK / NT teams of a CTA of
// BLOCK threads. FS: S is assembled from the Fourier terms `fs` instead of
// loaded. SPEC: the metric solve reduced to intensities (no U).
//
// Products run on the FP64 tensor cores in 8 x 8 tiles. In every k block of 8
// the MMA's k slot q of step s is column 2 q + s (any assignment that A and B
// share is valid), which makes the fragment accesses conflict-free for odd ld
// and an accumulator's layout (row l/4, columns 2 (l%4) + e) that of an A
// fragment.
//
// Global memory: the pencil's own output block U serves as scratch between
// the reduction and the back-transforms: X^H above and on its diagonal, the
// Householder vectors and their tau below. All of H and S is read before.
template <int NMAX, int NT, int BLOCK = NT, bool FS = false, bool SPEC = false>
__device__ SGEIG_CTA_BODY_INLINE void cta_solve(const CtaArgs& a, long long b, unsigned char* smem_raw,
                                                const CtaFourier* fs = nullptr) {
    constexpr int NW = NT / 32;     // warps
    constexpr int NB = NMAX / 8;    // 8-row tiles
    constexpr int R = (NMAX + (SPEC ? kSpecRows : 0) + 31) / 32;   // Householder rows per lane
    constexpr int PP = (NB + NW - 1) / NW;                         // 8-column panels per warp
    static_assert(NT % 32 == 0 && NW >= 1 && NW <= 16 && NMAX % 8 == 0, "team shape");
    const int n = a.n, ld = a.ld;
    const int rows = cta_rows(n, SPEC);
    double2* M = reinterpret_cast<double2*>(smem_raw);
    double2* work = M + cta_mat_elems(n, SPEC);
    unsigned char* after = reinterpret_cast<unsigned char*>(work) + cta_work_bytes(n, NW, SPEC);
    const bool pad = cta_pad_row(n, SPEC);
    double2* de = pad ? M + rows : reinterpret_cast<double2*>(after);   // (d_k, e_k) at de[k * des]
    const int des = pad ? ld : 1;
    int* rank = reinterpret_cast<int*>(after + (pad ? 0 : (size_t)n * 16));

    int tid = BLOCK == NT ? (int)threadIdx.x : (int)(threadIdx.x % NT), lane = tid & 31, warp = tid >> 5;
    int fr = lane >> 2, fq = lane & 3;           // fragment row / column index, k slots 2 fq + s
    auto phase = [&]() { forget(tid); forget(lane); forget(warp); forget(fr); forget(fq); };
    const int nb = (n + 7) >> 3;
    const size_t nn = (size_t)n * n;
    const double2 zero = c2(0.0, 0.0);

    const double2* Hb = a.H + (size_t)b * nn;
    const double2* Sb = a.S + (size_t)b * nn;
    double*  Wb = a.W + (size_t)b * n;
    double2* Ub = a.U + (size_t)b * nn;

    team_sync<NT, BLOCK>();   // the previous pencil's shared memory is free
    phase_mark(8);
    // ---- a1: lower triangle of S -> M
    if constexpr (FS) {
        // S(q) from its Fourier terms; they are shared by all pencils
        // (L1/L2-resident). Term values first, one term per thread (coalesced,
        // independent loads), into M's strict upper triangle, which is free
        // until a4, as many at a time as it holds; then each lower entry adds
        // its terms in table order. The triangle is folded into n/2 lines of
        // n1 = n - 1 slots (n even): line c holds column c (c entries), then
        // column n1 - c (n1 - c entries).
        const double q0 = __ldg(fs->q + 3 * b), q1 = __ldg(fs->q + 3 * b + 1), q2 = __ldg(fs->q + 3 * b + 2);
        const int nt = fs->nterms;
        const int n1 = n - 1, cap = (n >> 1) * n1;
        auto upper = [&](int s) -> double2* {
            const int c = s / n1, r = s - c * n1;
            return r < c ? M + r + (size_t)c * ld : M + (r - c) + (size_t)(n1 - c) * ld;
        };
#pragma unroll 1
        for (int idx = tid; idx < n * n; idx += NT) {
            const int j = idx / n, i = idx - j * n;
            if (i >= j) M[i + (size_t)j * ld] = zero;
        }
#pragma unroll 1
        for (int t0 = 0; t0 < nt; t0 += cap) {
            const int t1 = min(nt, t0 + cap);
#pragma unroll 1
            for (int t = t0 + tid; t < t1; t += NT) {
                const double x = fma(q0, __ldg(fs->disp + 3 * t),
                                 fma(q1, __ldg(fs->disp + 3 * t + 1), q2 * __ldg(fs->disp + 3 * t + 2)));
                double sn, cs;
                sincospi(2.0 * x, &sn, &cs);
                *upper(t - t0) = cmul(__ldg(fs->coef + t), c2(cs, sn));
            }
            team_sync<NT, BLOCK>();
#pragma unroll 1
            for (int idx = tid; idx < n * n; idx += NT) {
                const int j = idx / n, i = idx - j * n;
                if (i < j) continue;
                const int lo = max(__ldg(fs->start + idx), t0), hi = min(__ldg(fs->start + idx + 1), t1);
                if (lo >= hi) continue;
                double2 acc = M[i + (size_t)j * ld];
#pragma unroll 1
                for (int t = lo; t < hi; ++t) acc = cadd(acc, *upper(t - t0));
                M[i + (size_t)j * ld] = acc;
            }
            team_sync<NT, BLOCK>();
        }
        if (nt == 0) team_sync<NT, BLOCK>();
    } else {
        // one warp per column, copied asynchronously (every load in flight
        // at once, no registers)
#pragma unroll 1
        for (int j = warp; j < n; j += NW)
#pragma unroll 1
            for (int i = j + lane; i < n; i += 32) {
                const unsigned dst = (unsigned)__cvta_generic_to_shared(M + i + (size_t)j * ld);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(Sb + i + (size_t)j * n)
                             : "memory");
            }
        if (!a.sigma && a.stage >= 2) {   // H follows in a3: start it towards L2
            const char* hp = reinterpret_cast<const char*>(Hb);
#pragma unroll 1
            for (size_t o = (size_t)tid * 128; o < nn * 16; o += (size_t)NT * 128)
                asm volatile("prefetch.global.L2 [%0];" :: "l"(hp + o));
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        team_sync<NT, BLOCK>();
    }
    phase_mark(0);
    phase();

    // ---- a2: Cholesky S = L L^H together with X = L^-1, 8-column panels,
    // right-looking. In M's lower triangle, columns right of the current
    // panel p hold the Cholesky working matrix, columns up to p the inverse
    // accumulators Acc. With D = L_pp^-1 (from warp 0, in shared memory):
    //   L(i, p) = A(i, p) D^H  (i > p, into `work`),   X(p, c) = D Acc(p, c)  (c < p, in place)
    //   where L_pp is ill-conditioned: L(i, p) += (A(i, p) - L(i, p) L_pp^H) D^H
    // barrier
    //   Acc(i, c) -= L(i, p) X(p, c)  (c < p),  Acc(i, p) = -L(i, p) D,  A(i, j) -= L(i, p) L(j, p)^H
    // barrier; warp 0 updates the next diagonal tile first and factors it
    // while the other warps do the rest. Two barriers per 8 columns and all
    // products on the tensor cores; one barrier per column with a row in each
    // four-lane group's registers took 90 K CTA cycles at n = 54 and needed
    // 256 threads. Fragment rows past n read whatever lies there: they reach
    // discarded rows or columns of the result only.
    // Rounding is amplified in column c of A(i, p) D^H by at most kappa_c,
    // kappa_c^2 = sum_j A_jj |D(c, j)|^2 (|A(i, j)| <= ||L(i, :)|| sqrt(A_jj)). Where a
    // lane's share of it passes 8 the panel takes one step of refinement. N = 16,
    // cond(S) = 1e10, mean ||U^H S U - I||: 12.3e-8 without the step, 5.4e-8 with it,
    // 7.5e-8 LAPACK's. At cond(S) = 100 (kappa^2 up to 9) it is not needed; taken in
    // every panel it would cost N = 54 2.5 % of the solve.
    double2* Pn = work;                // n x 8 panel of L; rows 0 .. 7 (above every panel): L_pp
    const int ldp = n | 1;
    double2* Ds = work + 8 * ldp;      // D of even and odd panels: element (i, j) at i + 9 j
    // warp 0: L of the diagonal tile at o, row by lane, into rows 0 .. 7 of Pn, in
    // the same operations as factor() (D has to be this L's inverse; the scales are
    // D's diagonal; an infinite pivot's column is zero)
    auto tile_l = [&](int o, const double2* Dp) {
        double2* row = Pn + (lane & 7);
#pragma unroll 1
        for (int c = -1; c < 8; ++c) {
#pragma unroll 1
            for (int j = c + 1; j < 8 && lane < 8; ++j) {
                const double r = c < 0 ? 0.0 : Dp[10 * c].x;
                if (c < 0) row[j * ldp] = j <= lane ? M[o + lane + (o + j) * ld] : zero;
                else if (lane >= j) row[j * ldp] = cfms_bc(row[j * ldp], cscale(row[c * ldp], r * r), Pn[j + c * ldp]);
            }
            __syncwarp();
        }
#pragma unroll 1
        for (int j = 0; j <= lane && lane < 8; ++j) {
            const double2 v = row[j * ldp];
            const double r = Dp[10 * j].x, l = v.x * r;
            row[j * ldp] = j < lane ? cscale(v, r) : c2(r > 0.0 ? fma(l, fma(-l, r, 1.0), l) : 0.0, 0.0);
        }
        __syncwarp();
    };
    auto factor = [&](int p) {         // warp 0; lane: row fr, columns 2 fq + s of the tile
        const int o = 8 * p;
        double2* Dp = Ds + (p & 1) * kDElems;
        double2 x[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int j = 2 * fq + s;
            x[s] = (o + fr < n && j <= fr) ? M[o + fr + (o + j) * ld] : c2(fr == j ? 1.0 : 0.0, 0.0);
        }
        int bad = 0;
        double rr = 0.0;               // 1 / L of this lane's row
#pragma unroll 1
        for (int h = 0; h < 4; ++h) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int c = 2 * h + u;
                const double akk = __shfl_sync(0xffffffffu, x[u].x, 4 * c + h);
                if (!bad && o + c < n && !(akk > 0.0)) bad = o + c + 1;
                const double r = rsqrt(akk), r2 = r * r;
                if (fr == c) rr = r;
                const double2 aic = shfl2(x[u], (lane & 28) + h);
                double2 ajc[2], rc[2];
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    ajc[s] = shfl2(x[u], 4 * (2 * fq + s) + h);      // column c, row j
                    rc[s] = shfl2(x[s], 4 * c + fq);                 // row c, column j
                }
                if (a.stage == 1 && fq == h && o + fr < n && fr >= c && !bad)
                    Ub[o + fr + (size_t)(o + c) * n] = fr == c ? c2(1.0 / r, 0.0) : cscale(aic, r);
                if (fr > c) {
                    const double2 aik = cscale(aic, r2);
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const int j = 2 * fq + s;
                        if (j > c) { if (j <= fr) x[s] = cfms_bc(x[s], aik, ajc[s]); }
                        else if (j < c) x[s] = cfms(x[s], aik, rc[s]);
                        else x[s] = cscale(aik, -1.0);
                    }
                }
            }
        }
        if (lane == 0) rank[0] = bad;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int j = 2 * fq + s;
            Dp[fr + 9 * j] = j < fr ? cscale(x[s], rr) : c2(j == fr ? rr : 0.0, 0.0);
        }
    };
    int fail = 0;
#pragma unroll 1
    for (int p = -1; p < nb; ++p) {    // p = -1: the first diagonal tile only
        const int o = 8 * p;
        const double2* Dp = Ds + (p & 1) * kDElems;
        if (p >= 0) {
            fail = rank[0];
            if (fail) break;
            // (A's diagonal is in M until warp 0 puts D there below)
            double kap = 0.0;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int k = 2 * fq + s;
                const double2 d = Dp[fr + 9 * k];
                kap = fma(M[min(o + k, n - 1) * (ld + 1)].x, fma(d.x, d.x, d.y * d.y), kap);
            }
            const bool refine = __any_sync(0xffffffffu, kap > 8.0) && o + 8 < n;
#pragma unroll 1
            for (int t = warp; t < nb - 1; t += NW) {
                double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
                const bool xt = t < p;     // X(p, t) = D Acc(p, t), else L(t + 1, p) = A(t + 1, p) D^H
                const int i = 8 * (t + 1) + fr;
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const int k = 2 * fq + s;
                    const double2 dd = Dp[fr + 9 * k];
                    const double2 m = xt ? M[min(o + k, n - 1) + (8 * t + fr) * ld] : M[i + (o + k) * ld];
                    zmma(re, im, xt ? dd : m, xt ? m : cconj(dd));
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int j = 2 * fq + e;
                    if (xt) {
                        if (o + fr < n) M[o + fr + (8 * t + j) * ld] = c2(re[e], im[e]);
                    } else if (i < n) {
                        Pn[i + j * ldp] = c2(re[e], im[e]);
                        if (a.stage == 1) Ub[i + (size_t)(o + j) * n] = c2(re[e], im[e]);
                    }
                }
            }
            if (refine) {                  // the same verdict in every warp
                if (warp == 0) tile_l(o, Dp);
                team_sync<NT, BLOCK>();
                // every lane on the elements of L that it has just written (an
                // accumulator is laid out as the next A fragment)
#pragma unroll 1
                for (int t = warp; t < nb - 1; t += NW) {
                    if (t < p) continue;
                    const int i = 8 * (t + 1) + fr;
                    double re[2], im[2], dr[2], di[2];
                    double2 l[2];
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        l[s] = Pn[i + (2 * fq + s) * ldp];
                        re[s] = l[s].x;
                        im[s] = l[s].y;
                        const double2 m = M[i + (o + 2 * fq + s) * ld];
                        dr[s] = m.x;
                        di[s] = m.y;
                    }
#pragma unroll
                    for (int s = 0; s < 2; ++s)          // A - L L_pp^H
                        zmma(dr, di, c2(-l[s].x, -l[s].y), cconj(Pn[fr + (2 * fq + s) * ldp]));
#pragma unroll
                    for (int s = 0; s < 2; ++s) zmma(re, im, c2(dr[s], di[s]), cconj(Dp[fr + 9 * (2 * fq + s)]));
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int j = 2 * fq + e;
                        if (i >= n) continue;
                        Pn[i + j * ldp] = c2(re[e], im[e]);
                        if (a.stage == 1) Ub[i + (size_t)(o + j) * n] = c2(re[e], im[e]);
                    }
                }
            }
            team_sync<NT, BLOCK>();
        }
        auto update = [&](int i8, int j8) {
            const int i = 8 * i8 + fr;
            double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
            if (j8 != p) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const double2 c = M[i + (8 * j8 + 2 * fq + e) * ld];
                    re[e] = c.x; im[e] = c.y;
                }
            }
            // B(k, j) = conj(L(j, p)), X(p, j) or D, by the tile's column
            const double2* bp = j8 > p ? Pn + 8 * j8 + fr + 2 * fq * ldp
                              : j8 < p ? M + o + 2 * fq + (8 * j8 + fr) * ld : Dp + 2 * fq + 9 * fr;
            const int bs = j8 > p ? ldp : 1;
            const double sg = j8 > p ? 1.0 : -1.0;      // conj(B) for j8 > p, -A in place of A
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const double2 l = Pn[i + (2 * fq + s) * ldp], bv = bp[s * bs];
                mma884(re, -l.x, bv.x);
                mma884(re, -sg * l.y, bv.y);
                mma884(im, sg * l.x, bv.y);
                mma884(im, -l.y, bv.x);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int j = 8 * j8 + 2 * fq + e;
                if (i < n && j < n) M[i + j * ld] = c2(re[e], im[e]);
            }
        };
        // warp 0: the next diagonal tile, then its factor; the others (a lone
        // warp: the same one) the remaining tiles (i8, j8 <= i8), row by row
        if (p >= 0) {
            if (warp == 0 && o + fr < n) {
#pragma unroll
                for (int s = 0; s < 2; ++s)
                    if (2 * fq + s <= fr) M[o + fr + (o + 2 * fq + s) * ld] = Dp[fr + 9 * (2 * fq + s)];
            }
            int i8 = p + 1, j8 = NW == 1 ? 0 : warp == 0 ? p + 1 : warp - 1;
#pragma unroll 1
            for (;;) {
                while (i8 < nb && j8 > i8) { j8 -= i8 + 1; ++i8; }
                if (i8 >= nb) break;
                if (NW == 1 || warp == 0 || i8 != p + 1 || j8 != p + 1) update(i8, j8);
                j8 += NW == 1 ? 1 : warp == 0 ? nb * nb : NW - 1;
            }
            __syncwarp();
        }
        if (warp == 0 && p + 1 < nb) factor(p + 1);
        team_sync<NT, BLOCK>();
    }
    phase_mark(1);
    phase();
    int code = fail ? n + fail : 0;   // zhegv: info = n + order of the failing minor

    if (!code && a.stage == 1) {
#pragma unroll 1
        for (int j = warp; j < n; j += NW)
#pragma unroll 1
            for (int i = lane; i < j; i += 32) Ub[i + (size_t)j * n] = zero;
        if (tid == 0) a.info[b] = 0;
        return;
    }

    if (!code) {
        // M holds X = L^-1 in its lower triangle (diagonal real); the upper
        // triangle receives C below, so the tiles on the diagonal are masked.
        // C(i, j) of tile (ti, tj) (ti >= tj): conj into M(j, i), the diagonal's
        // real part into de[.].x
        auto put_c = [&](int ti, int tj, const double (&re)[2], const double (&im)[2]) {
            const int i = 8 * ti + fr;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int j = 8 * tj + 2 * fq + e;
                if (i < n && j < i) M[j + i * ld] = c2(re[e], -im[e]);
                else if (i < n && j == i) de[i * des] = c2(re[e], 0.0);
            }
        };
        if (SPEC || a.sigma) {
            // ---- a3 + a4, H = diag(I, -I): C = X diag(I, -I) X^H directly
            const int m = n >> 1;
            int i8 = 0, j8 = warp;
#pragma unroll 1
            for (;;) {
                while (i8 < nb && j8 > i8) { j8 -= i8 + 1; ++i8; }
                if (i8 >= nb) break;
                double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
                const double2* xi = M + 8 * i8 + fr;
                const double2* xj = M + 8 * j8 + fr;
#pragma unroll 1
                for (int kb = 0; kb <= j8; ++kb) {
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const int kr = 2 * fq + s, k = 8 * kb + kr;
                        double2 av = xi[k * ld], y = xj[k * ld];
                        if (kb == j8 && kr > fr) {       // above X's diagonal
                            y = zero;
                            if (i8 == j8) av = zero;
                        }
                        const double sg = k < m ? 1.0 : -1.0;
                        zmma(re, im, av, c2(sg * y.x, -sg * y.y));
                    }
                }
                put_c(i8, j8, re, im);
                j8 += NW;
            }
            phase_mark(2);
        } else {
            // ---- a3 + a4, one or two 8-column blocks of C at a time:
            // T(:, tj) = H X(tj, :)^H into `work` (H read in full, from global
            // memory, L2 after the first blocks), then C(ti, tj) = X(ti, :) T,
            // ti >= tj.
            double2* Tp = work;
            if constexpr (cta_two_panels(NW)) {
                // Two blocks of C at a time, a row tile per warp: each element
                // of H and of X serves both, and the sixteen warps meet half
                // as often.
#pragma unroll 1
                for (int tj = 0; tj < nb; tj += 2) {
                    const bool two = tj + 1 < nb;
                    const int kend = two ? tj + 1 : tj;
#pragma unroll 1
                    for (int t0 = warp; t0 < nb; t0 += NW) {
                        const int i0 = 8 * t0 + fr;
                        double re0[2] = {0.0, 0.0}, im0[2] = {0.0, 0.0}, re1[2] = {0.0, 0.0}, im1[2] = {0.0, 0.0};
                        const double2* x0 = M + 8 * tj + fr;
                        const double2* h0 = Hb + min(i0, n - 1);
                        double2 y[4][2];         // H of the next four k blocks, loaded ahead
#pragma unroll
                        for (int p = 0; p < 4; ++p)
#pragma unroll
                            for (int s = 0; s < 2; ++s) y[p][s] = __ldg(h0 + min(8 * p + 2 * fq + s, n - 1) * n);
#pragma unroll 1
                        for (int kb = 0; kb <= kend; ++kb) {
                            const double2 av[2] = {y[0][0], y[0][1]};
#pragma unroll
                            for (int p = 0; p < 3; ++p) {
                                y[p][0] = y[p + 1][0];
                                y[p][1] = y[p + 1][1];
                            }
                            if (kb + 4 <= kend) {
#pragma unroll
                                for (int s = 0; s < 2; ++s) y[3][s] = __ldg(h0 + min(8 * kb + 32 + 2 * fq + s, n - 1) * n);
                            }
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int kr = 2 * fq + s;
                                const double2* xk = x0 + (8 * kb + kr) * ld;
                                if (kb <= tj) {
                                    double2 bv = cconj(xk[0]);
                                    if (kb == tj && kr > fr) bv = zero;
                                    zmma(re0, im0, av[s], bv);
                                }
                                if (two) {
                                    double2 bv = cconj(xk[8]);
                                    if (kb == tj + 1 && kr > fr) bv = zero;
                                    zmma(re1, im1, av[s], bv);
                                }
                            }
                        }
                        if (i0 < n) {
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                double2* tc = Tp + (2 * fq + e) * ldp + i0;
                                tc[0] = c2(re0[e], im0[e]);
                                if (two) tc[8 * ldp] = c2(re1[e], im1[e]);
                            }
                        }
                    }
                    team_sync<NT, BLOCK>();
#pragma unroll 1
                    for (int ti = tj + warp; ti < nb; ti += NW) {
                        double re0[2] = {0.0, 0.0}, im0[2] = {0.0, 0.0}, re1[2] = {0.0, 0.0}, im1[2] = {0.0, 0.0};
                        const double2* xi = M + 8 * ti + fr;
                        const double2* tc = Tp + fr * ldp;
                        const bool both = two && ti > tj;
#pragma unroll 1
                        for (int kb = 0; kb <= ti; ++kb) {
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int kr = 2 * fq + s, k = 8 * kb + kr, kc = min(k, n - 1);
                                double2 av = xi[k * ld];
                                if (kb == ti && kr > fr) av = zero;
                                zmma(re0, im0, av, tc[kc]);
                                if (both) zmma(re1, im1, av, tc[8 * ldp + kc]);
                            }
                        }
                        put_c(ti, tj, re0, im0);
                        if (both) put_c(ti, tj + 1, re1, im1);
                    }
                    team_sync<NT, BLOCK>();
                }
            } else {
                // One block at a time; two row tiles per warp share each
                // fragment of X.
#pragma unroll 1
                for (int tj = 0; tj < nb; ++tj) {
#pragma unroll 1
                    for (int t0 = warp; t0 < nb; t0 += 2 * NW) {
                        const int i0 = 8 * t0 + fr, i1 = i0 + 8 * NW;
                        double re0[2] = {0.0, 0.0}, im0[2] = {0.0, 0.0}, re1[2] = {0.0, 0.0}, im1[2] = {0.0, 0.0};
                        const double2* xj = M + 8 * tj + fr;
                        const double2* h0 = Hb + min(i0, n - 1);
                        const double2* h1 = Hb + min(i1, n - 1);
                        const bool two = t0 + NW < nb;
                        double2 y0[2][2], y1[2][2];  // H of the next two k blocks, loaded ahead
#pragma unroll
                        for (int p = 0; p < 2; ++p)
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int k = min(8 * p + 2 * fq + s, n - 1);
                                y0[p][s] = __ldg(h0 + k * n);
                                y1[p][s] = __ldg(h1 + k * n);
                            }
#pragma unroll 1
                        for (int kb = 0; kb <= tj; ++kb) {
                            const double2 a0[2] = {y0[0][0], y0[0][1]}, a1[2] = {y1[0][0], y1[0][1]};
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int k = min(8 * kb + 16 + 2 * fq + s, n - 1);
                                y0[0][s] = y0[1][s];
                                y1[0][s] = y1[1][s];
                                if (kb + 2 <= tj) {
                                    y0[1][s] = __ldg(h0 + k * n);
                                    y1[1][s] = __ldg(h1 + k * n);
                                }
                            }
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int kr = 2 * fq + s;
                                double2 bv = cconj(xj[(8 * kb + kr) * ld]);
                                if (kb == tj && kr > fr) bv = zero;
                                zmma(re0, im0, a0[s], bv);
                                if (two) zmma(re1, im1, a1[s], bv);
                            }
                        }
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            double2* tc = Tp + (2 * fq + e) * ldp;
                            if (i0 < n) tc[i0] = c2(re0[e], im0[e]);
                            if (i1 < n) tc[i1] = c2(re1[e], im1[e]);
                        }
                    }
                    team_sync<NT, BLOCK>();
#pragma unroll 1
                    for (int ti = tj + warp; ti < nb; ti += NW) {
                        double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
                        const double2* xi = M + 8 * ti + fr;
                        const double2* tc = Tp + fr * ldp;
#pragma unroll 1
                        for (int kb = 0; kb <= ti; ++kb) {
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int kr = 2 * fq + s, k = 8 * kb + kr;
                                double2 av = xi[k * ld];
                                if (kb == ti && kr > fr) av = zero;
                                zmma(re, im, av, tc[min(k, n - 1)]);
                            }
                        }
                        put_c(ti, tj, re, im);
                    }
                    team_sync<NT, BLOCK>();
                }
            }
            phase_mark(2);
        }
        if constexpr (SPEC) {
            // P = O X^H (3 x n) into rows n .. n+2
            const double2* Ob = a.O + (size_t)b * 3 * n;
#pragma unroll 1
            for (int idx = tid; idx < 3 * n; idx += NT) {
                const int c = idx / n, k = idx - c * n;
                double2 acc = zero;
#pragma unroll 1
                for (int i = 0; i <= k; ++i) acc = cfma(acc, __ldg(Ob + c + 3 * i), cconj(M[k + (size_t)i * ld]));
                M[n + c + (size_t)k * ld] = acc;
            }
        } else if (a.stage == 4) {
            // X^H into the upper triangle and the diagonal of U's block
#pragma unroll 1
            for (int k = warp; k < n; k += NW)
#pragma unroll 1
                for (int i = lane; i <= k; i += 32) Ub[i + (size_t)k * n] = cconj(M[k + (size_t)i * ld]);
        }
        team_sync<NT, BLOCK>();
        // C to the lower triangle and the diagonal: M is exactly Hermitian
#pragma unroll 1
        for (int j = warp; j < n; j += NW)
#pragma unroll 1
            for (int i = j + lane; i < n; i += 32)
                M[i + (size_t)j * ld] = i == j ? c2(de[j * des].x, 0.0) : cconj(M[j + (size_t)i * ld]);
        team_sync<NT, BLOCK>();
        phase_mark(3);
    phase();
    }

    if (!code && a.stage == 2) {
#pragma unroll 1
        for (int j = warp; j < n; j += NW)
#pragma unroll 1
            for (int i = lane; i < n; i += 32) Ub[i + (size_t)j * n] = M[i + (size_t)j * ld];
        if (tid == 0) a.info[b] = 0;
        return;
    }

    double2* tpk = reinterpret_cast<double2*>(reinterpret_cast<unsigned char*>(work) + cta_dc_bytes(n, SPEC));
    auto tidx = [](int c, int l, int i) { return 36 * c + ((i * (i + 1)) >> 1) + l; };   // T_c(l, i), l <= i
    const int nref = n - 1;                      // reflectors 0 .. n-2
    const int nblk = (nref + 7) >> 3;            // WY blocks of 8
    DCShared dc;
    dc.Z = reinterpret_cast<double*>(M); dc.ldz = ld;
    dc.U = dc.Z + (size_t)n * ld;        dc.ldu = ld;
    dc.Zo = nullptr;
    dc.leaf = dc.Z; dc.leaf_lanes = kLeaf * nb;
    {
        double* dv = reinterpret_cast<double*>(work + n);
        dc.rows = SPEC ? dv + dc_vec_doubles(n) : nullptr;
        int* iv = reinterpret_cast<int*>(dv + dc_vec_doubles(n) + (SPEC ? kRowsTracked * n : 0));
        dc_carve(dc, dv, iv, n);
    }
    dc.d = reinterpret_cast<const double*>(work); dc.ds = 2;
    dc.e = dc.d + 1;                              dc.es = 2;

    if (!code) {
        // ---- a5a: Householder tridiagonalisation of C (lower), one pass over
        // the trailing matrix per step. Rows are counted from the last one up
        // in blocks of 32 (so that the blocks in use follow the trailing
        // matrix), a lane per row; with RB blocks in use, warp w takes block
        // w % RB of the columns j = w / RB mod NW / RB, so that a row has only
        // NW / RB partial products to add.
        // Step c (column c):
        //   one warp (a different one each step, so that the pencils of an SM
        //   spread over its schedulers): y = A v from the warps' partial
        //     products (v: reflector c - 1), p = tau y, w = p + alpha2 v
        //     (alpha2 = -|tau|^2/2 v^H A v, real), column c of the updated
        //     matrix and from it reflector c, v_c; w, v_c to shared memory
        //   barrier; every warp over its own columns j > c, one load and one
        //   store of each element:
        //     A(:, j) -= v conj(w_j) + w conj(v_j),   y_next += A(:, j) v_c(j)
        //   barrier
        // The update and the next product share one pass, where separate
        // ones took 232 K CTA cycles at n = 54. With every warp doing the
        // first part for itself (one barrier) a step took twice the
        // instructions.
        // Reflector k: I - tau_k v v^H on rows k+1.., v[k+1] = 1; column k of M
        // keeps v[k+2..] and tau_k at row k + 1. SPEC: rows n .. n+2 see the
        // same update with v = 0 there, which is P <- P (I - tau v v^H), so
        // that P Q is in their place at the end.
        // Rows above the trailing matrix are carried along unmasked: v is zero
        // there, so they only see A <- A (I - tau v v^H), which keeps them
        // bounded, and nothing reads them.
        double2* part = work;                    // 32 NW partial products
        double2* vb = part + 32 * NW;            // 2 x rows reflectors (this one, the next)
        double2* wb = vb + 2 * rows;             // rows
        const int last = rows - 1 - lane;        // row of block t: last - 32 t
        int off[R];                              // (no such row: row 0, not stored)
#pragma unroll
        for (int t = 0; t < R; ++t) off[t] = max(last - 32 * t, 0);
#pragma unroll 1
        for (int i = tid; i < rows; i += NT) vb[rows + i] = wb[i] = zero;   // "reflector -1"
        int rb = 0, G = 0, myt = 0, myg = 0;     // row blocks in use, column classes, this warp's block and class
#pragma unroll 1
        for (int c = 0; c < n; ++c) {
            const double2* vk = vb + ((c + 1) & 1) * rows;
            double2* vc = vb + (c & 1) * rows;
            if (warp == (unsigned)(c + (int)b) % NW) {
                double2 x[R], w[R];
                double2* mc = M + c * ld;
                const int ic = rows - 1 - c;     // slot of row c
#pragma unroll
                for (int t = 0; t < R; ++t) x[t] = mc[off[t]];
                if (c > 0) {
                    const double2 tau = mc[c - ld];
                    double2 v[R];
                    double s = 0.0;
                    const double2* pt = part + lane;
#pragma unroll
                    for (int t = 0; t < R; ++t) {
                        v[t] = vk[off[t]];
                        w[t] = zero;
                    }
                    // (the loads of several classes in flight at sixteen warps,
                    // n = 108: 5.3 K -> 4.8 K cycles a step)
#pragma unroll (NW >= 16 ? 4 : NW >= 8 ? 2 : 1)
                    for (int g = 0; g < G; ++g, pt += 32 * rb)
#pragma unroll
                        for (int t = 0; t < R; ++t)
                            if (t < rb) w[t] = cadd(w[t], pt[32 * t]);
#pragma unroll
                    for (int t = 0; t < R; ++t)
                        s = fma(w[t].x, v[t].x, fma(w[t].y, v[t].y, s));
                    const double h = -0.5 * fma(tau.x, tau.x, tau.y * tau.y) * warp_sum(s);
#pragma unroll
                    for (int t = 0; t < R; ++t) {
                        w[t] = cmul(tau, w[t]);
                        w[t] = c2(fma(h, v[t].x, w[t].x), fma(h, v[t].y, w[t].y));
                        wb[off[t]] = w[t];       // (lanes without a row repeat row 0, long dead or theirs alone)
                    }
                    double2 wc = w[0];
#pragma unroll
                    for (int t = 1; t < R; ++t) if ((ic >> 5) == t) wc = w[t];
                    wc = shfl2(wc, ic & 31);
#pragma unroll
                    for (int t = 0; t < R; ++t) {
                        x[t] = csub(cfms_bc(x[t], v[t], wc), w[t]);          // v(c) = 1
                        if (SPEC && last - 32 * t >= n) mc[off[t]] = x[t];   // the final P of column c
                    }
                }
                // reflector c from column c
                double2 xc = x[0], alpha = x[0];
#pragma unroll
                for (int t = 1; t < R; ++t) {
                    if ((ic >> 5) == t) xc = x[t];
                    if (((ic - 1) >> 5) == t) alpha = x[t];
                }
                double beta = 0.0;
                if (c < n - 1) {
                    alpha = shfl2(alpha, (ic - 1) & 31);
                    double ss = 0.0;
#pragma unroll
                    for (int t = 0; t < R; ++t) {
                        const int i = last - 32 * t;
                        const bool in = i > c + 1 && (!SPEC || i < n);
                        x[t] = c2(in ? x[t].x : 0.0, in ? x[t].y : 0.0);
                        ss = fma(x[t].x, x[t].x, fma(x[t].y, x[t].y, ss));
                    }
                    ss = warp_sum(ss);
                    const double rest = fma(alpha.y, alpha.y, ss), nn = fma(alpha.x, alpha.x, rest);
                    // (the test comes after the reflector, out of its chain: N=54, batch 100, 1 %)
                    Reflector h = reflector(alpha, nn);
                    if (!squares_safe(rest, nn)) {
                        const double f = column_scale(nn);
                        const double2 as = cscale(alpha, f);
                        ss = 0.0;
#pragma unroll
                        for (int t = 0; t < R; ++t) {
                            const double2 y = cscale(x[t], f);
                            ss = fma(y.x, y.x, fma(y.y, y.y, ss));
                        }
                        const double rs = fma(as.y, as.y, warp_sum(ss));
                        h = reflector_scaled(alpha, as, rs, f);
                    }
                    beta = h.beta;
#pragma unroll
                    for (int t = 0; t < R; ++t) {
                        const int i = last - 32 * t;
                        x[t] = cmul(x[t], h.scal);
                        if (i >= 0) vc[i] = i == c + 1 ? c2(1.0, 0.0) : x[t];
                        if (i > c && (!SPEC || i < n)) mc[i] = i == c + 1 ? h.tau : x[t];
                    }
                }
                if (lane == (ic & 31)) de[c * des] = c2(xc.x, beta);
            }
            if (c >= n - 1) break;
            team_sync<NT, BLOCK>();
            // this warp's row block and columns, four of them at a time so
            // that their loads and chains overlap
            if (const int r = (rows - 1 - c + 31) >> 5; r != rb) {
                rb = r;
                G = NW / rb;
                myg = warp / rb;
                myt = warp - myg * rb;
            }
            if (myg < G) {
                const int i = last - 32 * myt, o = max(i, 0);
                const double2 v = vk[o], w = wb[o];
                double2 y = zero;
                int j = c + 1 + myg;
                const double2 *pv = vk + j, *pw = wb + j, *pn = vc + j;
                double2* q = M + o + j * ld;
                const int qs = G * ld;
#pragma unroll 1
                for (; j + 3 * G < n; j += 4 * G, q += 4 * qs, pv += 4 * G, pw += 4 * G, pn += 4 * G) {
                    double2 z[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) z[u] = q[u * qs];
#pragma unroll
                    for (int u = 0; u < 4; ++u) z[u] = cfms_bc(cfms_bc(z[u], v, pw[u * G]), w, pv[u * G]);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (i >= 0) q[u * qs] = z[u];
                        y = cfma(y, z[u], pn[u * G]);
                    }
                }
#pragma unroll 1
                for (; j < n; j += G, q += qs, pv += G, pw += G, pn += G) {
                    const double2 z = cfms_bc(cfms_bc(*q, v, *pw), w, *pv);
                    if (i >= 0) *q = z;
                    y = cfma(y, z, *pn);
                }
                part[32 * (myg * rb + myt) + lane] = y;
            }
            team_sync<NT, BLOCK>();
        }
        team_sync<NT, BLOCK>();
#pragma unroll 1
        for (int k = tid; k < n; k += NT) work[k] = de[k * des];
        phase_mark(4);
    phase();
        if constexpr (SPEC) {
            // rows of P Q (re, im of each of the three) for the divide and conquer
#pragma unroll 1
            for (int idx = tid; idx < 3 * n; idx += NT) {
                const int c = idx / n, j = idx - c * n;
                const double2 p = M[n + c + (size_t)j * ld];
                double* rj = dc.rows + kRowsTracked * j;
                rj[2 + 2 * c] = p.x;
                rj[3 + 2 * c] = p.y;
                if (c == 0) rj[0] = rj[1] = 0.0;
            }
        } else {
            // WY factors: block c (reflectors 8c .. 8c+7) is I - Y_c T_c Y_c^H
            // (zlarft, forward columnwise: T(l, l) = tau_l, T(0:l, l) =
            // -tau_l T(0:l, 0:l) Y^H y_l), G = Y^H Y first, one warp per block,
            // while Y is still in M.
#pragma unroll 1
            for (int c = warp; c < nblk; c += NW) {
                double gr[2] = {0.0, 0.0}, gi[2] = {0.0, 0.0};
                const int ky = 8 * c + fr;       // reflector of both fragments
#pragma unroll 1
                for (int kb = c; kb < nb; ++kb) {
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const int r = 8 * kb + 2 * fq + s;
                        const double2 yr = (ky >= nref || r <= ky || r >= n) ? zero
                                         : r == ky + 1 ? c2(1.0, 0.0) : M[r + (size_t)ky * ld];
                        zmma(gr, gi, cconj(yr), yr);
                    }
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int i = 2 * fq + e;
                    if (fr < i && 8 * c + i < nref) tpk[tidx(c, fr, i)] = c2(gr[e], gi[e]);
                }
                __syncwarp();
                const int mc = min(8, nref - 8 * c), l = lane;
                double2 trow[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    trow[i] = zero;
                    if (i < mc && l <= i) {
                        const int k = 8 * c + i;
                        const double2 ti = M[k + 1 + (size_t)k * ld];
                        if (l == i) {
                            trow[i] = ti;
                        } else {
                            double2 s0 = zero, s1 = zero;
#pragma unroll
                            for (int m = 0; m < i; ++m) {
                                if (m < l) continue;
                                const double2 gm = tpk[tidx(c, m, i)];
                                if (m & 1) s1 = cfma(s1, trow[m], gm); else s0 = cfma(s0, trow[m], gm);
                            }
                            trow[i] = cscale(cmul(ti, cadd(s0, s1)), -1.0);
                        }
                    }
                    __syncwarp();                 // column i of G read before T overwrites it
                    if (i < mc && l <= i) tpk[tidx(c, l, i)] = trow[i];
                }
                __syncwarp();
            }
            // reflectors into the lower triangle of U's block
#pragma unroll 1
            for (int k = warp; k < nref; k += NW)
#pragma unroll 1
                for (int i = k + 1 + lane; i < n; i += 32)
                    Ub[i + (size_t)k * n] = i == k + 1 ? c2(1.0, 0.0) : M[i + k * ld];
        }
        team_sync<NT, BLOCK>();
        phase_mark(9);
        // ---- a5b: divide and conquer; Z (real) and its workspace in M
        tridiag_dc<NT, NMAX, BLOCK, SPEC>(n, dc);
        // a failed eigensolve shows as a non-finite value (every warp looks at
        // all of them: the verdict is uniform without a barrier)
        bool bad = false;
#pragma unroll 1
        for (int i = lane; i < n; i += 32) bad |= !isfinite(dc.w[i]);
        if (__any_sync(0xffffffffu, bad)) code = kEigFailCode;
        phase_mark(5);
    phase();
    }

    if (code) {
        const double qnan = __longlong_as_double(0x7ff8000000000000LL);
        if constexpr (SPEC) {
#pragma unroll 1
            for (int e = tid; e < a.ne; e += NT) a.spec[(size_t)b * a.ne + e] = qnan;
        } else {
            team_sync<NT, BLOCK>();   // earlier writes to U's block come first
#pragma unroll 1
            for (size_t idx = tid; idx < nn; idx += NT) Ub[idx] = c2(qnan, qnan);
        }
        if (SPEC || a.stage >= 3) for (int i = tid; i < n; i += NT) Wb[i] = qnan;
        if (tid == 0) a.info[b] = code == kEigFailCode ? eig_fail_info(n) : code;
        return;
    }

    // ---- ascending eigenvalues
#pragma unroll 1
    for (int t = tid; t < n; t += NT) {
        const int slot = dc.ord[t];
        rank[slot] = t;
        Wb[t] = dc.w[slot];
    }

    if constexpr (SPEC) {
        // ---- spin-wave intensities: column jj of P Q Z = O U is Y = O u of
        // eigenvalue w[jj]. For each positive eigenvalue lambda, t = u /
        // sqrt(lambda) is the Bogoliubov vector of the mode of energy omega =
        // 1 / lambda; Y = O t (3 components) and
        // I = sum_ab (delta_ab - q_a q_b) conj(Y_a) Y_b = |Y|^2 - |q . Y|^2;
        // then S(E_e) = sum_modes I g(E_e - omega) with the Gaussian g.
        double* om = reinterpret_cast<double*>(M);
        double* it = om + n;
        const double q0 = __ldg(a.qhat + 3 * b), q1 = __ldg(a.qhat + 3 * b + 1), q2 = __ldg(a.qhat + 3 * b + 2);
#pragma unroll 1
        for (int jj = tid; jj < n; jj += NT) {
            const double lam = dc.w[jj];
            const double* yj = dc.rows + kRowsTracked * jj + 2;
            const double yy = fma(yj[0], yj[0], fma(yj[1], yj[1], fma(yj[2], yj[2], fma(yj[3], yj[3],
                              fma(yj[4], yj[4], yj[5] * yj[5])))));
            const double2 qy = c2(fma(q0, yj[0], fma(q1, yj[2], q2 * yj[4])),
                                  fma(q0, yj[1], fma(q1, yj[3], q2 * yj[5])));
            const bool pos = lam > 0.0;
            om[jj] = pos ? 1.0 / lam : -1.0;
            it[jj] = pos ? (yy - fma(qy.x, qy.x, qy.y * qy.y)) / lam : 0.0;
        }
        team_sync<NT, BLOCK>();
#pragma unroll 1
        for (int e = tid; e < a.ne; e += NT) {
            const double E = __ldg(a.energies + e);
            double acc = 0.0;
#pragma unroll 1
            for (int jj = 0; jj < n; ++jj) {
                if (!(om[jj] > 0.0)) continue;
                const double x = E - om[jj];
                acc = fma(it[jj], exp(-x * x * a.ginv2), acc);
            }
            a.spec[(size_t)b * a.ne + e] = acc * a.gnorm;
        }
        if (tid == 0) a.info[b] = 0;
        return;
    } else {
        // ---- a5c: V = Q Z in compact-WY blocks of 8 reflectors, last block
        // first, V = Q_0 (Q_1 (... Q_last Z)), and a6: U = X^H V. Warp p owns
        // the 8-column panels p, p + NW of V and takes them through both
        // without a CTA barrier; they share every fragment of Y and X, which
        // are read from U's block (L2). Per block: W1 = Y_c^H V_p, W2 = T_c W1,
        // V_p -= Y_c W2, the 8 x 8 intermediates turned from accumulator into
        // B-fragment layout by shuffles.
        {   // Z (real) -> V (complex) in place, through registers, the last
            // columns first (column j of V lies at or above Z's columns 2j, 2j + 1)
            constexpr int CU = 8, RB = (NMAX + 31) / 32;
#pragma unroll 1
            for (int j0 = (n - 1) / (CU * NW) * (CU * NW); j0 >= 0; j0 -= CU * NW) {
                double zr[CU][RB];
#pragma unroll
                for (int u = 0; u < CU; ++u)
#pragma unroll
                    for (int t = 0; t < RB; ++t) {
                        const int j = j0 + warp + NW * u, i = lane + 32 * t;
                        zr[u][t] = (j < n && i < n) ? dc.Z[i + j * ld] : 0.0;
                    }
                team_sync<NT, BLOCK>();
#pragma unroll
                for (int u = 0; u < CU; ++u)
#pragma unroll
                    for (int t = 0; t < RB; ++t) {
                        const int j = j0 + warp + NW * u, i = lane + 32 * t;
                        if (j < n && i < n) M[i + j * ld] = c2(zr[u][t], 0.0);
                    }
                team_sync<NT, BLOCK>();
            }
        }
        // accumulator (row fr, columns 2 fq + e) -> B fragment (row 2 fq + s, column fr)
        auto to_b = [&](const double (&re)[2], const double (&im)[2], int s) -> double2 {
            const int src = 4 * (2 * fq + s) + (fr >> 1);
            const double2 y0 = shfl2(c2(re[0], im[0]), src), y1 = shfl2(c2(re[1], im[1]), src);
            return (fr & 1) ? y1 : y0;
        };
        // Y_c(r, l) is at Ub[r + k n], k = 8c + l, for r > k; the tile row c is
        // masked and rows past n are zero (clamped reads)
        const int np = (nb - warp + NW - 1) / NW;   // panels of this warp
        double2* vp[PP];                            // panel columns: B fragment column fr
#pragma unroll
        for (int u = 0; u < PP; ++u) vp[u] = M + min(8 * (warp + NW * u) + fr, n - 1) * ld;
#pragma unroll 1
        for (int c = nblk - 1; c >= 0; --c) {
            double wr[PP][2], wi[PP][2];
#pragma unroll
            for (int u = 0; u < PP; ++u) wr[u][0] = wr[u][1] = wi[u][0] = wi[u][1] = 0.0;
            const int ky = 8 * c + fr;
            const double2* yc = Ub + min(ky, n - 1) * n;
            double2 yn[2];                       // the next tile's Y, loaded ahead
#pragma unroll
            for (int s = 0; s < 2; ++s) yn[s] = yc[min(8 * c + 2 * fq + s, n - 1)];
#pragma unroll 1
            for (int kb = c; kb < nb; ++kb) {    // W1 = Y_c^H V
                const double2 yl[2] = {yn[0], yn[1]};
                if (kb + 1 < nb) {
#pragma unroll
                    for (int s = 0; s < 2; ++s) yn[s] = yc[min(8 * kb + 8 + 2 * fq + s, n - 1)];
                }
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const int r = 8 * kb + 2 * fq + s, rc = min(r, n - 1);
                    const bool in = r > ky && r < n;
                    const double2 ya = c2(in ? yl[s].x : 0.0, in ? -yl[s].y : 0.0);
#pragma unroll
                    for (int u = 0; u < PP; ++u)
                        if (u < np) zmma(wr[u], wi[u], ya, vp[u][rc]);
                }
            }
            const double2* yr[2];                // A fragments of Y: column 8 c + 2 fq + s
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                yr[s] = Ub + min(8 * c + 2 * fq + s, n - 1) * n;
                yn[s] = yr[s][min(8 * c + fr, n - 1)];
            }
            double2 bw[PP][2];
#pragma unroll
            for (int u = 0; u < PP; ++u) {       // W2 = T_c W1, negated
                if (u >= np) continue;
                double tr[2] = {0.0, 0.0}, ti[2] = {0.0, 0.0};
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const int k = 2 * fq + s;
                    const double2 ta = (fr <= k && 8 * c + k < nref) ? tpk[tidx(c, fr, k)] : zero;
                    zmma(tr, ti, c2(-ta.x, -ta.y), to_b(wr[u], wi[u], s));
                }
#pragma unroll
                for (int s = 0; s < 2; ++s) bw[u][s] = to_b(tr, ti, s);
            }
#pragma unroll 1
            for (int t = c; t < nb; ++t) {       // V -= Y_c W2 (rows up to 8c get 0)
                const int r = 8 * t + fr;
                double2 ya[2];
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const bool in = t > c || r > 8 * c + 2 * fq + s;
                    ya[s] = c2(in ? yn[s].x : 0.0, in ? yn[s].y : 0.0);
                    if (t + 1 < nb) yn[s] = yr[s][min(r + 8, n - 1)];
                }
#pragma unroll
                for (int u = 0; u < PP; ++u) {
                    if (u >= np) continue;
                    const int j = 8 * (warp + NW * u) + 2 * fq;
                    double2* q = M + r + j * ld;
                    double vr[2], vi[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) { const double2 x = q[e * ld]; vr[e] = x.x; vi[e] = x.y; }
#pragma unroll
                    for (int s = 0; s < 2; ++s) zmma(vr, vi, ya[s], bw[u][s]);
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (r < n && j + e < n) q[e * ld] = c2(vr[e], vi[e]);
                }
            }
            __syncwarp();
        }
        phase_mark(6);
    phase();
        if (a.stage == 4) {
            // U(i, j) = sum_{k >= i} conj(X(k, i)) V(k, j), in place from the top:
            // row tile ti needs the rows of V from 8 ti on only
#pragma unroll 1
            for (int ti = 0; ti < nb; ++ti) {
                double ur[PP][2], ui[PP][2];
#pragma unroll
                for (int u = 0; u < PP; ++u) ur[u][0] = ur[u][1] = ui[u][0] = ui[u][1] = 0.0;
                const int i = 8 * ti + fr;
                const double2* xi = Ub + min(i, n - 1);
                double2 xn[2];                   // the next tile's X^H, loaded ahead
#pragma unroll
                for (int s = 0; s < 2; ++s) xn[s] = xi[min(8 * ti + 2 * fq + s, n - 1) * n];
#pragma unroll 1
                for (int kb = ti; kb < nb; ++kb) {
                    const double2 xl[2] = {xn[0], xn[1]};
                    if (kb + 1 < nb) {
#pragma unroll
                        for (int s = 0; s < 2; ++s) xn[s] = xi[min(8 * kb + 8 + 2 * fq + s, n - 1) * n];
                    }
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const int k = 8 * kb + 2 * fq + s, kc = min(k, n - 1);
                        const bool in = k >= i && k < n;
                        const double2 xa = c2(in ? xl[s].x : 0.0, in ? xl[s].y : 0.0);
#pragma unroll
                        for (int u = 0; u < PP; ++u)
                            if (u < np) zmma(ur[u], ui[u], xa, vp[u][kc]);
                    }
                }
                __syncwarp();
#pragma unroll
                for (int u = 0; u < PP; ++u) {
                    if (u >= np) continue;
                    const int j = 8 * (warp + NW * u) + 2 * fq;
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (i < n && j + e < n) M[i + (j + e) * ld] = c2(ur[u][e], ui[u][e]);
                }
                __syncwarp();
            }
        }
        team_sync<NT, BLOCK>();   // the last reads of X and Y from U's block come before its results
        phase_mark(7);
        // ---- a7: store V or U, column j to position rank[j]
#pragma unroll 1
        for (int jj = warp; jj < n; jj += NW) {
            double2* uo = Ub + (size_t)rank[jj] * n;
#pragma unroll 1
            for (int i = lane; i < n; i += 32) uo[i] = M[i + (size_t)jj * ld];
        }
        if (tid == 0) a.info[b] = 0;
    }
}

}  // namespace cta
}  // namespace sgeig
