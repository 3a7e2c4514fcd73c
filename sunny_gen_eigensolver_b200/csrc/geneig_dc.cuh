// Divide-and-conquer eigensolver for the real symmetric tridiagonal matrix
// T = tridiag(e, d, e), one team of threads.
//
// Method (Cuppen's divide and conquer with the Gu-Eisenstat correction, the
// algorithm of LAPACK dstedc / dlaed0-dlaed4):
//   * T is torn at every multiple k of kLeaf in [1, n): d[k-1] and d[k] each
//     lose |e[k-1]|, so that T = blockdiag(T1', T2') + |e| v v^T with
//     v = e_{k-1} + sign(e) e_k.
//   * Leaves (kLeaf rows) are solved by the implicit QL iteration (Wilkinson
//     shift, as EISPACK imtql2), eight lanes per leaf: every lane runs the
//     same scalar recurrence on its own copy of d and e and keeps one row of
//     the leaf's eigenvectors, so a leaf needs no communication. Blocks are then merged
//     bottom-up: level `half` merges [a, a+half) with [a+half, a+2*half).
//   * A merge forms z = (last row of Q1, sign(e) * first row of Q2)/sqrt(2),
//     rho = 2|e|, deflates entries with rho|z_j| <= tol and pairs of nearly
//     equal poles (Givens rotation of the two eigenvector columns), solves the
//     secular equation 1 + rho sum_j z_j^2/(d_j - lambda) = 0 for the K
//     remaining roots (P lanes per root), recomputes z from the computed
//     roots with Loewner's formula so that the new eigenvectors are orthogonal
//     to working precision, and multiplies the old eigenvector columns by the
//     K x K eigenvector matrix of the rank-one problem. Rows of the first half
//     only meet columns of the first half (the others are zero there) unless
//     a rotation has mixed the halves, so the product runs over half of K.
// The secular solver is this file's own: each root is bracketed between its
// two poles, measured from the nearer pole (so that every d_j - lambda is
// formed without cancellation), and iterated with a two-pole rational model
// (fit value and slope of the left and right partial sums at the current
// point, solve the resulting quadratic), safeguarded by bisection.
//
// Output: Z (n x n, column slot j holds the eigenvector of w[j]); w[] in the
// caller's units; ord[t] the slot of the t-th smallest eigenvalue.
//
// NMAX > 0 bounds n at compile time (Z, U in shared memory; merge products
// accumulate in registers). NMAX == 0 is the any-n form for matrices kept in
// global memory: merges wider than 32 columns are 16 x 16 FP64 tensor-core
// tiles written to the separate buffer Zo and copied back.
//
// ROWS: instead of Z, the caller wants only a few combinations of Z's rows
// (R Z for 6 real rows R). Then only those rows and the first and last row of
// every block are carried through the merges (kRowsTracked doubles per column
// slot), which needs neither Z nor U and replaces the O(n^3) merge products by
// O(n^2) ones.
#pragma once

#include "geneig_common.cuh"

namespace sgeig {

constexpr int kLeaf = 8;          // rows of a leaf
constexpr int kLeafStride = 25;   // d, e and a row of z of a lane's leaf (odd: no bank conflicts)
// Off-diagonals of the scaled T (max |T_ij| in [0.5, 1)) up to this are zero to
// a leaf whatever its diagonal is, and so is a rotation's pair whose squares sum
// to less than 2^-996 (1e-300): squares that underflow lose the rotation's bits,
// and beside a zero diagonal nothing is negligible by comparison.
constexpr double kLeafTiny = 0x1p-332;
constexpr int kRowsTracked = 8;   // ROWS: first row, last row, 6 caller rows per column slot

struct DCShared {
    double* Z;  int ldz;    // eigenvectors
    double* U;  int ldu;    // K x K blocks of each merge at [a, a+K)^2
    double* Zo;             // NMAX == 0 only: n x ldz product buffer of the merge GEMMs
    const double* d; int ds;  // diagonal, element i at d[i * ds]
    const double* e; int es;  // off-diagonal, element i at e[i * es]
    double* w;              // eigenvalue of column slot j
    double* z;              // merge z-vector by column slot
    double* dl;             // non-deflated poles [a, a+K), ascending
    double* zz;             // their z
    double* zh;             // Loewner z-hat
    double* rt;             // root offsets from their origin pole
    double* rho;            // rho per merge, indexed by a
    double* leaf;           // kLeafStride doubles for each of leaf_lanes lanes (may overlap Z)
    int leaf_lanes;         // multiple of kLeaf; fewer than n: several passes, which must not overlap Z
    double* rows;           // ROWS only: rows[kRowsTracked * slot + r]
    int* org;               // origin pole (merge-local index) of each root
    int* nd;                // column slots of a merge: the K non-deflated ones ascending, then the deflated ones
    int* perm;              // ascending order of the merge's poles before deflation
    int* ord;               // ascending order of each block's eigenvalues
    int* kl;                // non-deflated (position | slot << 16): first-half slots, then second-half slots
    int* kcnt;              // per merge at a: K (-1: ord is current), K of the first half, rotated flag
};

// Number of doubles / ints of scratch DCShared needs for size n (excluding Z, U, rows).
__host__ __device__ inline int dc_vec_doubles(int n) { return 7 * n + 1; }
__host__ __device__ inline int dc_vec_ints(int n) { return 6 * n; }

__host__ __device__ constexpr int dc_leaf_doubles(int n) { return kLeafStride * kLeaf * ((n + kLeaf - 1) / kLeaf); }

// Points the scratch members at `dbl` (dc_vec_doubles(n), eigenvalues first)
// and `ints` (dc_vec_ints(n)).
__host__ __device__ inline void dc_carve(DCShared& s, double* dbl, int* ints, int n) {
    s.w = dbl; s.z = s.w + n; s.dl = s.z + n; s.zz = s.dl + n; s.zh = s.zz + n; s.rt = s.zh + n; s.rho = s.rt + n;
    s.org = ints; s.nd = s.org + n; s.perm = s.nd + n; s.ord = s.perm + n; s.kl = s.ord + n; s.kcnt = s.kl + n;
}

// Sum over the P consecutive lanes that share one root (P = 1, 2 or 4); on
// the host (P = 1) it is the identity. Every lane ends with the same value
// (the butterfly adds the same pairs in the same order up to commutation).
template <int P>
__host__ __device__ __forceinline__ double lanes_sum(double v, unsigned mask) {
#ifdef __CUDA_ARCH__
    if (P >= 2) v += __shfl_xor_sync(mask, v, 1);
    if (P >= 4) v += __shfl_xor_sync(mask, v, 2);
#else
    (void)mask;
#endif
    return v;
}
template <int P>
__host__ __device__ __forceinline__ double lanes_prod(double v, unsigned mask) {
#ifdef __CUDA_ARCH__
    if (P >= 2) v *= __shfl_xor_sync(mask, v, 1);
    if (P >= 4) v *= __shfl_xor_sync(mask, v, 2);
#else
    (void)mask;
#endif
    return v;
}

// Root i (0-based) of 1 + rho sum_j zz_j^2 / (dl_j - x) = 0 with dl ascending,
// rho > 0, sum zz_j^2 <= 1 to rounding, computed by P lanes together (lane qq
// sums the terms j = qq mod P). Returns the offset tau of the root from pole
// `org`; the return value is the number of iterations taken.
// The last root (no pole to its right, bracket rho long) takes the same path
// with that pole's weight zero. Every sum runs over all poles with the left
// ones' share picked by a select, so the lanes of a warp, which hold different
// roots, do not diverge (N=54, one pencil on an SM, the three levels: 47.9 K
// cycles, 64.0 K with two loops that meet at pole i).
template <int P>
__host__ __device__ inline int secular_root_p(int i, int K, const double* dl, const double* zz, double rho,
                                              int qq, unsigned mask, double& tau_out, int& org_out) {
    if (K == 1) { org_out = 0; tau_out = rho * zz[0] * zz[0]; return 0; }
    const bool right = i < K - 1;
    const int ir = right ? i + 1 : i;
    const double di = dl[i], gap = dl[ir] - di;
    const double mid = 0.5 * (right ? gap : rho * (1.0 + 1e-10));
    double gs = 0.0;
#pragma unroll 2
    for (int j = qq; j < K; j += P) {
        const double zj = zz[j];
        gs = fma(zj, zj * fast_rcp((dl[j] - di) - mid), gs);
    }
    const double gm = fma(rho, lanes_sum<P>(gs, mask), 1.0);
    const bool low = !right || gm >= 0.0;
    const int o = low ? i : ir;
    double lo = low ? 0.0 : -mid, hi = low ? (right ? mid : 2.0 * mid) : 0.0, tau = low ? hi : lo;
    const double dlo = dl[o];
    const double p = di - dlo, q = dl[ir] - dlo;       // one of them is 0
    {
        // Starting point: the two nearest poles' terms exactly, the others
        // frozen at their midpoint value c (the fixed-weight start), i.e. the
        // root of c + a/(p - x) + b/(q - x) in origin coordinates, taken when
        // it lies inside the bracket (otherwise the bracket's end stays).
        const double a = rho * zz[i] * zz[i], b = right ? rho * zz[ir] * zz[ir] : 0.0;
        const double c = fma(a - b, fast_rcp(mid), gm);
        const double B = -(c * (p + q) + a + b), C = a * q + b * p;
        if (c != 0.0) {
            double disc = B * B - 4.0 * c * C;
            if (disc < 0.0) disc = 0.0;
            const double qq2 = -0.5 * (B + copysign(sqrt(disc), B));
            const double x1 = qq2 * fast_rcp(c), x2 = (qq2 != 0.0) ? C * fast_rcp(qq2) : x1;
            if (x1 > lo && x1 < hi) tau = x1;
            else if (x2 > lo && x2 < hi) tau = x2;
        }
    }
    int it = 0;
    for (; it < 80; ++it) {
        // sums over all poles, and over those up to i (left of the root)
        double tot = 0.0, dtot = 0.0, psi = 0.0, dpsi = 0.0;
#pragma unroll 2
        for (int j = qq; j < K; j += P) {
            const double zj = zz[j];
            const double t = zj * fast_rcp((dl[j] - dlo) - tau);
            const double tl = j <= i ? t : 0.0;
            tot = fma(zj, t, tot);
            dtot = fma(t, t, dtot);
            psi = fma(zj, tl, psi);
            dpsi = fma(tl, tl, dpsi);
        }
        tot = rho * lanes_sum<P>(tot, mask);
        dtot = rho * lanes_sum<P>(dtot, mask);
        psi = rho * lanes_sum<P>(psi, mask);
        dpsi = rho * lanes_sum<P>(dpsi, mask);
        const double phi = tot - psi, dphi = dtot - dpsi;      // psi <= 0 <= phi
        const double g = 1.0 + tot;
        const double err = kEps * (2.0 + 8.0 * (phi - psi) + 3.0 * fabs(tau) * dtot);
        if (fabs(g) <= err) break;
        if (g < 0.0) lo = tau; else hi = tau;
        if (hi - lo <= 2.0 * kEps * fmax(fabs(lo), fabs(hi))) break;
        const double bpsi = dpsi * (p - tau) * (p - tau);
        const double apsi = psi - dpsi * (p - tau);
        const double bphi = right ? dphi * (q - tau) * (q - tau) : 0.0;
        const double aphi = right ? phi - dphi * (q - tau) : 0.0;
        const double c = 1.0 + apsi + aphi;
        // c + bpsi/(p - x) + bphi/(q - x) = 0 in origin coordinates
        // (one of p, q is 0, so p q = 0):
        //   c x^2 - (c (p + q) + bpsi + bphi) x + (bpsi q + bphi p) = 0
        const double B = -(c * (p + q) + bpsi + bphi);
        const double C = bpsi * q + bphi * p;
        double tn;
        if (c == 0.0) {
            tn = -C * fast_rcp(B);
        } else {
            double disc = B * B - 4.0 * c * C;
            if (disc < 0.0) disc = 0.0;
            const double qq2 = -0.5 * (B + copysign(sqrt(disc), B));
            const double x1 = qq2 * fast_rcp(c), x2 = (qq2 != 0.0) ? C * fast_rcp(qq2) : x1;
            tn = (x1 > lo && x1 < hi) ? x1 : x2;
        }
        // converged when the model step is within a few ulps of the iterate
        // (it may then round just outside the bracket)
        if (fabs(tn - tau) <= 4.0 * kEps * fabs(tau)) {
            if (tn > lo && tn < hi) tau = tn;
            break;
        }
        if (!(tn > lo && tn < hi) || it >= 30) tn = 0.5 * (lo + hi);
        if (tn == tau) break;
        tau = tn;
    }
    tau_out = tau;
    org_out = o;
    return it;
}

// Phase E of a level for NMAX > 0: the merges' products on the FP64 tensor
// cores (mma.m8n8k4.f64), a warp per 8-row tile with all K columns of the
// result in registers, so that the tile is read (and its old columns used up)
// before the same warp overwrites it, without a barrier. A row tile lies in
// one half of its merge (half is a multiple of 8), so its k loop runs over the
// columns of that half only, unless a rotation mixed them. Columns past K are
// computed from whatever lies there and not stored.
template <int NT, int NMAX, int BLOCK = NT>
__device__ __forceinline__ void dc_merge_panels(int n, int half, int span, const DCShared& s) {
    const int lane = team_tid<NT, BLOCK>() & 31, warp = team_tid<NT, BLOCK>() >> 5;
    constexpr int NW = NT / 32, NB = NMAX / 8;
    const int fr = lane >> 2, fq = lane & 3;
#pragma unroll 1
    for (int r0 = 8 * warp; r0 < n; r0 += 8 * NW) {
        const int a = r0 - r0 % span;
        const int K = a + half < n ? s.kcnt[a] : 0;
        if (K == 0) continue;
        const int K1 = s.kcnt[a + 1], r = r0 + fr;
        const bool dense = s.kcnt[a + 2] != 0, upper = r0 - a < half;
        const int k0 = (dense || upper) ? 0 : K1, k1 = (dense || !upper) ? K : K1;
        const int* kl = s.kl + a;
        const double* zr = s.Z + min(r, n - 1);
        const double* uc = s.U + a + (size_t)(a + fr) * s.ldu;
        double acc[NB][2];
#pragma unroll
        for (int t = 0; t < NB; ++t) acc[t][0] = acc[t][1] = 0.0;
#pragma unroll 1
        for (int k = k0; k < k1; k += 4) {
            const int ka = k + fq;
            const int ps = kl[min(ka, k1 - 1)];
            double av = zr[(size_t)(ps >> 16) * s.ldz];
            if (ka >= k1) av = 0.0;
            const double* ur = uc + (ps & 0xffff);
#pragma unroll
            for (int t = 0; t < NB; ++t) {
                if (8 * t >= K) continue;
                const double bv = ur[(size_t)(8 * t) * s.ldu];
                asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                    : "+d"(acc[t][0]), "+d"(acc[t][1]) : "d"(av), "d"(bv));
            }
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < NB; ++t) {
            const int j = 8 * t + 2 * fq;
            if (r < n && j < K) s.Z[r + (size_t)s.nd[a + j] * s.ldz] = acc[t][0];
            if (r < n && j + 1 < K) s.Z[r + (size_t)s.nd[a + j + 1] * s.ldz] = acc[t][1];
        }
    }
}

// Phase E of a level of merges at most 4 * UMAX columns wide: four lanes per
// row, lane q accumulating output columns j = q + 4u in registers. A row's
// reads and writes stay within its quad, so no barrier is needed between them.
template <int NT, int UMAX, int BLOCK = NT>
__device__ __forceinline__ void dc_merge_rows_regs(int n, int half, int span, const DCShared& s) {
    for (int p0 = 0; p0 < 4 * n; p0 += NT) {
        const int pidx = p0 + team_tid<NT, BLOCK>();
        const int r = pidx >> 2, part = pidx & 3;
        const int a = (r < n) ? r - r % span : n;
        const bool active = r < n && a + half < n && s.kcnt[a] > 0;
        const int K = active ? s.kcnt[a] : 0;
        double acc[UMAX];
#pragma unroll
        for (int u = 0; u < UMAX; ++u) acc[u] = 0.0;
        for (int l = 0; l < K; ++l) {
            const double x = s.Z[r + (size_t)s.nd[a + l] * s.ldz];
            const double* ur = s.U + (a + l) + (size_t)(a + part) * s.ldu;
#pragma unroll
            for (int u = 0; u < UMAX; ++u)
                if (part + 4 * u < K) acc[u] = fma(x, ur[(size_t)(4 * u) * s.ldu], acc[u]);
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < UMAX; ++u) {
            const int j = part + 4 * u;
            if (j < K) s.Z[r + (size_t)s.nd[a + j] * s.ldz] = acc[u];
        }
    }
}

// Phase E for any merge width (NMAX == 0): for every merge [a, a+m) of the
// level, the m x K product Z(a:a+m, nd) * U on the FP64 tensor cores in
// 16 x 16 warp tiles (2 x 2 mma.m8n8k4 tiles), rows outside [a, a+m) being
// zero in those columns. Tiles are dealt round-robin to the warps across all
// merges of the level; products go to Zo, then back into Z after a barrier.
// Each half's rows take that half's columns only, as in dc_merge_panels, and
// operands are clamped, not masked (n = 216: 16.06 -> 15.72 ms a solve of 444).
template <int NT, int BLOCK = NT>
__device__ __forceinline__ void dc_merge_tiled(int n, int half, int span, const DCShared& s) {
    const int lane = team_tid<NT, BLOCK>() & 31, warp = team_tid<NT, BLOCK>() >> 5;
    constexpr int NW = NT / 32;
    int dealt = 0;
    for (int a = 0; a + half < n; a += span) {
        const int K = s.kcnt[a];
        if (K == 0) continue;
        const int m = min(span, n - a);
        const int tn = (K + 15) >> 4, T = ((m + 15) >> 4) * tn;
        const int K1 = s.kcnt[a + 1];
        const bool dense = s.kcnt[a + 2] != 0;
        const int *nd = s.nd + a, *kl = s.kl + a;
        const double* Ub = s.U + a + (size_t)a * s.ldu;
        int t = (warp - dealt % NW + NW) % NW;
        for (; t < T; t += NW) {
            const int ti = t / tn, tj = t - ti * tn;
            const int r0 = 16 * ti + (lane >> 2), j0 = 16 * tj + (lane >> 2);
            double acc[2][2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int g = 0; g < 2; ++g) acc[h][g][0] = acc[h][g][1] = 0.0;
            // only the poles of the tile's own half have nonzeros in its rows
            // (half is a multiple of 16 here), unless a rotation mixed the two
            const bool upper = 16 * ti < half;
            const int k0 = (dense || upper) ? 0 : K1, k1 = (dense || !upper) ? K : K1;
            const double* z0 = s.Z + a + min(r0, m - 1);
            const double* z1 = s.Z + a + min(r0 + 8, m - 1);
            const double* u0 = Ub + (size_t)min(j0, K - 1) * s.ldu;
            const double* u1 = Ub + (size_t)min(j0 + 8, K - 1) * s.ldu;
#pragma unroll 4
            for (int k = k0; k < k1; k += 4) {
                const int ka = k + (lane & 3), ps = kl[min(ka, k1 - 1)], pos = ps & 0xffff;
                const size_t zo = (size_t)(ps >> 16) * s.ldz;
                double av[2] = {z0[zo], z1[zo]};
                const double bv[2] = {u0[pos], u1[pos]};
                if (ka >= k1) av[0] = av[1] = 0.0;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int g = 0; g < 2; ++g)
                        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                            : "+d"(acc[h][g][0]), "+d"(acc[h][g][1]) : "d"(av[h]), "d"(bv[g]));
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = 16 * ti + 8 * h + (lane >> 2);
                if (r >= m) continue;
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const int j = 16 * tj + 8 * g + 2 * (lane & 3);
                    if (j < K) s.Zo[a + r + (size_t)nd[j] * s.ldz] = acc[h][g][0];
                    if (j + 1 < K) s.Zo[a + r + (size_t)nd[j + 1] * s.ldz] = acc[h][g][1];
                }
            }
        }
        dealt += T;
    }
    team_sync<NT, BLOCK>();
    const int width = min(span, n);
    for (int idx = team_tid<NT, BLOCK>(); idx < n * width; idx += NT) {
        const int jj = idx / n, r = idx - jj * n;
        const int a = r - r % span;
        if (a + half >= n || jj >= s.kcnt[a]) continue;
        const size_t o = r + (size_t)s.nd[a + jj] * s.ldz;
        s.Z[o] = s.Zo[o];
    }
}

// Implicit QL with Wilkinson shift on a leaf of m <= kLeaf rows: d, e (e[i]
// couples i and i+1) and one row z of the eigenvector matrix, all private to
// the calling lane (shared memory: the indices are data-dependent); every
// lane of the leaf's group runs the same recurrence on the same data. Returns
// false when it did not converge (non-finite input).
__device__ __forceinline__ bool leaf_ql(int m, double* d, double* e, double* z) {
    unsigned small = ~0u << (m - 1);                           // bit i: e[i] is negligible
#pragma unroll 1
    for (int i = 0; i < m - 1; ++i)
        if (fabs(e[i]) <= kEps * (fabs(d[i]) + fabs(d[i + 1])) + kLeafTiny) small |= 1u << i;
#pragma unroll 1
    for (int it = 0; it < 30 * kLeaf; ++it) {
        if (small == ~0u) return true;
        const int l = __ffs(~small) - 1;                       // first off-diagonal left
        const int top = l + __ffs(small >> l) - 1;             // its block is [l, top]
        const double dl = d[l], el = e[l];
        const double hd = 0.5 * (d[l + 1] - dl);
        double dnext = d[top], znext = z[top];
        const double h2 = fma(hd, hd, el * el);
        const double qs = hd + copysign(h2 > 0.0 ? h2 * rsqrt(h2) : 0.0, hd);
        double g = dnext - dl + (qs != 0.0 ? el * el * fast_rcp(qs) : 0.0);
        double s = 1.0, c = 1.0, p = 0.0, dabove = 0.0;        // |d| above the last rotation, with the floor
        int i = top - 1;
#pragma unroll 1
        for (; i >= l; --i) {
            const double ei = e[i], di = d[i], zi = z[i];
            const double f = s * ei, b = c * ei;
            const double q = fma(f, f, g * g);
            // the chase ended early: the block splits here (never at the first
            // rotation, whose f is above kLeafTiny)
            if (__double2hiint(q) < 0x01b00000) break;
            const double inv = rsqrt(q), en = q * inv;
            e[i + 1] = en;
            s = f * inv;
            c = g * inv;
            g = dnext - p;
            const double r = fma(di - g, s, 2.0 * c * b);
            p = s * r;
            const double dn = g + p;
            d[i + 1] = dn;
            g = fma(c, r, -b);
            z[i + 1] = fma(s, zi, c * znext);
            znext = fma(c, zi, -s * znext);
            dnext = di;
            // e[i + 1] against its new neighbours (not for the first
            // rotation: e[top] is outside the block)
            if (i + 1 < top && en <= kEps * (fabs(dn) + dabove)) small |= 2u << i;
            dabove = fabs(dn) + kLeafTiny / kEps;
        }
        const double dn = dnext - p;
        z[i + 1] = znext;
        d[i + 1] = dn;
        if (i < l) {
            e[l] = g;
            if (fabs(g) <= kEps * (fabs(dn) + dabove)) small |= 1u << l;
        } else {
            e[i] *= c;                                         // the last rotation's share
            e[i + 1] = 0.0;
            small |= 2u << i;
        }
        e[top] = 0.0;
    }
    return false;
}

// One warp: ord[a, b), the ascending order of a block, from its last merge
// (nothing to do when it has had none since ord was written). Roots and
// deflated values are two ascending lists, merged by binary search, unless a
// rotation changed deflated values (then by counting). The counts form a
// permutation for finite values; with NaN they may collide, which leaves
// stale but valid slots of the block in ord.
__device__ __forceinline__ void dc_order(int a, int b, const DCShared& s, int lane) {
    const int K = s.kcnt[a];
    if (K < 0) return;
    const int m = b - a;
    const int* nd = s.nd + a;
    const bool rotated = s.kcnt[a + 2] != 0;
    for (int t = lane; t < m; t += 32) {
        const int slot = nd[t];
        const double key = order_key(s.w[slot]);
        int pos;
        if (rotated) {
            pos = 0;
            for (int q = 0; q < m; ++q) {
                const double kq = order_key(s.w[nd[q]]);
                pos += (kq < key) || (kq == key && q < t);
            }
        } else {
            // first element of the other list that goes after this one
            int lo = t < K ? K : 0, hi = t < K ? m : K;
            const int lo0 = lo;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                const double km = order_key(s.w[nd[mid]]);
                if (t < K ? km < key : km <= key) lo = mid + 1; else hi = mid;
            }
            pos = (lo - lo0) + (t < K ? t : t - K);
        }
        s.ord[a + pos] = slot;
    }
}

// All NT threads of the team call this. n >= 1. On return Z (or rows), w and
// ord hold the eigen-decomposition of the tridiagonal (d, e), which is only
// read. ROWS: on entry rows[kRowsTracked * j + 2 ..] hold the six caller rows
// R (R[.][j]) and Z is scratch for the leaves (at least n x kLeaf, ldz >= n).
template <int NT, int NMAX, int BLOCK = NT, bool ROWS = false>
__device__ void tridiag_dc(int n, DCShared s) {
    const int tid = team_tid<NT, BLOCK>(), lane = tid & 31, warp = tid >> 5;
    constexpr int NW = NT / 32;
    // lanes per secular root and rank-one column: as many as let one pass of
    // the team cover every root (more lanes shorten each root's term loop)
    constexpr int P = NMAX == 0 || NT >= 4 * NMAX ? 4 : NT >= 2 * NMAX ? 2 : 1;

    // ---- scale T by a power of two so that max |T_ij| is in [0.5, 1); every
    // warp finds the scale by itself (no barrier)
    double sc = 1.0;
    {
        double mx = 0.0;
#pragma unroll 1
        for (int i = lane; i < n; i += 32) mx = fmax(mx, fabs(s.d[(size_t)i * s.ds]));
#pragma unroll 1
        for (int i = lane; i < n - 1; i += 32) mx = fmax(mx, fabs(s.e[(size_t)i * s.es]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (mx > 0.0 && isfinite(mx)) {
            int ex = 0;
            frexp(mx, &ex);
            sc = ldexp(1.0, -ex);
        }
    }
    // ---- leaves: torn at multiples of kLeaf, solved by eight lanes each, as
    // many at a time as the leaf buffer holds
    const int lanes = min(s.leaf_lanes, NT) & ~(kLeaf - 1);
#pragma unroll 1
    for (int f0 = 0; f0 * kLeaf < n; f0 += lanes / kLeaf) {
        const int f = f0 + tid / kLeaf, o = f * kLeaf, m = min(kLeaf, n - o), r = tid % kLeaf;
        const bool mine = tid < lanes && o < n;
        double zr[kLeaf], dr = 0.0;
        int pos = 0;
        if (mine) {
            double* d = s.leaf + tid * kLeafStride;
            double* e = d + kLeaf;
            double* z = e + kLeaf;
            bool ok = true;
#pragma unroll 1
            for (int i = 0; i < m; ++i) {
                double di = s.d[(o + i) * s.ds] * sc, ei = i < m - 1 ? s.e[(o + i) * s.es] * sc : 0.0;
                if (i == 0 && o > 0) di -= fabs(s.e[(o - 1) * s.es] * sc);
                if (i == kLeaf - 1 && o + kLeaf < n) di -= fabs(s.e[(o + i) * s.es] * sc);
                ok = ok && isfinite(di) && isfinite(ei);
                d[i] = di;
                e[i] = ei;
                z[i] = i == r ? 1.0 : 0.0;
            }
            if (ok) ok = leaf_ql(m, d, e, z);
            if (!ok) for (int i = 0; i < m; ++i) d[i] = __longlong_as_double(0x7ff8000000000000LL);
            if (r < m) {
                dr = d[r];
                const double key = order_key(dr);
#pragma unroll 1
                for (int i = 0; i < m; ++i) {
                    const double ki = order_key(d[i]);
                    pos += (ki < key) || (ki == key && i < r);
                }
            }
#pragma unroll
            for (int i = 0; i < kLeaf; ++i) zr[i] = i < m ? z[i] : 0.0;
        }
        if (lanes >= n) team_sync<NT, BLOCK>();               // every leaf is done before Z overwrites the buffer
        if (!ROWS && f0 == 0) {
#pragma unroll 1
            for (int j = warp; j < n; j += NW)
#pragma unroll 1
                for (int i = lane; i < n; i += 32)
                    if ((i ^ j) >= kLeaf) s.Z[i + (size_t)j * s.ldz] = 0.0;   // outside the leaves' blocks
        }
        if (mine && r < m) {
            s.ord[o + pos] = o + r;
            s.w[o + r] = dr;
            if (r == 0) s.kcnt[o] = -1;
#pragma unroll
            for (int i = 0; i < kLeaf; ++i) {
                if (i >= m) continue;
                s.Z[o + r + (size_t)(ROWS ? i : o + i) * s.ldz] = zr[i];
                if (ROWS) {
                    if (r == 0) s.rows[kRowsTracked * (o + i)] = zr[i];
                    if (r == m - 1) s.rows[kRowsTracked * (o + i) + 1] = zr[i];
                }
            }
        }
    }
    team_sync<NT, BLOCK>();
    if constexpr (ROWS) {
        // the caller's rows times the leaves' eigenvectors
        constexpr int RQ = (6 * NMAX + NT - 1) / NT;
        double v[RQ];
#pragma unroll
        for (int u = 0; u < RQ; ++u) {
            const int idx = tid + NT * u, j = idx / 6, q = idx - 6 * j;
            v[u] = 0.0;
            if (j < n) {
                const int o = j & ~(kLeaf - 1), m = min(kLeaf, n - o);
#pragma unroll 1
                for (int r = 0; r < m; ++r)
                    v[u] = fma(s.rows[kRowsTracked * (o + r) + 2 + q], s.Z[o + r + (size_t)(j - o) * s.ldz], v[u]);
            }
        }
        team_sync<NT, BLOCK>();
#pragma unroll
        for (int u = 0; u < RQ; ++u) {
            const int idx = tid + NT * u, j = idx / 6, q = idx - 6 * j;
            if (j < n) s.rows[kRowsTracked * j + 2 + q] = v[u];
        }
        team_sync<NT, BLOCK>();
    }
    phase_mark(10);

#pragma unroll 1
    for (int half = kLeaf;; half <<= 1) {
        const int span = half << 1;
        // ---- phase A: one warp per merge: order, z, deflation (after the
        // last merge only the order of the whole)
#pragma unroll 1
        for (int a = warp * span; a < n; a += NW * span) {
            const int k = a + half;
            const int b = min(a + span, n);
            const int m = b - a;
#pragma unroll 1
            for (int h0 = a; h0 < b; h0 += half) dc_order(h0, min(h0 + half, b), s, lane);
            if (k >= n) {
                __syncwarp();
                if (lane == 0) s.kcnt[a] = -1;
                continue;
            }
#pragma unroll 1
            for (int t = lane; t < m; t += 32) s.perm[a + t] = a + t;
            __syncwarp();
            // ascending order of the merged poles: two ascending lists
#pragma unroll 1
            for (int t = lane; t < m; t += 32) {
                const bool first = t < half;
                const int slot = s.ord[a + t];
                const double key = order_key(s.w[slot]);
                int lo = first ? half : 0, hi = first ? m : half;
                const int lo0 = lo;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    const double km = order_key(s.w[s.ord[a + mid]]);
                    if (first ? km < key : km <= key) lo = mid + 1; else hi = mid;
                }
                s.perm[a + (lo - lo0) + (first ? t : t - half)] = slot;
            }
            const double er = s.e[(size_t)(k - 1) * s.es] * sc;
            const double sgn = er < 0.0 ? -1.0 : 1.0;
            const double rho = 2.0 * fabs(er);
            double mx = 0.0;
#pragma unroll 1
            for (int j = a + lane; j < b; j += 32) {
                double zj;
                if constexpr (ROWS) {
                    // last row of the first half, first row of the second; the
                    // merged block's first (last) row is zero in the second
                    // (first) half's columns
                    double* rj = s.rows + kRowsTracked * j;
                    zj = (j < k ? rj[1] : sgn * rj[0]) * 0.70710678118654752440;
                    rj[j < k ? 1 : 0] = 0.0;
                } else {
                    zj = (j < k ? s.Z[(k - 1) + (size_t)j * s.ldz] : sgn * s.Z[k + (size_t)j * s.ldz]) *
                         0.70710678118654752440;
                }
                s.z[j] = zj;
                mx = fmax(mx, fmax(fabs(zj), fabs(s.w[j])));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const double tol = 8.0 * kEps * mx;
            __syncwarp();
            // keep entries with rho|z| > tol, in ascending order (none when
            // the tear is zero): counts first, then the lists
            int K0 = 0, K1 = 0;
#pragma unroll 1
            for (int t0 = 0; t0 < m; t0 += 32) {
                const int t = t0 + lane;
                const int j = t < m ? s.perm[a + t] : a;
                const bool keep = t < m && rho * fabs(s.z[j]) > tol;
                const unsigned mask = __ballot_sync(0xffffffffu, keep);
                const unsigned mask1 = __ballot_sync(0xffffffffu, keep && j < k);
                K0 += __popc(mask);
                K1 += __popc(mask1);
            }
            int base = 0, base1 = 0;
#pragma unroll 1
            for (int t0 = 0; t0 < m; t0 += 32) {
                const int t = t0 + lane;
                const int j = t < m ? s.perm[a + t] : a;
                const bool keep = t < m && rho * fabs(s.z[j]) > tol;
                const unsigned mask = __ballot_sync(0xffffffffu, keep);
                const unsigned mask1 = __ballot_sync(0xffffffffu, keep && j < k);
                const unsigned below = (1u << lane) - 1u;
                const int pos = base + __popc(mask & below);
                const int pos1 = base1 + __popc(mask1 & below);
                if (keep) {
                    s.nd[a + pos] = j; s.dl[a + pos] = s.w[j]; s.zz[a + pos] = s.z[j];
                    s.kl[a + (j < k ? pos1 : K1 + pos - pos1)] = pos | (j << 16);
                } else if (t < m) {
                    s.nd[a + K0 + t - pos] = j;
                }
                base += __popc(mask);
                base1 += __popc(mask1);
            }
            __syncwarp();
            bool close = false;
#pragma unroll 1
            for (int p = 1 + lane; p < K0; p += 32) {
                const double T = s.dl[a + p] - s.dl[a + p - 1];
                const double zn = s.zz[a + p], zp = s.zz[a + p - 1];
                close |= fabs(T) * fabs(zn * zp) <= tol * (zn * zn + zp * zp);
            }
            close = __any_sync(0xffffffffu, close);
            if (lane == 0) {
                int K = K0;
                if (close) {
                    // sequential deflation with rotations of nearly equal
                    // poles; deflated slots fill nd from the back
                    K = 0;
                    int pj = -1, back = m;
#pragma unroll 1
                    for (int t = 0; t < m; ++t) {
                        const int nj = s.perm[a + t];
                        if (!(rho * fabs(s.z[nj]) > tol)) { s.org[a + --back] = nj; continue; }
                        if (pj < 0) { pj = nj; continue; }
                        const double T = s.w[nj] - s.w[pj];
                        const double zn = s.z[nj], zp = s.z[pj];
                        const double t2 = zn * zn + zp * zp;
                        if (fabs(T) * fabs(zn * zp) <= tol * t2) {
                            const double ta = sqrt(t2);
                            const double c = zn / ta, sn = -zp / ta;
                            s.z[nj] = ta; s.z[pj] = 0.0;
                            if constexpr (ROWS) {
                                double* x = s.rows + kRowsTracked * pj;
                                double* y = s.rows + kRowsTracked * nj;
#pragma unroll 1
                                for (int r = 0; r < kRowsTracked; ++r) {
                                    const double xr = x[r], yr = y[r];
                                    x[r] = c * xr + sn * yr;
                                    y[r] = c * yr - sn * xr;
                                }
                            } else {
#pragma unroll 1
                                for (int r = a; r < b; ++r) {
                                    const double x = s.Z[r + (size_t)pj * s.ldz], y = s.Z[r + (size_t)nj * s.ldz];
                                    s.Z[r + (size_t)pj * s.ldz] = c * x + sn * y;
                                    s.Z[r + (size_t)nj * s.ldz] = c * y - sn * x;
                                }
                            }
                            const double wp = s.w[pj], wn = s.w[nj];
                            s.w[pj] = wp * c * c + wn * sn * sn;
                            s.w[nj] = wp * sn * sn + wn * c * c;
                            s.org[a + --back] = pj;
                        } else {
                            s.nd[a + K] = pj; s.dl[a + K] = s.w[pj]; s.zz[a + K] = s.z[pj];
                            s.kl[a + K] = K | (pj << 16);
                            ++K;
                        }
                        pj = nj;
                    }
                    if (pj >= 0) {
                        s.nd[a + K] = pj; s.dl[a + K] = s.w[pj]; s.zz[a + K] = s.z[pj];
                        s.kl[a + K] = K | (pj << 16);
                        ++K;
                    }
#pragma unroll 1
                    for (int t = K; t < m; ++t) s.nd[a + t] = s.org[a + t];   // back == K here
                }
                s.kcnt[a] = K;
                s.kcnt[a + 1] = K1;
                s.kcnt[a + 2] = close ? 1 : 0;
                s.rho[a] = rho;
            }
        }
        team_sync<NT, BLOCK>();
        phase_mark(11);
        if (half >= n) break;
        // ---- phase B: secular roots, P lanes per root
        const int qq = tid & (P - 1);
        const unsigned qmask = (P == 4 ? 0xFu : P == 2 ? 0x3u : 0x1u) << (lane & ~(P - 1));
#pragma unroll 1
        for (int p0 = 0; p0 < P * n; p0 += NT) {
            const int pidx = (p0 + tid) / P;
            if (pidx >= n) continue;
            const int a = pidx - pidx % span;
            if (a + half >= n) continue;
            const int i = pidx - a, K = s.kcnt[a];
            if (i >= K) continue;
            double t; int o;
            const int its = secular_root_p<P>(i, K, s.dl + a, s.zz + a, s.rho[a], qq, qmask, t, o);
            if (qq == 0) {
                s.rt[pidx] = t; s.org[pidx] = o;
                phase_count(27, (unsigned long long)its);
                phase_count(29, 1);
                phase_level_max((unsigned)its);
            }
        }
        team_sync<NT, BLOCK>();
        phase_mark(12);
        phase_level_flush(28);
        // ---- phase C: Loewner z-hat, P lanes per root
#pragma unroll 1
        for (int p0 = 0; p0 < P * n; p0 += NT) {
            const int pidx = (p0 + tid) / P;
            if (pidx >= n) continue;
            const int a = pidx - pidx % span;
            if (a + half >= n) continue;
            const int i = pidx - a, K = s.kcnt[a];
            if (i >= K) continue;
            const double* dl = s.dl + a;
            const double dli = dl[i];
            double W = (qq == 0) ? (dli - dl[s.org[a + i]]) - s.rt[a + i] : 1.0;
#pragma unroll 2
            for (int j = qq; j < K; j += P) {
                if (j == i) continue;
                const double del = (dli - dl[s.org[a + j]]) - s.rt[a + j];
                W *= del * fast_rcp(dli - dl[j]);
            }
            W = lanes_prod<P>(W, qmask);
            if (qq == 0) s.zh[pidx] = copysign(sqrt(fmax(-W, 0.0)), s.zz[pidx]);
        }
        team_sync<NT, BLOCK>();
        phase_mark(13);
        // ---- phase D: eigenvector columns of the rank-one problem (P lanes
        // per column), new eigenvalues; ROWS: the tracked rows times them
        if constexpr (ROWS) {
            constexpr int RP = (P * NMAX + NT - 1) / NT;
            static_assert(RP == 1, "one pass over the columns");
            const int pidx = tid / P;
            const int a = pidx - pidx % span;
            double nr[kRowsTracked];
#pragma unroll
            for (int r = 0; r < kRowsTracked; ++r) nr[r] = 0.0;
            const bool on = pidx < n && a + half < n && pidx - a < s.kcnt[a < n ? a : 0];
            if (on) {
                const int j = pidx - a, K = s.kcnt[a];
                const double* dl = s.dl + a;
                const double base = dl[s.org[a + j]], tj = s.rt[a + j];
                double nrm = 0.0;
#pragma unroll 1
                for (int l = qq; l < K; l += P) {
                    const double v = s.zh[a + l] * fast_rcp((dl[l] - base) - tj);
                    nrm = fma(v, v, nrm);
                    const double* rl = s.rows + kRowsTracked * s.nd[a + l];
#pragma unroll
                    for (int r = 0; r < kRowsTracked; ++r) nr[r] = fma(v, rl[r], nr[r]);
                }
                const double inv = rsqrt(lanes_sum<P>(nrm, qmask));
#pragma unroll
                for (int r = 0; r < kRowsTracked; ++r) nr[r] = lanes_sum<P>(nr[r], qmask) * inv;
                if (qq == 0) s.w[s.nd[a + j]] = base + tj;
            }
            team_sync<NT, BLOCK>();
            phase_mark(14);
            if (on && qq == 0) {
                double* rj = s.rows + kRowsTracked * s.nd[pidx];
#pragma unroll
                for (int r = 0; r < kRowsTracked; ++r) rj[r] = nr[r];
            }
        } else {
#pragma unroll 1
            for (int p0 = 0; p0 < P * n; p0 += NT) {
                const int pidx = (p0 + tid) / P;
                if (pidx >= n) continue;
                const int a = pidx - pidx % span;
                if (a + half >= n) continue;
                const int j = pidx - a, K = s.kcnt[a];
                if (j >= K) continue;
                const double* dl = s.dl + a;
                const double base = dl[s.org[a + j]], tj = s.rt[a + j];
                double* ucol = s.U + a + (size_t)(a + j) * s.ldu;
                double nrm = 0.0;
#pragma unroll 2
                for (int l = qq; l < K; l += P) {
                    const double v = s.zh[a + l] * fast_rcp((dl[l] - base) - tj);
                    ucol[l] = v;
                    nrm = fma(v, v, nrm);
                }
                const double inv = rsqrt(lanes_sum<P>(nrm, qmask));
#pragma unroll 1
                for (int l = qq; l < K; l += P) ucol[l] *= inv;
                if (qq == 0) s.w[s.nd[a + j]] = base + tj;
            }
            team_sync<NT, BLOCK>();
            phase_mark(14);
            // ---- phase E: Z(:, nd) <- Z(:, nd) * U.
            if constexpr (NMAX > 0) {
                dc_merge_panels<NT, NMAX, BLOCK>(n, half, span, s);
            } else {
                if (span <= 32) dc_merge_rows_regs<NT, 8, BLOCK>(n, half, span, s);
                else dc_merge_tiled<NT, BLOCK>(n, half, span, s);
            }
        }
        team_sync<NT, BLOCK>();
        phase_mark(15);
    }
    // ---- back to the caller's units
    const double inv = 1.0 / sc;
#pragma unroll 1
    for (int i = tid; i < n; i += NT) s.w[i] *= inv;
    team_sync<NT, BLOCK>();
}

}  // namespace sgeig
