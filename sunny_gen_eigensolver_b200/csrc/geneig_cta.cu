// Batched generalized Hermitian-definite eigensolver, shared-memory regime
// (N <= 64) and the l2-slot class up to N = 110: a team of NT threads (32 to
// 512 by N) holds one matrix per pencil in shared memory and solves it end to end; a CTA is one team or, with
// several pencils per CTA, up to four, each with its own barrier and
// shared-memory slice; CTAs loop over the batch. Further kernel forms
// assemble S(q) from Fourier terms in the load stage (the metric solve of a
// spin-wave dynamical matrix that never exists in memory) and reduce the
// metric solve to intensities.
//
// Stage chain (reference: src/unified/kernel_source.hpp:233-276):
//   a1  load the lower triangle of S                          (:233-242)
//   a2  Cholesky S = L L^H fused with X = L^-1, in place, 8-column panels on
//       the FP64 tensor cores (mma.m8n8k4.f64), two barriers per panel (:244)
//   a3+a4  C = L^-1 H L^-H, 8 (N > 80: 16) columns at a time: T = H X^H (H from global
//       memory, in full, as the reference's two triangular solves read it),
//       then C = X T; C fills the upper triangle beside X       (:246-248)
//   a5  Householder tridiagonalisation (lower; the rank-2 update and the next
//       matrix-vector product share one pass, two barriers per step), divide
//       and conquer on the tridiagonal, back-transform V = Q Z in compact-WY
//       blocks of 8 reflectors on the FP64 tensor cores, 8-column panels of
//       V per warp                                                  (:250)
//   a6  U = L^-H V = X^H V, on the same panels                     (:252)
//   a7  W (ascending) and U, columns permuted by eigenvalue rank (:268-276)
// X and the reflectors wait for a5/a6 in the pencil's own block of the output
// U, so that one n x n matrix and ~10 KB of vectors per pencil are all the
// shared memory it takes.

#include "geneig_cta_kernel.cuh"

namespace sgeig {

size_t cta_smem_bytes(int n, bool spec) { return cta_bytes(n, cta_team_threads(cta_nmax_for(n)) / 32, spec); }

// Compile-time row bounds: the register arrays and unrolled loops are sized by
// NMAX, so a bound close above n wastes less (56 covers the N=54 workload).
int cta_nmax_for(int n) {
    return n <= 16 ? 16 : n <= 24 ? 24 : n <= 32 ? 32 : n <= 40 ? 40 : n <= 48 ? 48 : n <= 56 ? 56 : n <= 64 ? 64
         : n <= 72 ? 72 : n <= 80 ? 80 : n <= 96 ? 96 : 112;
}

static CtaKernelFn cta_kernel(int nmax, int teams, bool fs, bool spec) {
    if (fs || spec) return cta_kernel_spec(nmax, fs ? 1 : teams, fs, spec);
    return nmax <= 32 ? cta_kernel_small(nmax, teams) : nmax <= kCtaMaxN ? cta_kernel_mid(nmax) : cta_kernel_wide(nmax);
}

int cta_max_teams(int nmax) { return nmax <= 16 ? 4 : nmax <= 32 ? 2 : 1; }

// Default pencils per CTA, measured on B200 (solves/s at batch 65,536, one
// pencil per CTA -> default): N=8 45.6 M -> 47.2 M, N=12 24.7 M -> 25.4 M, N=16
// 20.9 M -> 21.7 M (4 teams of 32 threads); N=32 5.30 M -> 6.09 M (2 of 64);
// N=24 has two on request (7.17 M, 8.51 M with two) and starts with one, so that
// the reported pencils per CTA stay what they were.
int cta_default_teams(int nmax) { return nmax <= 16 ? 4 : nmax == 32 ? 2 : 1; }

size_t cta_teams_smem_bytes(int n, int teams, bool spec) { return teams * cta_smem_bytes(n, spec); }

int cta_threads_for(int nmax) { return cta_team_threads(nmax); }

// `smem` is the per-CTA shared-memory limit; the kernel's own static shared
// memory (profiling builds have some) comes off the dynamic allowance.
cudaError_t cta_set_attributes(int nmax, size_t smem, bool extra) {
    for (int form = 0; form < (extra ? 4 : 1); ++form)
        for (int teams = 1; teams <= cta_max_teams(nmax); teams *= 2) {
            const CtaKernelFn k = cta_kernel(nmax, teams, (form & 1) != 0, (form & 2) != 0);
            cudaFuncAttributes fa{};
            cudaError_t e = cudaFuncGetAttributes(&fa, k);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(smem - fa.sharedSizeBytes));
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

static cudaError_t cta_start(const CtaArgs& a, const CtaFourier& f, int nmax, int teams, bool fs, bool spec,
                             cudaStream_t stream, cudaEvent_t started = nullptr) {
    const long long ctas = (a.batch + teams - 1) / teams;
    const long long grid = ctas < 0x7fffffffLL ? ctas : 0x7fffffffLL;
    return launch_with_event(cta_kernel(nmax, teams, fs, spec), (unsigned)grid, teams * cta_threads_for(nmax),
                             cta_teams_smem_bytes(a.n, teams, spec), stream, started, a, f);
}

cudaError_t cta_launch(int n, int nmax, int stage, const void* H, const void* S, double* W, void* U,
                       int* info, long long batch, cudaStream_t stream, bool sigma, int teams, bool retry,
                       cudaEvent_t started) {
    CtaArgs a{};
    a.H = static_cast<const double2*>(H);
    a.S = static_cast<const double2*>(S);
    a.W = W;
    a.U = static_cast<double2*>(U);
    a.info = info;
    a.batch = batch;
    a.n = n;
    a.ld = cta_ld(n, false);
    a.stage = stage;
    a.sigma = sigma ? 1 : 0;
    a.retry = retry ? 1 : 0;
    return cta_start(a, CtaFourier{}, nmax, teams, false, false, stream, started);
}

// Arguments of the intensity form (no U).
static void spec_args(CtaArgs& a, int n, const void* O, const double* qhat, const double* energies, int ne,
                      double fwhm, double* spec) {
    a.ld = cta_ld(n, true);
    a.O = static_cast<const double2*>(O);
    a.qhat = qhat;
    a.energies = energies;
    a.spec = spec;
    a.ne = ne;
    const double sigma_e = fwhm / (2.0 * std::sqrt(2.0 * std::log(2.0)));
    a.gnorm = 1.0 / (sigma_e * std::sqrt(2.0 * M_PI));
    a.ginv2 = 1.0 / (2.0 * sigma_e * sigma_e);
}

cudaError_t cta_launch_intensity(int n, int nmax, const void* S, const void* O, const double* qhat,
                                 const double* energies, int ne, double fwhm, double* W, double* spec, int* info,
                                 long long batch, cudaStream_t stream, int teams) {
    CtaArgs a{};
    a.S = static_cast<const double2*>(S);
    a.W = W;
    a.info = info;
    a.batch = batch;
    a.n = n;
    a.stage = 4;
    a.sigma = 1;
    spec_args(a, n, O, qhat, energies, ne, fwhm, spec);
    return cta_start(a, CtaFourier{}, nmax, teams, false, true, stream);
}

cudaError_t cta_launch_fourier(int n, int nmax, const FourierTerms& ft, const double* q,
                               const void* O, const double* qhat, const double* energies, int ne, double fwhm,
                               double* W, void* U, double* spec, int* info, long long batch, cudaStream_t stream) {
    CtaArgs a{};
    a.W = W;
    a.U = static_cast<double2*>(U);
    a.info = info;
    a.batch = batch;
    a.n = n;
    a.ld = cta_ld(n, false);
    a.stage = 4;
    a.sigma = 1;
    CtaFourier f{};
    f.start = ft.start;
    f.coef = static_cast<const double2*>(ft.coef);
    f.disp = ft.disp;
    f.q = q;
    f.nterms = ft.nterms;
    if (O) spec_args(a, n, O, qhat, energies, ne, fwhm, spec);
    return cta_start(a, f, nmax, 1, true, O != nullptr, stream);
}

}  // namespace sgeig

#ifdef SGEIG_PHASE_TIMERS
// Profiling builds only: the per-phase cycle counters of the kernels (see
// phase_mark in geneig_common.cuh) into `out`; a nonzero `reset` clears them.
// Not part of the product library's ABI.
#pragma GCC visibility push(default)
extern "C" int sunny_geneig_phase_cycles(unsigned long long* out, int count, int reset) {
    using namespace sgeig;
    if (count > kPhaseSlots) count = kPhaseSlots;
    cudaError_t e = cudaDeviceSynchronize();
    unsigned long long sum[kPhaseSlots] = {};
    for (PhaseReader f : phase_readers())
        if (e == cudaSuccess) e = f(sum, kPhaseSlots, reset != 0);
    for (int i = 0; out && i < count; ++i) out[i] = sum[i];
    return e == cudaSuccess ? 0 : -1;
}
#pragma GCC visibility pop
#endif
