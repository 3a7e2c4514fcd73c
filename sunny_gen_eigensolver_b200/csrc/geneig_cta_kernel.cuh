// The shared-memory kernel (geneig_cta.cu describes it) and its launch shapes,
// instantiated in four translation units that compile side by side:
// geneig_cta_small.cu (N <= 32), _mid.cu (N <= 64), _wide.cu (N <= 112) and
// _spec.cu (the Fourier and intensity forms).
#pragma once

#include "geneig_cta_body.cuh"

namespace sgeig {
using namespace cta;

using CtaKernelFn = void (*)(CtaArgs, CtaFourier);
// The instance for a row bound (and pencils per CTA, form); each unit knows its own.
CtaKernelFn cta_kernel_small(int nmax, int teams);
CtaKernelFn cta_kernel_mid(int nmax);
CtaKernelFn cta_kernel_wide(int nmax);
CtaKernelFn cta_kernel_spec(int nmax, int teams, bool fs, bool spec);

namespace {

// Pencils per SM that the register allocation is sized for, by row bound.
template <int NMAX> struct CtaShape {
    static constexpr int nt = cta_team_threads(NMAX);
    static constexpr int per_sm = NMAX <= 16 ? 16 : NMAX <= 32 ? 8 : NMAX <= 56 ? 4 : NMAX <= 64 ? 3 : NMAX <= 80 ? 2 : 1;
};

// TEAMS pencils per CTA at a time (the reference's batches per block): the
// CTA has TEAMS teams of CtaShape<NMAX>::nt threads, each with its own
// barrier and shared-memory slice, team t taking pencils TEAMS * cta + t,
// then a grid's stride on. FS: S from Fourier terms. SPEC: intensities.
template <int NMAX, int TEAMS, bool FS, bool SPEC>
__global__ void __launch_bounds__(CtaShape<NMAX>::nt * TEAMS, (CtaShape<NMAX>::per_sm + TEAMS - 1) / TEAMS)
geneig_cta_kernel(CtaArgs a, CtaFourier f) {
    constexpr int NT = CtaShape<NMAX>::nt;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    phase_start();
    const int t = TEAMS == 1 ? 0 : (int)(threadIdx.x / NT);
    unsigned char* sm = smem_raw + (TEAMS == 1 ? 0 : (size_t)t * cta_bytes(a.n, NT / 32, SPEC));
    for (long long b = (long long)blockIdx.x * TEAMS + t; b < a.batch; b += (long long)gridDim.x * TEAMS) {
        if (a.retry && a.info[b] != kRetryInfo) continue;
        cta_solve<NMAX, NT, NT * TEAMS, FS, SPEC>(a, b, sm, &f);
    }
}

}  // namespace
}  // namespace sgeig
