// Shared-memory kernel, forms with S assembled from Fourier terms (one pencil
// per CTA) or reduced to intensities, N <= 64 (see geneig_cta_kernel.cuh).
#include "geneig_cta_kernel.cuh"

namespace sgeig {

template <int NMAX>
static CtaKernelFn pick(int teams, bool fs, bool spec) {
    if (fs) return spec ? geneig_cta_kernel<NMAX, 1, true, true> : geneig_cta_kernel<NMAX, 1, true, false>;
    if constexpr (NMAX <= 16) {
        if (teams == 4) return geneig_cta_kernel<NMAX, 4, false, true>;
    }
    if constexpr (NMAX <= 32) {
        if (teams == 2) return geneig_cta_kernel<NMAX, 2, false, true>;
    }
    return geneig_cta_kernel<NMAX, 1, false, true>;
}

CtaKernelFn cta_kernel_spec(int nmax, int teams, bool fs, bool spec) {
    switch (nmax) {
        case 16: return pick<16>(teams, fs, spec);
        case 24: return pick<24>(teams, fs, spec);
        case 32: return pick<32>(teams, fs, spec);
        case 40: return pick<40>(teams, fs, spec);
        case 48: return pick<48>(teams, fs, spec);
        case 56: return pick<56>(teams, fs, spec);
        default: return pick<64>(teams, fs, spec);
    }
}

}  // namespace sgeig
