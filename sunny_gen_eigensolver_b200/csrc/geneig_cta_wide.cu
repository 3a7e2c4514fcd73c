// Shared-memory kernel, 64 < N <= 112 (see geneig_cta_kernel.cuh).
#include "geneig_cta_kernel.cuh"

namespace sgeig {

CtaKernelFn cta_kernel_wide(int nmax) {
    switch (nmax) {
        case 72: return geneig_cta_kernel<72, 1, false, false>;
        case 80: return geneig_cta_kernel<80, 1, false, false>;
        case 96: return geneig_cta_kernel<96, 1, false, false>;
        default: return geneig_cta_kernel<112, 1, false, false>;
    }
}

}  // namespace sgeig
