// Shared-memory kernel, N <= 32 (see geneig_cta_kernel.cuh).
#include "geneig_cta_kernel.cuh"

namespace sgeig {

CtaKernelFn cta_kernel_small(int nmax, int teams) {
    switch (nmax) {
        case 16: return teams == 4 ? geneig_cta_kernel<16, 4, false, false>
                      : teams == 2 ? geneig_cta_kernel<16, 2, false, false> : geneig_cta_kernel<16, 1, false, false>;
        case 24: return teams == 2 ? geneig_cta_kernel<24, 2, false, false> : geneig_cta_kernel<24, 1, false, false>;
        default: return teams == 2 ? geneig_cta_kernel<32, 2, false, false> : geneig_cta_kernel<32, 1, false, false>;
    }
}

}  // namespace sgeig
