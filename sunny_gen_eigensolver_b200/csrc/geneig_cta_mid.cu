// Shared-memory kernel, 32 < N <= 64 (see geneig_cta_kernel.cuh).
#include "geneig_cta_kernel.cuh"

namespace sgeig {

CtaKernelFn cta_kernel_mid(int nmax) {
    switch (nmax) {
        case 40: return geneig_cta_kernel<40, 1, false, false>;
        case 48: return geneig_cta_kernel<48, 1, false, false>;
        case 56: return geneig_cta_kernel<56, 1, false, false>;
        default: return geneig_cta_kernel<64, 1, false, false>;
    }
}

}  // namespace sgeig
