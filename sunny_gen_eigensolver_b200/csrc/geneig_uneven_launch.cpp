// Host side of an uneven-size launch (see geneig_uneven.cu): which kernels run,
// on which streams, and how they are joined.
#include "geneig_kernels.h"

namespace sgeig {

cudaError_t uneven_launch(const UnevenLaunch& L, unsigned long long* head, void* scratch, size_t slot_elems,
                          int grid, size_t smem, cudaStream_t stream, const UnevenSide& side) {
    int nside = 0, nsmall = 0;
    for (int i = 0; i < L.ngroups; ++i)
        if (L.count[i] > 0) ++(L.kind[i] >= kUnevenResident ? nside : nsmall);
    // The side sizes first, largest first (the groups' order): their pencils
    // take longest, and the persistent kernel's small ones fill the SMs that
    // they leave.
    const bool fork = nside + (nsmall > 0 ? 1 : 0) > 1;
    cudaError_t e = fork ? cudaEventRecord(side.fork, stream) : cudaSuccess;
    int open = 0;                                    // side streams that have taken the fork
    for (int i = 0; i < L.ngroups && e == cudaSuccess; ++i) {
        if (L.count[i] <= 0 || L.kind[i] < kUnevenResident) continue;
        const cudaStream_t st = fork ? side.stream[open] : stream;
        if (fork) {
            e = cudaStreamWaitEvent(st, side.fork, 0);
            if (e != cudaSuccess) break;
            ++open;
        }
        if (L.kind[i] == kUnevenResident)
            e = cta_launch(L.n[i], cta_nmax_for(L.n[i]), 4, L.H[i], L.S[i], L.W[i], L.U[i], L.info[i], L.count[i], st);
        else
            e = tiled_launch(L.n[i], L.slots[i], 4, L.H[i], L.S[i], L.W[i], L.U[i], L.info[i],
                             L.count[i], L.scratch[i], st, false);
    }
    if (e == cudaSuccess && nsmall > 0) e = uneven_persistent_launch(L, head, scratch, slot_elems, grid, smem, stream);
    // Whatever failed, `stream` waits for what the side streams were given:
    // the caller's buffers and the slots are theirs until then.
    for (int s = 0; s < open; ++s) {
        cudaError_t j = cudaEventRecord(side.join[s], side.stream[s]);
        if (j == cudaSuccess) j = cudaStreamWaitEvent(stream, side.join[s], 0);
        if (j != cudaSuccess) cudaStreamSynchronize(side.stream[s]);
        if (e == cudaSuccess) e = j;
    }
    return e;
}

}  // namespace sgeig
