// Host side of an uneven-size launch (see geneig_uneven.cu): which kernels run
// beside one another and how they are joined.
#include "geneig_kernels.h"

#include <vector>

namespace sgeig {
namespace {

// Branches of work from one point of `stream` that come together again there.
class Fork {
public:
    Fork(cudaStream_t stream, const UnevenSide& side, bool capturing) : stream_(stream), side_(side), capturing_(capturing) {}

    cudaError_t begin() {
        forked_ = true;
        return capturing_ ? dependencies(root_) : cudaEventRecord(side_.fork, stream_);
    }
    // The stream of the next branch.
    cudaError_t next(cudaStream_t* st) {
        *st = stream_;
        if (!forked_) return cudaSuccess;
        if (capturing_) return back_to_root();
        const cudaError_t e = cudaStreamWaitEvent(side_.stream[open_], side_.fork, 0);
        if (e == cudaSuccess) *st = side_.stream[open_++];
        return e;
    }
    // The stream of the last branch: the caller's own.
    cudaError_t last(cudaStream_t* st) {
        *st = stream_;
        return forked_ && capturing_ ? back_to_root() : cudaSuccess;
    }
    // Whatever failed, `stream` waits for what the branches were given: the
    // caller's buffers and the slots are theirs until then. First error.
    cudaError_t join(cudaError_t first) {
        for (int s = 0; s < open_; ++s) {
            cudaError_t j = cudaEventRecord(side_.join[s], side_.stream[s]);
            if (j == cudaSuccess) j = cudaStreamWaitEvent(stream_, side_.join[s], 0);
            if (j != cudaSuccess) cudaStreamSynchronize(side_.stream[s]);
            if (first == cudaSuccess) first = j;
        }
        if (forked_ && capturing_ && !ends_.empty()) {
            const cudaError_t j = set_dependencies(ends_, cudaStreamAddCaptureDependencies);
            if (first == cudaSuccess) first = j;
        }
        return first;
    }

private:
    // A capture's branches are made of its graph's dependencies on the caller's
    // stream alone: a side stream would belong to the capture until its end and
    // refuse the handle's other launches till then.
    cudaError_t dependencies(std::vector<cudaGraphNode_t>& out) const {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        const cudaGraphNode_t* nodes = nullptr;
        size_t count = 0;
        const cudaError_t e = cudaStreamGetCaptureInfo_v2(stream_, &cs, nullptr, nullptr, &nodes, &count);
        if (e != cudaSuccess) return e;
        if (cs != cudaStreamCaptureStatusActive) return cudaErrorStreamCaptureInvalidated;
        out.insert(out.end(), nodes, nodes + count);
        return cudaSuccess;
    }
    cudaError_t set_dependencies(std::vector<cudaGraphNode_t>& nodes, unsigned flags) const {
        return cudaStreamUpdateCaptureDependencies(stream_, nodes.data(), nodes.size(), flags);
    }
    cudaError_t back_to_root() {
        if (!branches_++) return cudaSuccess;
        const cudaError_t e = dependencies(ends_);
        return e == cudaSuccess ? set_dependencies(root_, cudaStreamSetCaptureDependencies) : e;
    }

    cudaStream_t stream_;
    const UnevenSide& side_;
    bool capturing_, forked_ = false;
    int open_ = 0;                            // side streams that have taken the fork
    int branches_ = 0;                        // captured so far
    std::vector<cudaGraphNode_t> root_, ends_;   // where the branches start; the last nodes of all but the current one
};

}  // namespace

cudaError_t uneven_launch(const UnevenLaunch& L, unsigned long long* head, void* scratch, size_t slot_elems,
                          int grid, size_t smem, cudaStream_t stream, const UnevenSide& side, bool capturing) {
    int nside = 0, nsmall = 0;
    for (int i = 0; i < L.ngroups; ++i)
        if (L.count[i] > 0) ++(L.kind[i] >= kUnevenResident ? nside : nsmall);
    // The side sizes first, largest first (the groups' order): their pencils
    // take longest, and the persistent kernel's small ones fill the SMs that
    // they leave.
    Fork fork(stream, side, capturing);
    cudaStream_t st = stream;
    cudaError_t e = nside + (nsmall > 0 ? 1 : 0) > 1 ? fork.begin() : cudaSuccess;
    for (int i = 0; i < L.ngroups && e == cudaSuccess; ++i) {
        if (L.count[i] <= 0 || L.kind[i] < kUnevenResident) continue;
        e = fork.next(&st);
        if (e != cudaSuccess) break;
        if (L.kind[i] == kUnevenResident)
            e = cta_launch(L.n[i], cta_nmax_for(L.n[i]), 4, L.H[i], L.S[i], L.W[i], L.U[i], L.info[i], L.count[i], st);
        else
            e = tiled_launch(L.n[i], L.slots[i], 4, L.H[i], L.S[i], L.W[i], L.U[i], L.info[i],
                             L.count[i], L.scratch[i], st, false);
    }
    if (e == cudaSuccess && nsmall > 0) e = fork.last(&st);
    if (e == cudaSuccess && nsmall > 0) e = uneven_persistent_launch(L, head, scratch, slot_elems, grid, smem, st);
    return fork.join(e);
}

}  // namespace sgeig
