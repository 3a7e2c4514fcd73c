// Host side of an uneven-size launch (see geneig_uneven.cu): which kernels run
// beside one another and how they are joined.
#include "geneig_kernels.h"

#include <vector>

namespace sgeig {
namespace {

// Branches of work from one point of `stream` that come together again there. A
// branch starts when all CTAs of the one before it have begun: what takes longest
// gets its SMs first, also when several calls are queued and every branch is ready
// at the fork. 12 to 216 rows, 4000 pencils, ms a call back to back: 9.42, 10.60
// without, 9.51 with stream priorities, which put the call before all other work
// of the device; 24, 60, 130 and 162 rows, 800 pencils: 4.23, 6.44, 6.44.
class Fork {
public:
    Fork(cudaStream_t stream, const UnevenSide& side, bool capturing) : stream_(stream), side_(side), capturing_(capturing) {}

    cudaError_t begin() {
        forked_ = true;
        return capturing_ ? add_dependencies(root_) : cudaEventRecord(side_.fork, stream_);
    }
    // The stream of the next branch, one kernel, and the event that it records
    // when its last CTA has begun (NULL: none).
    cudaError_t next(cudaStream_t* st, cudaEvent_t* started) {
        *st = stream_;
        *started = nullptr;
        if (!forked_) return cudaSuccess;
        if (capturing_) return next_captured();
        const cudaError_t e = cudaStreamWaitEvent(side_.stream[open_], turn(), 0);
        if (e != cudaSuccess) return e;
        *st = side_.stream[open_++];
        *started = turn();
        return cudaSuccess;
    }
    // The last branch, on the caller's own stream.
    cudaError_t last() {
        if (!forked_) return cudaSuccess;
        return capturing_ ? next_captured() : cudaStreamWaitEvent(stream_, turn(), 0);
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
        if (!ends_.node.empty()) {
            const cudaError_t j = set_dependencies(ends_, cudaStreamAddCaptureDependencies);
            if (first == cudaSuccess) first = j;
        }
        return first;
    }

private:
    struct Dependencies {
        std::vector<cudaGraphNode_t> node;
        std::vector<cudaGraphEdgeData> edge;
        void add(cudaGraphNode_t n, cudaGraphEdgeData d) {
            node.push_back(n);
            edge.push_back(d);
        }
    };

    // A branch's event, recorded by its kernel as the next branch's turn and
    // again at the end to join.
    cudaEvent_t turn() const { return open_ ? side_.join[open_ - 1] : side_.fork; }

    // A capture's branches are made of its graph's dependencies on the caller's
    // stream alone: a side stream would belong to the capture until its end and
    // refuse the handle's other launches till then.
    cudaError_t next_captured() {
        if (!branches_++) return cudaSuccess;
        Dependencies from = root_, before;
        const cudaError_t e = add_dependencies(before);
        if (e != cudaSuccess) return e;
        for (size_t i = 0; i < before.node.size(); ++i) {
            ends_.add(before.node[i], before.edge[i]);
            cudaGraphEdgeData begun{};
            begun.from_port = cudaGraphKernelNodePortLaunchCompletion;
            from.add(before.node[i], begun);
        }
        return set_dependencies(from, cudaStreamSetCaptureDependencies);
    }
    cudaError_t add_dependencies(Dependencies& out) const {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        const cudaGraphNode_t* nodes = nullptr;
        const cudaGraphEdgeData* edges = nullptr;
        size_t count = 0;
        const cudaError_t e = cudaStreamGetCaptureInfo_v3(stream_, &cs, nullptr, nullptr, &nodes, &edges, &count);
        if (e != cudaSuccess) return e;
        if (cs != cudaStreamCaptureStatusActive) return cudaErrorStreamCaptureInvalidated;
        for (size_t i = 0; i < count; ++i) out.add(nodes[i], edges ? edges[i] : cudaGraphEdgeData{});
        return cudaSuccess;
    }
    cudaError_t set_dependencies(Dependencies& d, unsigned flags) const {
        return cudaStreamUpdateCaptureDependencies_v2(stream_, d.node.data(), d.edge.data(), d.node.size(), flags);
    }

    cudaStream_t stream_;
    const UnevenSide& side_;
    bool capturing_, forked_ = false;
    int open_ = 0;                            // side streams that have taken the fork
    int branches_ = 0;                        // captured so far
    Dependencies root_, ends_;                // where the branches start; the last nodes of all but the current one
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
    cudaEvent_t started = nullptr;
    const bool several = nside + (nsmall > 0 ? 1 : 0) > 1;
    cudaError_t e = several && side.fork ? fork.begin() : cudaSuccess;
    for (int i = 0; i < L.ngroups && e == cudaSuccess; ++i) {
        if (L.count[i] <= 0 || L.kind[i] < kUnevenResident) continue;
        e = fork.next(&st, &started);
        if (e != cudaSuccess) break;
        if (L.kind[i] == kUnevenResident)
            e = cta_launch(L.n[i], cta_nmax_for(L.n[i]), 4, L.H[i], L.S[i], L.W[i], L.U[i], L.info[i], L.count[i], st,
                           false, 1, false, started);
        else
            e = tiled_launch(L.n[i], L.slots[i], 4, L.H[i], L.S[i], L.W[i], L.U[i], L.info[i],
                             L.count[i], L.scratch[i], st, false, false, kRefineMaxIters, false, started);
    }
    if (e == cudaSuccess && nsmall > 0) e = fork.last();
    if (e == cudaSuccess && nsmall > 0) e = uneven_persistent_launch(L, head, scratch, slot_elems, grid, smem, stream);
    return fork.join(e);
}

}  // namespace sgeig
