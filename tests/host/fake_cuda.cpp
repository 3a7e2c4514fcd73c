// Stands in for the CUDA runtime and the kernel launchers under the C ABI
// (c_api.cpp), so that what it creates, records, waits for and launches can be
// checked without a GPU. Every call is a line of the log; a call can be told to
// fail. Handles are small numbers.
#include "geneig_kernels.h"

#include <cuda_runtime.h>

#include <map>
#include <set>
#include <string>
#include <vector>

using namespace sgeig;

static std::string g_log, g_fail;      // "name:k": the k-th call (from 0) of `name` fails
static std::map<std::string, int> g_calls;
// Captures: the origin of each capturing stream; the origin of each event recorded in one; and each
// capturing stream's current dependencies (nodes are numbers).
static std::map<size_t, size_t> g_capturing, g_event;
static std::map<size_t, std::vector<cudaGraphNode_t>> g_deps;
static std::map<size_t, std::vector<cudaGraphEdgeData>> g_edges;
static size_t g_next = 100, g_memory = (size_t)1 << 40, g_used = 0;
static std::map<size_t, size_t> g_blocks;

static bool say(const std::string& name, const std::string& rest = "") {
    const int k = g_calls[name]++;
    const bool fails = g_fail == name + ":" + std::to_string(k);
    g_log += name + (rest.empty() ? "" : " " + rest) + (fails ? " FAILS" : "") + "\n";
    return fails;
}
static std::string num(const void* p) { return std::to_string((size_t)p); }
template <class T> static T fresh() { return reinterpret_cast<T>(++g_next); }
// A kernel on stream s: in a capture a node after the stream's dependencies.
static cudaError_t kernel(const std::string& name, const std::string& what, cudaStream_t s, const std::string& rest = "") {
    std::string line = what + "on " + std::to_string((size_t)s) + rest;
    if (g_capturing.count((size_t)s)) {
        auto& d = g_deps[(size_t)s];
        const auto node = fresh<cudaGraphNode_t>();
        line += " node " + num(node) + " after";
        for (size_t i = 0; i < d.size(); ++i)
            line += " " + num(d[i]) + (g_edges[(size_t)s][i].from_port ? "-begun" : "");
        d = {node};
        g_edges[(size_t)s] = {cudaGraphEdgeData{}};
    }
    return say(name, line) ? cudaErrorLaunchFailure : cudaSuccess;
}
static cudaError_t result(bool fails) { return fails ? cudaErrorLaunchFailure : cudaSuccess; }

extern "C" {
void fake_reset(const char* fail, size_t memory) {
    g_log.clear();
    g_calls.clear();
    g_fail = fail;
    g_memory = memory;
}
void fake_capture(size_t stream, int on) {
    if (on) { g_capturing[stream] = stream; g_deps[stream] = {fresh<cudaGraphNode_t>()}; g_edges[stream] = {cudaGraphEdgeData{}}; return; }
    std::map<size_t, size_t> left;
    for (auto& c : g_capturing) if (c.second != stream) left.insert(c);
    g_capturing = left;
}
const char* fake_dependencies(size_t stream) {
    static std::string out;
    out.clear();
    for (auto n : g_deps[stream]) out += num(n) + " ";
    return out.c_str();
}
const char* fake_log() { return g_log.c_str(); }
size_t fake_memory_used() { return g_used; }

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 232448;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t bytes) {
    if (g_used + bytes > g_memory) { say("malloc", "refused"); return cudaErrorMemoryAllocation; }
    *p = fresh<void*>();
    g_used += g_blocks[(size_t)*p] = bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p) { g_used -= g_blocks[(size_t)p]; g_blocks.erase((size_t)p); }
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = fresh<cudaEvent_t>(); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return result(say("sync_event", num(e))); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return result(say("sync_stream", num(s))); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (say("record", num(e) + " on " + num(s))) return cudaErrorLaunchFailure;
    g_event.erase((size_t)e);
    if (g_capturing.count((size_t)s)) g_event[(size_t)e] = g_capturing[(size_t)s];
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    if (say("wait", num(e) + " on " + num(s))) return cudaErrorLaunchFailure;
    const bool in = g_event.count((size_t)e);
    if (!in && g_capturing.count((size_t)s)) return cudaErrorStreamCaptureIsolation;
    if (in && g_capturing.count((size_t)s) && g_capturing[(size_t)s] != g_event[(size_t)e]) return cudaErrorStreamCaptureMerge;
    if (in) g_capturing[(size_t)s] = g_event[(size_t)e];
    return cudaSuccess;
}
cudaError_t cudaStreamGetCaptureInfo_v3(cudaStream_t s, cudaStreamCaptureStatus* cs, unsigned long long*, cudaGraph_t*,
                                        const cudaGraphNode_t** nodes, const cudaGraphEdgeData** edges, size_t* count) {
    const bool in = g_capturing.count((size_t)s);
    *cs = in ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    if (in) { *nodes = g_deps[(size_t)s].data(); *edges = g_edges[(size_t)s].data(); *count = g_deps[(size_t)s].size(); }
    return result(say("capture_info"));
}
cudaError_t cudaStreamUpdateCaptureDependencies_v2(cudaStream_t s, cudaGraphNode_t* nodes, const cudaGraphEdgeData* edges,
                                                   size_t count, unsigned flags) {
    if (say("set_dependencies")) return cudaErrorLaunchFailure;
    if (!g_capturing.count((size_t)s)) return cudaErrorIllegalState;
    auto& d = g_deps[(size_t)s];
    auto& x = g_edges[(size_t)s];
    if (flags == cudaStreamSetCaptureDependencies) { d.clear(); x.clear(); }
    d.insert(d.end(), nodes, nodes + count);
    x.insert(x.end(), edges, edges + count);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* cs) {
    *cs = g_capturing.count((size_t)s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int priority) {
    *s = fresh<cudaStream_t>();
    return result(say("stream", num(*s) + " priority " + std::to_string(priority)));
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned flags) { return cudaStreamCreateWithPriority(s, flags, 0); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
}

namespace sgeig {

static void started(cudaEvent_t e, cudaStream_t s) { if (e) g_log += "starts " + num(e) + " with " + num(s) + "\n"; }
bool plain_plan(int n, int, PlainPlan* p, std::string*, bool mixed, const char* regime, int slots, int) {
    p->n = n;
    p->mixed = mixed;
    const bool l2 = regime && std::string(regime) == "l2-slot";
    p->regime = mixed || l2 || n > kCtaPreferredMaxN ? Regime::L2Slot : Regime::SmemCta;
    p->resident = !mixed && p->regime == Regime::L2Slot && slots == 0 && n > kCtaPreferredMaxN && n <= kResidentMaxN;
    p->scratch_bytes = p->regime == Regime::L2Slot && !p->resident ? 4096 : 0;
    return true;
}
cudaError_t plain_launch(const PlainPlan& p, int, const void*, const void*, double*, void*, int*, long long, void*,
                         cudaStream_t s, bool) {
    return result(say("launch", std::to_string(p.n) + " on " + num(s)));
}
cudaError_t cta_launch_intensity(int, int, const void*, const void*, const double*, const double*, int, double, double*,
                                 double*, int*, long long, cudaStream_t, int) { return cudaSuccess; }
cudaError_t cta_launch_fourier(int, int, const FourierTerms&, const double*, const void*, const double*, const double*,
                               int, double, double*, void*, double*, int*, long long, cudaStream_t) { return cudaSuccess; }
std::string tune_key(int, int, int) { return ""; }
bool tune_lookup(const std::string&, int, std::string*) { return false; }
void tune_store(const std::string&, int, const std::string&) {}
int tune_pick(int, int, const std::vector<std::pair<std::string, int>>&, std::string*) { return 0; }
int cta_nmax_for(int) { return 0; }
cudaError_t cta_set_attributes(int, size_t, bool) { return cudaSuccess; }
cudaError_t tiled_set_attributes(int, bool, size_t) { return cudaSuccess; }
cudaError_t uneven_set_attributes(size_t) { return cudaSuccess; }
int tiled_slots_for(int n) { return n > 200 ? 1 : 2; }
int uneven_kind(int n, bool l2) { return !l2 ? 0 : n <= kCtaPreferredMaxN ? 5 : n <= kResidentMaxN ? kUnevenResident : kUnevenBig; }
size_t uneven_smem_bytes(int, int) { return 1024; }
cudaError_t cta_launch(int n, int, int, const void*, const void*, double*, void*, int*, long long, cudaStream_t s, bool,
                       int, bool, cudaEvent_t e) { started(e, s); return kernel("cta", std::to_string(n) + " ", s); }
cudaError_t tiled_launch(int n, int, int, const void*, const void*, double*, void*, int*, long long, void* scratch,
                         cudaStream_t s, bool, bool, int, bool, cudaEvent_t e) {
    started(e, s);
    return kernel("tiled", std::to_string(n) + " ", s, " slots " + num(scratch));
}
cudaError_t uneven_persistent_launch(const UnevenLaunch&, unsigned long long*, void*, size_t, int, size_t, cudaStream_t s) {
    return kernel("persistent", "", s);
}

}  // namespace sgeig
