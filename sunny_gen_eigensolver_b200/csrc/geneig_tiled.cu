// Tiled FP64 batched generalized Hermitian-definite eigensolver for sm_100a,
// for matrices too large to keep in one CTA's shared memory (the "l2-slot"
// regime). One CTA solves one pencil at a time, persistent over the batch;
// its working matrices live in a per-CTA global-memory slot
//     M0, M1, M2: n x ld complex,  Zo: n x ld real (at least 16 n complex)
// and every O(n^3) step except the Householder matrix-vector products is a complex GEMM
// on the FP64 tensor cores (mma.sync.m8n8k4.f64; a complex 8x8x4 step is four
// real MMAs), one 16 x 16 output tile per warp at a time:
//
//   a1  M0 <- S (lower triangle)                      (kernel_source.hpp:233-242)
//   a2  blocked Cholesky S = L L^H in M0: 16-column panels factored column
//       by column, trailing lower tiles updated as C -= L_p L_p^H   (:244)
//   a3  X = L^-1 in M1, one 16-row block at a time: R = L_rk X_kc (GEMM),
//       X_r = L_rr^-1 (e_r - R) (one thread per column)            (:246)
//   a4  T = H X^H in M2, C = X T in M0 (lower tiles, mirrored), so that
//       C = L^-1 H L^-H; for the spin-wave metric H = diag(I, -I) the first
//       product is a sign flip of X^H                              (:248)
//   a5  C = Q T Q^H (Householder, lower; v_k kept in column k of M0 below
//       the subdiagonal; in 16-column panels whose trailing update A -= V W^H +
//       W V^H is a GEMM, small n (tiled_rows) in one pass per column),
//       T = Z diag(w) Z^T by divide and conquer (Z and its merge workspace in
//       M2, merge products through Zo), V = Q Z with compact-WY
//       blocks of 16 reflectors, Q_b = I - Y T_b Y^H, two blocks at a time on
//       strips of 8 columns of V, a warp each, V in the output U   (:250)
//   a6  U = X^H V into M2, copied to the output                   (:252)
//   a7  W ascending, U columns in the same order                  (:268-276)
//
// Stage-wise outputs (stage 1: L, 2: C, 3: W and V) follow the reference's
// static kernels in src/geneig_fixed.cu.
//
// Mixed-precision form (kernel mode MIXED): the Householder reduction runs in
// FP32 on a single-precision copy of C (reflectors stored in FP32); divide
// and conquer, the back-transform and everything else stay FP64; then
// Ogita-Aishima refinement steps (FP64 tensor-core GEMMs against the FP64 C,
// repeated until the correction is negligible) recover FP64 eigenpairs of C
// before U = X^H V. A pencil whose refinement does not converge, or that FP32
// cannot hold, is solved in FP64: from C in this kernel, or (`defer`) by the shared-memory kernel, which
// is the plain form of the sizes it holds.

#include "geneig_tiled_body.cuh"
#include "sunny_geneig.h"

namespace sgeig {
using namespace tiled;
namespace {

template <int NT, bool MIXED, bool ROWS>
__global__ void __launch_bounds__(NT, NT == kTiledWide ? 1 : 2) geneig_tiled_kernel(TiledArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* slot = a.scratch + (size_t)blockIdx.x * tiled_slot_elems(a.n, MIXED);
    phase_start();
    for (long long b = blockIdx.x; b < a.batch; b += gridDim.x) tiled_solve<NT, MIXED, ROWS>(a, b, slot, smem_raw);
}

using TiledKernelFn = void (*)(TiledArgs);
TiledKernelFn tiled_kernel(int n, bool mixed) {
    constexpr int W = kTiledWide, N = kTiledNarrow;
    if (tiled_threads(n) == W) return mixed ? geneig_tiled_kernel<W, true, false> : geneig_tiled_kernel<W, false, false>;
    if (tiled_rows(n, mixed)) return mixed ? geneig_tiled_kernel<N, true, true> : geneig_tiled_kernel<N, false, true>;
    return mixed ? geneig_tiled_kernel<N, true, false> : geneig_tiled_kernel<N, false, false>;
}

}  // namespace

int tiled_threads_for(int n) { return tiled_threads(n); }
int tiled_slots_for(int n) { return tiled_threads(n) == kTiledWide ? 1 : 2; }

size_t tiled_vec_bytes(int n, bool mixed) {
    return tiled_base_bytes(n) + (!tiled_rows(n, mixed) ? tiled_work_elems(n) * 16
                                : mixed && tiled_keep32(n) ? tiled_c32_bytes(n) : 0);
}

// `smem` is the per-CTA shared-memory limit; the kernel's own static shared
// memory (profiling builds have some) comes off the dynamic allowance.
cudaError_t tiled_set_attributes(int n, bool mixed, size_t smem) {
    const TiledKernelFn k = tiled_kernel(n, mixed);
    cudaFuncAttributes fa{};
    const cudaError_t e = cudaFuncGetAttributes(&fa, k);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem - fa.sharedSizeBytes));
}

cudaError_t tiled_launch(int n, int slots, int stage, const void* H, const void* S, double* W, void* U,
                         int* info, long long batch, void* scratch, cudaStream_t stream, bool sigma, bool mixed,
                         int refine_max, bool defer, cudaEvent_t started) {
    if (batch <= 0) return cudaSuccess;
    TiledArgs a;
    a.H = static_cast<const double2*>(H);
    a.S = static_cast<const double2*>(S);
    a.W = W;
    a.U = static_cast<double2*>(U);
    a.info = info;
    a.scratch = static_cast<double2*>(scratch);
    a.batch = batch;
    a.n = n;
    a.ld = n | 1;
    a.stage = stage;
    a.sigma = sigma ? 1 : 0;
    a.refine_max = refine_max;
    a.defer = defer ? 1 : 0;
    a.work = tiled_rows(n, mixed) ? 0 : 1;
    a.keep32 = mixed && tiled_keep32(n) ? 1 : 0;
    const size_t smem = tiled_vec_bytes(n, mixed);
    const long long grid = batch < slots ? batch : slots;
    return launch_with_event(tiled_kernel(n, mixed), (unsigned)grid, tiled_threads(n), smem, stream, started, a);
}

}  // namespace sgeig
