// migrate_dispatch.cuh -- picks the kernel instantiation.  Every traveltime
// kind is instantiated in its own translation unit (migrate_k<kind>.cu) so
// that they compile in parallel.
#pragma once
#include <mutex>

#include "launch.h"
#include "migrate.cuh"

namespace pstm {

// Dynamic shared-memory opt-in of one kernel.  cudaFuncSetAttribute applies to
// the calling thread's current device only, so the size set so far is kept per
// device; the mutex orders host threads that launch concurrently.
struct SmemOptIn {
    static constexpr int kMaxDevices = 64;
    std::mutex mu;
    size_t configured[kMaxDevices] = {};
};

template <typename Kernel>
static cudaError_t opt_in_smem(SmemOptIn &state, Kernel kern, size_t smem) {
    if (smem <= 48 * 1024) return cudaSuccess;   // within the default limit
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= SmemOptIn::kMaxDevices)
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    std::lock_guard<std::mutex> lock(state.mu);
    if (smem <= state.configured[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) state.configured[dev] = smem;
    return e;
}

template <int TT, int PREC, bool W2, bool AA, bool KZ>
static cudaError_t launch_one(const KParams &P, const Launch &L) {
    auto kern = gather_kernel<TT, PREC, W2, AA, KZ>;
    static SmemOptIn opt_in;   // per instantiation
    cudaError_t e = opt_in_smem(opt_in, kern, L.smem);
    if (e != cudaSuccess || L.configure_only) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(L.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = L.smem;
    cfg.stream = L.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)P.n_splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = P.n_splits > 1 ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kern, P);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

template <int TT, int PREC, bool KZ>
static cudaError_t launch_weights(const KParams &P, const Launch &L) {
    const bool w2 = P.spreading && P.obliquity;
    if (P.aa) return w2 ? launch_one<TT, PREC, true, true, KZ>(P, L) : launch_one<TT, PREC, false, true, KZ>(P, L);
    return w2 ? launch_one<TT, PREC, true, false, KZ>(P, L) : launch_one<TT, PREC, false, false, KZ>(P, L);
}

template <int TT, int PREC>
static cudaError_t launch_prec(const KParams &P, const Launch &L) {
    if constexpr (TT == TT_CURVED || TT == TT_CURVED_VTI)
        if (P.cr_k_zero) return launch_weights<TT, PREC, true>(P, L);
    return launch_weights<TT, PREC, false>(P, L);
}

template <int TT>
cudaError_t launch_gather(const KParams &P, int prec, const Launch &L) {
    if (prec == PSTM_PREC_EXACT) return launch_prec<TT, PSTM_PREC_EXACT>(P, L);
    if (prec == PSTM_PREC_FAST) return launch_prec<TT, PSTM_PREC_FAST>(P, L);
    return launch_prec<TT, PSTM_PREC_FP32>(P, L);
}

}  // namespace pstm
