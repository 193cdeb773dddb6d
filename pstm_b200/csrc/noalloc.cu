// noalloc.cu -- pstm_cuda_migrate_tile_noalloc: the migration of one tile
// without any device-memory allocation.
//
// Some callers cannot allocate device memory while they run: a host
// application whose memory manager reserves the whole GPU up front and owns
// every byte of it, or a long-running job that must not fail on an allocation
// (or stall the device: cudaMalloc synchronizes it) once it has started
// processing tiles.  The gather kernel needs no scratch buffers: its parameters
// travel with the launch, and this entry point adds only an error word in this
// module's device memory.  The caller passes its inputs and outputs as device
// pointers, as to pstm_cuda_migrate_tile_dev.
//
// One call takes at most the sizes below; larger trace sets can be split over
// several calls, since the image and fold are accumulated with "+=".  All calls
// share the error word, so calls whose work overlaps on the GPU (different
// streams, different host threads) race for it and must be serialised by the
// caller.
//
// The kernel reports device-side failures (a bounded wait for a chunk of traces
// that gave up) in the error word; pstm_cuda_noalloc_status reads it back once
// the caller's stream has drained.
#include <cuda_runtime.h>
#include <cstdio>
#include <mutex>
#include <string>

#include "pstm_cuda.h"
#include "kparams.h"
#include "launch.h"
#include "plan.h"

namespace pstm {
void set_context_free_error(const std::string &msg);
}  // namespace pstm

using namespace pstm;

namespace {

constexpr int64_t kMaxTraces = 131072;               // limits of one call (the interface's)
constexpr int64_t kMaxTable = 262144;                // (pillar | 0, time) points
constexpr int kMaxTimes = 8192;

// The error word.  Host code must not use the symbol as a pointer: it is a
// host-side stand-in.  Its device address comes from cudaGetSymbolAddress.
static __device__ int32_t g_err;

constexpr int kMaxDevices = 64;
std::mutex g_setup_mu;
int32_t *g_err_dev[kMaxDevices] = {};   // device address of g_err, per device
int g_smem_optin[kMaxDevices] = {};

int32_t fail(int32_t code, const std::string &msg) {
    set_context_free_error(msg);
    return code;
}

int32_t cuda_fail(cudaError_t e, const char *what) {
    return fail(e == cudaErrorMemoryAllocation ? PSTM_ERR_OUT_OF_MEMORY : PSTM_ERR_CUDA,
                std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")");
}

// Once per device, with that device current: the error word's device address
// and the shared-memory limit.
int32_t setup(int dev, int32_t **err, int *optin) {
    std::lock_guard<std::mutex> lock(g_setup_mu);
    if (!g_err_dev[dev]) {
        void *ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_err);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(error word)");
        int smem = 0;
        e = cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute");
        g_smem_optin[dev] = smem;
        g_err_dev[dev] = static_cast<int32_t *>(ptr);
    }
    *err = g_err_dev[dev];
    *optin = g_smem_optin[dev];
    return PSTM_OK;
}

}  // namespace

extern "C" int32_t pstm_cuda_migrate_tile_noalloc(const pstm_traces_desc *tr, const pstm_output_desc *out,
                                                  const pstm_velocity_desc *vel, const pstm_params *prm,
                                                  void *stream) {
    const char *msg = "";
    int32_t rc = plan::check_args(tr, out, vel, prm, msg);
    if (rc) return fail(rc, msg);
    if (prm->interpolation != PSTM_INTERP_LINEAR)
        return fail(PSTM_ERR_UNSUPPORTED, "the allocation-free entry point interpolates linearly");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= kMaxDevices) return fail(PSTM_ERR_UNSUPPORTED, "device index beyond the supported range");

    // size limits of one call
    const bool per_pillar = vel->is_3d || (prm->eta && prm->eta_is_3d);
    const int64_t n_p = per_pillar ? (int64_t)out->nx * out->ny : 1;
    char buf[256];
    if (tr->n_traces > kMaxTraces) {
        std::snprintf(buf, sizeof(buf),
                      "n_traces %lld exceeds the %lld traces one allocation-free call holds; split the traces "
                      "over several calls (image and fold accumulate) or use pstm_cuda_migrate_tile_dev",
                      (long long)tr->n_traces, (long long)kMaxTraces);
        return fail(PSTM_ERR_INVALID_ARGUMENT, buf);
    }
    if (out->nt > kMaxTimes || n_p * out->nt > kMaxTable) {
        std::snprintf(buf, sizeof(buf),
                      "tile tables of %lld entries (nt %d) exceed the allocation-free limits (%lld entries, "
                      "nt <= %d); use smaller tiles or pstm_cuda_migrate_tile_dev",
                      (long long)(n_p * out->nt), out->nt, (long long)kMaxTable, kMaxTimes);
        return fail(PSTM_ERR_INVALID_ARGUMENT, buf);
    }

    int32_t *err = nullptr;
    int optin = 0;
    if ((rc = setup(dev, &err, &optin)) != PSTM_OK) return rc;
    cudaStream_t st = stream ? reinterpret_cast<cudaStream_t>(stream) : cudaStreamLegacy;

    KParams P = plan::make_params(tr, out, vel, prm);
    if (tr->n_traces == 0) return PSTM_OK;   // image += 0, fold += 0
    if (!plan::row_fits(tr, prm, out->nt, optin))
        return fail(PSTM_ERR_UNSUPPORTED, "trace rows too long to stage in shared memory");
    P.err = err;
    if ((e = cudaMemsetAsync(P.err, 0, sizeof(int32_t), st)) != cudaSuccess)
        return cuda_fail(e, "clearing the error word");
    Launch L;
    if (!plan::plan_grid(P, 1, L.grid)) return fail(PSTM_ERR_UNSUPPORTED, "tile too large for one launch");
    L.smem = plan::gather_smem(prm->traveltime);
    L.stream = st;
    e = launch_kind(prm->traveltime, P, prm->precision, L);
    if (e != cudaSuccess) return cuda_fail(e, "migrate kernel launch");
    return PSTM_OK;
}

// Status of the last allocation-free call on the current device: waits for
// `stream`, then reads the kernel's error word (a copy from its symbol into a
// host int: nothing is allocated).
extern "C" int32_t pstm_cuda_noalloc_status(void *stream) {
    cudaStream_t st = stream ? reinterpret_cast<cudaStream_t>(stream) : cudaStreamLegacy;
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(e, "waiting for the allocation-free call");
    int32_t w = 0;
    e = cudaMemcpyFromSymbol(&w, g_err, sizeof(w), 0, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "reading the allocation-free error word");
    if (w & KERR_WAIT_TIMEOUT)
        return fail(PSTM_ERR_TIMEOUT,
                    "a bounded wait for a chunk of traces gave up in the last allocation-free call; its image "
                    "and fold may hold partial sums and must be discarded");
    return PSTM_OK;
}
