// capi.cu -- the C ABI declared in include/pstm_cuda.h: contexts, argument
// validation, launch-parameter derivation and the host-pointer staging path.
#include <cuda_runtime.h>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "pstm_cuda.h"
#include "kparams.h"
#include "launch.h"
#include "plan.h"
#include "ctx.h"

using namespace pstm;

namespace {
thread_local std::string g_create_err;
}

namespace pstm {
// Message of the last failing call that has no context (create, noalloc).
void set_context_free_error(const std::string &msg) { g_create_err = msg; }

namespace ctx {

int32_t fail(Ctx *c, int32_t code, const std::string &msg) {
    if (c) c->err = msg;
    else g_create_err = msg;
    return code;
}

int32_t cuda_fail(Ctx *c, cudaError_t e, const char *what) {
    std::string m = std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")";
    return fail(c, e == cudaErrorMemoryAllocation ? PSTM_ERR_OUT_OF_MEMORY : PSTM_ERR_CUDA, m);
}

bool injected(const char *site) {
    const char *v = std::getenv("PSTM_CUDA_INJECT_FAULT");
    if (!v || !*v) return false;
    return std::strcmp(v, site) == 0 || std::strcmp(v, "all") == 0;
}

cudaError_t ensure(DevBuf &b, size_t bytes) {
    if (bytes <= b.bytes && b.ptr) return cudaSuccess;
    if (b.ptr) {
        cudaFree(b.ptr);
        b.ptr = nullptr;
        b.bytes = 0;
    }
    size_t want = bytes < 256 ? 256 : bytes;
    cudaError_t e = cudaMalloc(&b.ptr, want);
    if (e == cudaSuccess) b.bytes = want;
    return e;
}

void release(DevBuf &b) {
    if (b.ptr) cudaFree(b.ptr);
    b.ptr = nullptr;
    b.bytes = 0;
}

}  // namespace ctx
}  // namespace pstm

namespace {

using namespace pstm::ctx;

using plan::amp_elem_bytes;
using plan::make_params;

int32_t validate(Ctx *c, const pstm_traces_desc *tr, const pstm_output_desc *out,
                 const pstm_velocity_desc *vel, const pstm_params *prm) {
    const char *msg = "";
    const int32_t rc = plan::check_args(tr, out, vel, prm, msg);
    return rc ? fail(c, rc, msg) : PSTM_OK;
}

}  // namespace

namespace pstm {
namespace ctx {

int32_t prepare_tile(Ctx *c, const pstm_traces_desc *tr, const pstm_output_desc *out, const pstm_velocity_desc *vel,
                     const pstm_params *prm, cudaStream_t st, TilePlan &tp) {
    tp.empty = true;
    int32_t rc = validate(c, tr, out, vel, prm);
    if (rc) return rc;
    if (injected("migrate")) return fail(c, PSTM_ERR_INJECTED, "injected fault: migrate");
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return cuda_fail(c, e, "cudaSetDevice");
    KParams &P = tp.P;
    P = make_params(tr, out, vel, prm);
    if (tr->n_traces == 0) return PSTM_OK;   // nothing to add: image += 0, fold += 0
    if (!plan::row_fits(tr, prm, out->nt, c->smem_optin))
        return fail(c, PSTM_ERR_UNSUPPORTED, "trace rows too long to stage in shared memory");
    if ((e = ensure(c->errword, sizeof(int32_t))) != cudaSuccess)
        return cuda_fail(c, e, "allocating the error word");
    P.err = reinterpret_cast<int32_t *>(c->errword.ptr);
    if ((e = cudaMemsetAsync(P.err, 0, sizeof(int32_t), st)) != cudaSuccess)
        return cuda_fail(c, e, "clearing the error word");
    tp.L = Launch();
    if (!plan::plan_grid(P, 1, tp.L.grid)) return fail(c, PSTM_ERR_UNSUPPORTED, "tile too large for one launch");
    tp.L.smem = plan::gather_smem(prm->traveltime);
    tp.L.stream = st;
    tp.tt = prm->traveltime;
    tp.amp = tr->amp_dtype;
    tp.exact = prm->precision == PSTM_PREC_EXACT;
    tp.prec = prm->precision;
    tp.empty = false;
    return PSTM_OK;
}

int32_t launch_tile(Ctx *c, const TilePlan &tp) {
    const cudaError_t e = launch_kind(tp.tt, tp.P, tp.prec, tp.L);
    return e == cudaSuccess ? PSTM_OK : cuda_fail(c, e, "migrate kernel launch");
}

}  // namespace ctx
}  // namespace pstm

namespace {

int32_t run_dev(Ctx *c, const pstm_traces_desc *tr, const pstm_output_desc *out,
                const pstm_velocity_desc *vel, const pstm_params *prm, cudaStream_t st) {
    TilePlan tp;
    const int32_t rc = prepare_tile(c, tr, out, vel, prm, st, tp);
    if (rc || tp.empty) return rc;
    if (prm->interpolation != PSTM_INTERP_LINEAR) return launch_interp(c, tp, prm->interpolation, out);
    return launch_tile(c, tp);
}

}  // namespace

// Read back the kernels' error word (after the stream has drained).
int32_t pstm::ctx::check_error_word(Ctx *c) {
    if (!c->errword.ptr) return PSTM_OK;
    int32_t w = 0;
    cudaError_t e = cudaMemcpy(&w, c->errword.ptr, sizeof(w), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(c, e, "reading the error word");
    if (w & KERR_UNSORTED_AXIS)
        return fail(c, PSTM_ERR_INVALID_ARGUMENT,
                    "the scatter schedule needs ascending x and y axes; the image and fold were not computed "
                    "correctly and must be discarded");
    if (w & KERR_WAIT_TIMEOUT)
        return fail(c, PSTM_ERR_TIMEOUT,
                    "a bounded wait for a chunk of traces gave up; the image and fold may hold partial sums "
                    "of this call and must be discarded");
    return PSTM_OK;
}

namespace {

template <typename T>
cudaError_t stage(DevBuf &b, const T *src, size_t count, cudaStream_t st, const T **dst) {
    if (!src) {
        *dst = nullptr;
        return cudaSuccess;
    }
    cudaError_t e = ensure(b, count * sizeof(T));
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(b.ptr, src, count * sizeof(T), cudaMemcpyHostToDevice, st);
    *dst = reinterpret_cast<const T *>(b.ptr);
    return e;
}

}  // namespace

extern "C" {

int32_t pstm_cuda_abi_version(void) { return PSTM_CUDA_ABI_VERSION; }

int32_t pstm_cuda_create(int32_t device, void **ctx_out) {
    if (!ctx_out) return fail(nullptr, PSTM_ERR_INVALID_ARGUMENT, "ctx_out is null");
    *ctx_out = nullptr;
    if (injected("create")) return fail(nullptr, PSTM_ERR_INJECTED, "injected fault: create");
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaGetDeviceCount");
    if (device < 0 || device >= n) return fail(nullptr, PSTM_ERR_INVALID_ARGUMENT, "device index out of range");
    e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaSetDevice");
    Ctx *c = new Ctx();
    c->device = device;
    e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete c;
        return cuda_fail(nullptr, e, "cudaStreamCreate");
    }
    e = cudaDeviceGetAttribute(&c->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) {
        cudaStreamDestroy(c->stream);
        delete c;
        return cuda_fail(nullptr, e, "cudaDeviceGetAttribute");
    }
    *ctx_out = c;
    return PSTM_OK;
}

void pstm_cuda_destroy(void *ctx) {
    Ctx *c = reinterpret_cast<Ctx *>(ctx);
    if (!c) return;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    release(c->errword);
    release(c->amps);
    for (auto &g : c->geo) release(g);
    release(c->xa); release(c->ya); release(c->xg); release(c->yg); release(c->ta);
    release(c->vel); release(c->eta); release(c->image); release(c->fold);
    release(c->runs);
    release(c->seg_boxes);
    release(c->scatter_ends);
    release_batch(c);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
}

int32_t pstm_cuda_migrate_tile_dev(void *ctx, const pstm_traces_desc *traces, const pstm_output_desc *output,
                                   const pstm_velocity_desc *velocity, const pstm_params *params, void *stream) {
    Ctx *c = reinterpret_cast<Ctx *>(ctx);
    if (!c) return fail(nullptr, PSTM_ERR_NOT_INITIALIZED, "Kernel not initialized");
    cudaStream_t st = stream ? reinterpret_cast<cudaStream_t>(stream) : c->stream;
    return run_dev(c, traces, output, velocity, params, st);
}

namespace {

// The traces [a, a + n) of a panel as a panel of their own (no copy).
pstm_traces_desc sub_panel(const pstm_traces_desc &t, int64_t a, int64_t n) {
    pstm_traces_desc s = t;
    s.amplitudes = static_cast<const unsigned char *>(t.amplitudes) +
                   a * t.amp_row_stride * (int64_t)amp_elem_bytes(t.amp_dtype);
    s.source_x = t.source_x + a;
    s.source_y = t.source_y + a;
    s.receiver_x = t.receiver_x + a;
    s.receiver_y = t.receiver_y + a;
    s.midpoint_x = t.midpoint_x + a;
    s.midpoint_y = t.midpoint_y + a;
    if (t.weights) s.weights = t.weights + a;
    s.n_traces = n;
    return s;
}

}  // namespace

int32_t pstm_cuda_migrate_tile_runs_dev(void *ctx, const pstm_traces_desc *traces, const int64_t *runs,
                                        int32_t n_runs, const pstm_output_desc *output,
                                        const pstm_velocity_desc *velocity, const pstm_params *params,
                                        void *stream) {
    Ctx *c = reinterpret_cast<Ctx *>(ctx);
    if (!c) return fail(nullptr, PSTM_ERR_NOT_INITIALIZED, "Kernel not initialized");
    if (!traces || n_runs < 0 || (n_runs > 0 && !runs))
        return fail(c, PSTM_ERR_INVALID_ARGUMENT, "runs: n_runs >= 0 [begin, end) pairs required");
    int32_t rc = validate(c, traces, output, velocity, params);
    if (rc) return rc;
    std::vector<std::pair<int64_t, int64_t>> rv;
    int64_t prev = 0;
    for (int32_t i = 0; i < n_runs; ++i) {
        const int64_t a = runs[2 * i], b = runs[2 * i + 1];
        if (a < prev || b < a || b > traces->n_traces)
            return fail(c, PSTM_ERR_INVALID_ARGUMENT,
                        "runs must be ascending, disjoint [begin, end) trace ranges inside the panel");
        prev = b;
        if (b > a) rv.emplace_back(a, b);
    }
    if (rv.empty()) return PSTM_OK;   // no traces: image += 0, fold += 0
    cudaStream_t st = stream ? reinterpret_cast<cudaStream_t>(stream) : c->stream;
    if (params->interpolation != PSTM_INTERP_LINEAR || rv.size() == 1) {
        for (const auto &r : rv) {
            const pstm_traces_desc sub = sub_panel(*traces, r.first, r.second - r.first);
            if ((rc = run_dev(c, &sub, output, velocity, params, st)) != PSTM_OK) return rc;
        }
        return PSTM_OK;
    }
    // One launch whose CTAs walk the ranges.
    TilePlan tp;
    if ((rc = prepare_tile(c, traces, output, velocity, params, st, tp)) != PSTM_OK || tp.empty) return rc;
    cudaError_t e;
    if ((e = ensure(c->runs, rv.size() * 2 * sizeof(int64_t))) != cudaSuccess)
        return cuda_fail(c, e, "allocating the run list");
    std::vector<int64_t> flat;
    for (const auto &r : rv) {
        flat.push_back(r.first);
        flat.push_back(r.second);
        tp.P.n_run_traces += r.second - r.first;
    }
    if ((e = cudaMemcpyAsync(c->runs.ptr, flat.data(), flat.size() * sizeof(int64_t), cudaMemcpyHostToDevice, st)) !=
        cudaSuccess)
        return cuda_fail(c, e, "writing the run list");
    tp.P.runs = reinterpret_cast<const int64_t *>(c->runs.ptr);
    tp.P.n_runs = (int32_t)rv.size();
    tp.P.n_splits = plan::split_traces((int64_t)tp.P.n_pblk_x * tp.P.n_pblk_y * tp.P.n_tblk, tp.P.n_run_traces);
    if (!plan::plan_grid(tp.P, 1, tp.L.grid)) return fail(c, PSTM_ERR_UNSUPPORTED, "tile too large for one launch");
    return launch_tile(c, tp);
}

static int32_t migrate_host_impl(Ctx *c, const pstm_traces_desc *traces, const pstm_output_desc *output,
                                 const pstm_velocity_desc *velocity, const pstm_params *params);

int32_t pstm_cuda_migrate_tile_host(void *ctx, const pstm_traces_desc *traces, const pstm_output_desc *output,
                                    const pstm_velocity_desc *velocity, const pstm_params *params) {
    Ctx *c = reinterpret_cast<Ctx *>(ctx);
    if (!c) return fail(nullptr, PSTM_ERR_NOT_INITIALIZED, "Kernel not initialized");
    int32_t rc = migrate_host_impl(c, traces, output, velocity, params);
    // On failure, drain the stream so no queued copy outlives the caller's buffers.
    if (rc != PSTM_OK && c->stream) cudaStreamSynchronize(c->stream);
    return rc;
}

static int32_t migrate_host_impl(Ctx *c, const pstm_traces_desc *traces, const pstm_output_desc *output,
                                 const pstm_velocity_desc *velocity, const pstm_params *params) {
    int32_t rc = validate(c, traces, output, velocity, params);
    if (rc) return rc;
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return cuda_fail(c, e, "cudaSetDevice");
    cudaStream_t st = c->stream;
    const int64_t N = traces->n_traces;
    const int nx = output->nx, ny = output->ny, nt = output->nt;
    const size_t npix = (size_t)nx * ny * nt;

    pstm_traces_desc dt = *traces;
    pstm_output_desc dout = *output;
    pstm_velocity_desc dv = *velocity;
    pstm_params dp = *params;
    const size_t eb = amp_elem_bytes(traces->amp_dtype);
    // amplitudes: packed to n_samples per row on the device
    if (N > 0) {
        // rows padded to a 16-byte pitch so the kernel can stage them with TMA bulk copies
        const size_t per16 = 16 / eb;
        const size_t pitch = ((size_t)traces->n_samples + per16 - 1) / per16 * per16;
        e = ensure(c->amps, (size_t)N * pitch * eb);
        if (e != cudaSuccess) return cuda_fail(c, e, "staging amplitudes");
        e = cudaMemcpy2DAsync(c->amps.ptr, pitch * eb, traces->amplitudes,
                              traces->amp_row_stride * eb, traces->n_samples * eb, (size_t)N,
                              cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return cuda_fail(c, e, "copying amplitudes");
        dt.amplitudes = c->amps.ptr;
        dt.amp_row_stride = (int64_t)pitch;
    }
    const double *src_geo[7] = {traces->source_x, traces->source_y, traces->receiver_x, traces->receiver_y,
                                traces->midpoint_x, traces->midpoint_y, traces->weights};
    const double *dst_geo[7];
    for (int i = 0; i < 7; ++i) {
        e = stage(c->geo[i], N > 0 ? src_geo[i] : nullptr, (size_t)N, st, &dst_geo[i]);
        if (e != cudaSuccess) return cuda_fail(c, e, "copying geometry");
    }
    dt.source_x = dst_geo[0]; dt.source_y = dst_geo[1];
    dt.receiver_x = dst_geo[2]; dt.receiver_y = dst_geo[3];
    dt.midpoint_x = dst_geo[4]; dt.midpoint_y = dst_geo[5];
    dt.weights = dst_geo[6];

    if ((e = stage(c->xa, output->x_axis, (size_t)nx, st, &dout.x_axis)) != cudaSuccess ||
        (e = stage(c->ya, output->y_axis, (size_t)ny, st, &dout.y_axis)) != cudaSuccess ||
        (e = stage(c->xg, output->x_grid, (size_t)nx * ny, st, &dout.x_grid)) != cudaSuccess ||
        (e = stage(c->yg, output->y_grid, (size_t)nx * ny, st, &dout.y_grid)) != cudaSuccess ||
        (e = stage(c->ta, output->t_axis_ms, (size_t)nt, st, &dout.t_axis_ms)) != cudaSuccess)
        return cuda_fail(c, e, "copying output axes");
    const size_t nvel = velocity->is_3d ? npix : (size_t)nt;
    if ((e = stage(c->vel, velocity->vrms, nvel, st, &dv.vrms)) != cudaSuccess)
        return cuda_fail(c, e, "copying velocity");
    if (params->eta) {
        const size_t neta = params->eta_is_3d ? npix : (size_t)nt;
        if ((e = stage(c->eta, params->eta, neta, st, &dp.eta)) != cudaSuccess)
            return cuda_fail(c, e, "copying eta");
    }
    const size_t img_bytes = npix * (output->image_dtype == PSTM_IMAGE_F32 ? 4 : 8);
    if ((e = ensure(c->image, img_bytes)) != cudaSuccess) return cuda_fail(c, e, "staging image");
    if ((e = cudaMemcpyAsync(c->image.ptr, output->image, img_bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return cuda_fail(c, e, "copying image");
    dout.image = c->image.ptr;
    const size_t fold_bytes = (output->fold_is_3d ? npix : (size_t)nx * ny) * sizeof(int32_t);
    if (output->fold) {
        if ((e = ensure(c->fold, fold_bytes)) != cudaSuccess) return cuda_fail(c, e, "staging fold");
        if ((e = cudaMemcpyAsync(c->fold.ptr, output->fold, fold_bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess)
            return cuda_fail(c, e, "copying fold");
        dout.fold = reinterpret_cast<int32_t *>(c->fold.ptr);
    }
    rc = run_dev(c, &dt, &dout, &dv, &dp, st);
    if (rc) return rc;
    if ((e = cudaMemcpyAsync(output->image, c->image.ptr, img_bytes, cudaMemcpyDeviceToHost, st)) != cudaSuccess)
        return cuda_fail(c, e, "reading image back");
    if (output->fold &&
        (e = cudaMemcpyAsync(output->fold, c->fold.ptr, fold_bytes, cudaMemcpyDeviceToHost, st)) != cudaSuccess)
        return cuda_fail(c, e, "reading fold back");
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return cuda_fail(c, e, "migrate_tile");
    return check_error_word(c);
}

int32_t pstm_cuda_synchronize(void *ctx) {
    Ctx *c = reinterpret_cast<Ctx *>(ctx);
    if (!c) return fail(nullptr, PSTM_ERR_NOT_INITIALIZED, "Kernel not initialized");
    if (injected("sync")) return fail(c, PSTM_ERR_INJECTED, "injected fault: sync");
    cudaError_t e = cudaSetDevice(c->device);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "synchronize");
    return check_error_word(c);
}

const char *pstm_cuda_last_error(void *ctx) {
    Ctx *c = reinterpret_cast<Ctx *>(ctx);
    return c ? c->err.c_str() : g_create_err.c_str();
}

}  // extern "C"
