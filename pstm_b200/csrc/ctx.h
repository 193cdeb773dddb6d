// ctx.h -- the context behind a pstm_cuda handle: its stream, the device
// buffers it reuses from call to call, and the state of the batched form
// (cached CUDA graph, tuned chunk depths).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <map>
#include <string>
#include <vector>

#include "pstm_cuda.h"
#include "launch.h"

namespace pstm {
namespace ctx {

struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
};

struct Ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    DevBuf errword;
    // staging for the host-pointer path
    DevBuf amps, geo[7], xa, ya, xg, yg, ta, vel, eta, image, fold;
    int smem_optin = 0;   // max dynamic shared memory per block
    // batched form
    DevBuf bins, tune_image, tune_fold;
    DevBuf probe;                           // learned form: per-probe residuals
    DevBuf runs;                            // trace ranges of a call on runs
    DevBuf seg_boxes, scatter_ends;         // scatter schedule: the segments' boxes, prefix counts of their items
    std::vector<unsigned char> graph_key;   // arguments the cached graph was captured with
    cudaGraphExec_t graph = nullptr;
    std::map<std::string, int> tuned;       // autotuned traces per chunk by workload class
};

// A launch prepared by prepare_tile: the parameters and grid of one tile, its
// error word cleared; the migration launch is not enqueued.
struct TilePlan {
    KParams P;
    Launch L;
    int tt = 0, amp = 0;
    bool exact = false;
    int prec = PSTM_PREC_EXACT;   // pstm_precision of the launch
    bool empty = true;   // no traces: nothing to launch
};

int32_t prepare_tile(Ctx *c, const pstm_traces_desc *tr, const pstm_output_desc *out, const pstm_velocity_desc *vel,
                     const pstm_params *prm, cudaStream_t st, TilePlan &tp);
int32_t launch_tile(Ctx *c, const TilePlan &tp);
int32_t launch_interp(Ctx *c, const TilePlan &tp, int method, const pstm_output_desc *out);   // interp.cu
int32_t check_error_word(Ctx *c);   // after the stream has drained

int32_t fail(Ctx *c, int32_t code, const std::string &msg);
int32_t cuda_fail(Ctx *c, cudaError_t e, const char *what);
bool injected(const char *site);
cudaError_t ensure(DevBuf &b, size_t bytes);
void release(DevBuf &b);
void release_batch(Ctx *c);   // batch.cu

}  // namespace ctx
}  // namespace pstm
