// launch.h -- host-side launch descriptor of the gather kernel.  The kernel
// template is instantiated only in migrate_k<kind>.cu; host files include this
// header, not the kernel source.
#pragma once
#include <cuda_runtime.h>

#include "kparams.h"
#include "pstm_cuda.h"

namespace pstm {

// One launch: `grid` CTAs, in clusters of P.n_splits.
struct Launch {
    unsigned grid = 0;
    size_t smem = 0;
    cudaStream_t stream = nullptr;
    bool configure_only = false;   // set the shared-memory opt-in and launch nothing
};

template <int TT>
cudaError_t launch_gather(const KParams &P, int prec, const Launch &L);
// each kind is instantiated in its own migrate_k<kind>.cu, nowhere else
extern template cudaError_t launch_gather<TT_STRAIGHT>(const KParams &, int, const Launch &);
extern template cudaError_t launch_gather<TT_CURVED>(const KParams &, int, const Launch &);
extern template cudaError_t launch_gather<TT_VTI>(const KParams &, int, const Launch &);
extern template cudaError_t launch_gather<TT_CURVED_VTI>(const KParams &, int, const Launch &);

// prec (pstm_precision) selects the FP64 sample-index path, FP32 traveltime
// with FP64 trace-end re-decisions, or FP32 throughout.
inline cudaError_t launch_kind(int traveltime, const KParams &P, int prec, const Launch &L) {
    switch (traveltime) {
    case PSTM_TT_STRAIGHT: return launch_gather<TT_STRAIGHT>(P, prec, L);
    case PSTM_TT_CURVED: return launch_gather<TT_CURVED>(P, prec, L);
    case PSTM_TT_VTI: return launch_gather<TT_VTI>(P, prec, L);
    default: return launch_gather<TT_CURVED_VTI>(P, prec, L);
    }
}

}  // namespace pstm
