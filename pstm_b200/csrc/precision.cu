// precision.cu -- the precision form's trace format: FP32 traces stored as
// FP16 with one power-of-two scale per trace.
//
// FP16 keeps 11 significant bits (BF16 keeps 8), so a noise-dominated panel
// stored in FP16 stays within the 1e-3 image error of the FP32 panel where
// BF16 does not; its narrow exponent range (normal numbers from 2^-14 to
// 65504) is what the per-trace scale is for.  Each trace is multiplied by
// 2^e, e chosen so that its largest |amplitude| lands in [2^13, 2^14) -- exact
// in FP32, and with headroom to FP16's largest finite value -- and its weight
// is multiplied by 2^-e, also exact.  The migration kernel already multiplies
// every contribution by the trace weight, so the scale costs nothing per pair:
// amplitude * weight is the FP32 trace's, up to the FP16 rounding.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cmath>
#include <string>

#include "pstm_cuda.h"
#include "ctx.h"

using namespace pstm;
using namespace pstm::ctx;

namespace {

constexpr int kWarpsPerCta = 8;

// The exponent e of a trace's scale 2^e from its largest |amplitude|.
__device__ __forceinline__ int scale_exponent(float m) {
    if (!(m > 0.f && isfinite(m))) return 0;
    int ex;
    frexpf(m, &ex);   // m = f 2^ex, f in [0.5, 1)
    return 14 - ex;   // m 2^e in [2^13, 2^14)
}
__device__ __forceinline__ float warp_max(float m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
}
__device__ __forceinline__ float max4(float m, const float4 &v) {
    return fmaxf(fmaxf(fmaxf(m, fabsf(v.x)), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
}

// One warp per trace: the largest |amplitude|, then the scaled FP16 row and
// the trace weight divided by the scale.
//
// Bound by memory: 6 bytes a sample.  The row is read once, 16 bytes a lane, and
// waits in registers (kVectors float4 a lane) for its maximum; FP16 samples are
// written 8 bytes a lane.  Rows start on any element, so the vectors start at the
// first 16-byte boundary of the source, which is an 8-byte boundary of the
// destination whenever both start on the same element modulo 4 (always, for
// panels of one stride on aligned bases); rows where they do not, and rows longer
// than the registers hold, are read twice, a sample at a time.  40,000 x 1501
// samples: 78 us a call that way, 61 us this way (360 MB at 5.9 TB/s, 0.90 of the
// measured copy).
constexpr int kVectors = 16;
__global__ void __launch_bounds__(32 * kWarpsPerCta)
traces_to_f16_kernel(const float *__restrict__ src, int64_t n, int ns, int64_t src_stride, __half *__restrict__ dst,
                     int64_t dst_stride, const double *__restrict__ w_in, double *__restrict__ w_out) {
    const int lane = threadIdx.x & 31;
    const int64_t tr = (int64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
    if (tr >= n) return;
    const float *row = src + tr * src_stride;
    __half *out = dst + tr * dst_stride;
    const int head = min(ns, (int)((4 - (reinterpret_cast<uintptr_t>(row) / 4 & 3)) & 3));
    const int n4 = (ns - head) / 4, tail = head + 4 * n4;   // samples [tail, ns) are left over
    int e;
    if (n4 <= 32 * kVectors && ((reinterpret_cast<uintptr_t>(out) / 2 + head) & 3) == 0) {
        const float4 *rv = reinterpret_cast<const float4 *>(row + head);
        float4 v[kVectors];
#pragma unroll
        for (int j = 0; j < kVectors; ++j)
            v[j] = lane + 32 * j < n4 ? __ldcs(rv + lane + 32 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
        // the up to 3 + 3 samples around the vectors, one a lane
        const int loose = lane < head ? lane : (lane - head < ns - tail ? tail + lane - head : -1);
        const float x = loose >= 0 ? row[loose] : 0.f;
        float m = fabsf(x);
        m = fmaxf(0.f, m);   // (a NaN does not count)
#pragma unroll
        for (int j = 0; j < kVectors; ++j) m = max4(m, v[j]);
        e = scale_exponent(warp_max(m));
        const float scale = ldexpf(1.f, e);
        uint2 *ov = reinterpret_cast<uint2 *>(out + head);
#pragma unroll
        for (int j = 0; j < kVectors; ++j) {
            if (lane + 32 * j >= n4) continue;
            const __half2 a = __floats2half2_rn(v[j].x * scale, v[j].y * scale);
            const __half2 b = __floats2half2_rn(v[j].z * scale, v[j].w * scale);
            __stcs(ov + lane + 32 * j, make_uint2(*reinterpret_cast<const unsigned *>(&a),
                                                  *reinterpret_cast<const unsigned *>(&b)));
        }
        if (loose >= 0) out[loose] = __float2half_rn(x * scale);
    } else {
        float m = 0.f;
        for (int i = lane; i < ns; i += 32) m = fmaxf(m, fabsf(row[i]));
        e = scale_exponent(warp_max(m));
        const float scale = ldexpf(1.f, e);
        for (int i = lane; i < ns; i += 32) out[i] = __float2half_rn(row[i] * scale);
    }
    if (lane == 0) w_out[tr] = (w_in ? w_in[tr] : 1.0) * ldexp(1.0, -e);
}

}  // namespace

extern "C" int32_t pstm_cuda_traces_to_f16(void *ctx, const float *src, int64_t n_traces, int32_t n_samples,
                                           int64_t src_stride, void *dst, int64_t dst_stride,
                                           const double *weights, double *weights_out, void *stream) {
    Ctx *c = reinterpret_cast<Ctx *>(ctx);
    if (!c) return fail(nullptr, PSTM_ERR_NOT_INITIALIZED, "Kernel not initialized");
    if (n_traces < 0 || n_samples < 1 || src_stride < n_samples || dst_stride < n_samples)
        return fail(c, PSTM_ERR_INVALID_ARGUMENT, "traces_to_f16: bad sizes or strides");
    if (n_traces == 0) return PSTM_OK;
    if (!src || !dst || !weights_out) return fail(c, PSTM_ERR_INVALID_ARGUMENT, "traces_to_f16: null pointer");
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return cuda_fail(c, e, "cudaSetDevice");
    cudaStream_t st = stream ? reinterpret_cast<cudaStream_t>(stream) : c->stream;
    const int64_t blocks = (n_traces + kWarpsPerCta - 1) / kWarpsPerCta;
    if (blocks > 0x7fffffff) return fail(c, PSTM_ERR_UNSUPPORTED, "traces_to_f16: too many traces for one launch");
    traces_to_f16_kernel<<<(unsigned)blocks, 32 * kWarpsPerCta, 0, st>>>(
        src, n_traces, n_samples, src_stride, reinterpret_cast<__half *>(dst), dst_stride, weights, weights_out);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(c, e, "traces_to_f16 launch");
    return PSTM_OK;
}
