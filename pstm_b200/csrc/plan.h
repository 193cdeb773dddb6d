// plan.h -- host-side launch planning shared by the entry points: argument
// checks, launch parameters and the grid.
#pragma once
#include <cuda_runtime.h>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "pstm_cuda.h"
#include "kparams.h"
#include "migrate.cuh"

namespace pstm {
namespace plan {

inline size_t amp_elem_bytes(int32_t dt) { return dt == PSTM_AMP_F32 ? 4 : 2; }

// Largest double B such that the correctly rounded sqrt(B) <= a, i.e. the
// FP64 predicate "sqrt(d2) > a" used by the reference equals "d2 > B".
inline double sqrt_threshold(double a) {
    double b = a * a;
    while (std::sqrt(b) > a) b = std::nextafter(b, 0.0);
    while (std::sqrt(std::nextafter(b, INFINITY)) <= a) b = std::nextafter(b, INFINITY);
    return b;
}

// Argument checks shared by every entry point; on failure `msg` says why.
inline int32_t check_args(const pstm_traces_desc *tr, const pstm_output_desc *out,
                          const pstm_velocity_desc *vel, const pstm_params *prm, const char *&msg) {
    auto fail = [&](int32_t code, const char *m) { msg = m; return code; };
    if (!tr || !out || !vel || !prm) return fail(PSTM_ERR_INVALID_ARGUMENT, "null descriptor");
    if (tr->n_traces < 0) return fail(PSTM_ERR_INVALID_ARGUMENT, "n_traces < 0");
    if (tr->n_samples < 2) return fail(PSTM_ERR_INVALID_ARGUMENT, "n_samples must be >= 2");
    if (tr->amp_dtype < PSTM_AMP_F32 || tr->amp_dtype > PSTM_AMP_F16)
        return fail(PSTM_ERR_INVALID_ARGUMENT, "unknown amplitude dtype");
    if (tr->amp_row_stride < tr->n_samples)
        return fail(PSTM_ERR_INVALID_ARGUMENT, "amp_row_stride < n_samples");
    if (tr->n_traces > 0 && (!tr->amplitudes || !tr->source_x || !tr->source_y || !tr->receiver_x ||
                             !tr->receiver_y || !tr->midpoint_x || !tr->midpoint_y))
        return fail(PSTM_ERR_INVALID_ARGUMENT, "null trace array");
    if (!(tr->sample_rate_ms > 0.0)) return fail(PSTM_ERR_INVALID_ARGUMENT, "sample_rate_ms must be > 0");
    if (out->nx <= 0 || out->ny <= 0 || out->nt <= 0)
        return fail(PSTM_ERR_INVALID_ARGUMENT, "empty output tile");
    if (!out->image) return fail(PSTM_ERR_INVALID_ARGUMENT, "null image");
    if (out->image_dtype != PSTM_IMAGE_F64 && out->image_dtype != PSTM_IMAGE_F32)
        return fail(PSTM_ERR_INVALID_ARGUMENT, "unknown image dtype");
    if (!out->t_axis_ms) return fail(PSTM_ERR_INVALID_ARGUMENT, "null t axis");
    if ((!out->x_grid || !out->y_grid) && (!out->x_axis || !out->y_axis))
        return fail(PSTM_ERR_INVALID_ARGUMENT, "need x/y axes or x/y grids");
    if ((out->x_grid == nullptr) != (out->y_grid == nullptr))
        return fail(PSTM_ERR_INVALID_ARGUMENT, "x_grid and y_grid must be given together");
    if (!vel->vrms) return fail(PSTM_ERR_INVALID_ARGUMENT, "null velocity");
    if (prm->traveltime < PSTM_TT_STRAIGHT || prm->traveltime > PSTM_TT_CURVED_VTI)
        return fail(PSTM_ERR_INVALID_ARGUMENT, "unknown traveltime kind");
    if (prm->precision != PSTM_PREC_EXACT && prm->precision != PSTM_PREC_FAST && prm->precision != PSTM_PREC_FP32)
        return fail(PSTM_ERR_INVALID_ARGUMENT, "unknown precision");
    if (prm->interpolation < PSTM_INTERP_LINEAR || prm->interpolation > PSTM_INTERP_LANCZOS5)
        return fail(PSTM_ERR_INVALID_ARGUMENT, "unknown interpolation method");
    if (!(prm->max_aperture_m >= 0.0) || !(prm->taper_fraction >= 0.0) || !(prm->taper_fraction <= 1.0))
        return fail(PSTM_ERR_INVALID_ARGUMENT, "bad aperture/taper parameters");
    if ((prm->traveltime == PSTM_TT_CURVED || prm->traveltime == PSTM_TT_CURVED_VTI) && !(prm->curved_v0 > 0.0))
        return fail(PSTM_ERR_INVALID_ARGUMENT, "curved_v0 must be > 0");
    return PSTM_OK;
}

// CTAs of a cluster that share the traces of an item.  A CTA's start -- its
// points' state, the first selection and copies -- costs about kStartChunks chunks
// of traces, and 2 x 148 CTAs run at a time, so S CTAs per item take about
// ceil(items S / 296) (kStartChunks + chunks / S).  A cluster also starts and ends
// together, which cost 14 % on a 32 x 32 x 800 tile (1664 items, 625 chunks) that
// this count has gain 2 % from S = 4; so every doubling has to win 15 %.  By the
// tile's size and the output's own traces alone, so that
// a bin and the same traces as a tile of their own are summed in the same order.
constexpr int kStartChunks = 4;
inline int split_traces(int64_t items, int64_t n_traces) {
    int best = 1;
    double least = INFINITY;
    for (int s = 1; s <= kMaxSplits; s *= 2) {
        const int64_t waves = (items * s + 295) / 296;
        const int64_t chunks = (n_traces + (int64_t)kChunk * s - 1) / ((int64_t)kChunk * s);
        const double cost = (double)waves * (double)(kStartChunks + chunks);
        if (cost < 0.85 * least) {
            least = cost;
            best = s;
        }
    }
    return best;
}

inline KParams make_params(const pstm_traces_desc *tr, const pstm_output_desc *out, const pstm_velocity_desc *vel,
                    const pstm_params *prm) {
    KParams P;
    std::memset(&P, 0, sizeof(P));
    P.amps = tr->amplitudes;
    P.amp_kind = tr->amp_dtype;
    P.amps_end = static_cast<const unsigned char *>(tr->amplitudes) +
                 (tr->n_traces > 0 ? ((tr->n_traces - 1) * tr->amp_row_stride + tr->n_samples) *
                                         (int64_t)amp_elem_bytes(tr->amp_dtype) : 0);
    P.amp_stride = tr->amp_row_stride;
    P.n_traces = tr->n_traces;
    P.ns = tr->n_samples;
    P.elem = (int32_t)amp_elem_bytes(tr->amp_dtype);
    P.sx = tr->source_x; P.sy = tr->source_y;
    P.rx = tr->receiver_x; P.ry = tr->receiver_y;
    P.mx = tr->midpoint_x; P.my = tr->midpoint_y;
    P.w = tr->weights;
    P.dt_s = tr->sample_rate_ms / 1000.0;
    P.inv_dt = 1.0 / P.dt_s;
    P.tstart_s = tr->start_time_ms / 1000.0;
    P.s_scale = (float)(1.0 / P.dt_s);
    P.s_offset = (float)(-P.tstart_s / P.dt_s);
    const float g = 1e-2f;   // guard band in samples around the FP64 decision boundaries
    const float smax = (float)(tr->n_samples - 1);
    P.s_guard_lo = g;
    P.s_guard_hi = smax - g;
    P.s_rej_lo = -g;
    P.s_rej_hi = smax + g;
    P.s_max_clamp = std::nextafter(smax, 0.0f);
    P.s_magic = (kIndexMagic - P.tstart_s / P.dt_s) * kTimeScale;
    P.inv_dt_f = (float)(1.0 / P.dt_s);

    P.image = out->image;
    P.fold = out->fold;
    P.image_f32 = out->image_dtype == PSTM_IMAGE_F32;
    P.fold3d = out->fold_is_3d;
    P.nx = out->nx; P.ny = out->ny; P.nt = out->nt;
    P.xa = out->x_axis; P.ya = out->y_axis;
    P.xg = out->x_grid; P.yg = out->y_grid;
    P.ta = out->t_axis_ms;

    P.vrms = vel->vrms;
    P.vel3d = vel->is_3d;
    P.eta = prm->eta;
    P.eta3d = prm->eta ? prm->eta_is_3d : 0;
    P.eta_const = prm->eta_constant;

    P.max_ap = prm->max_aperture_m;
    P.min_ap = prm->min_aperture_m;
    P.tan_dip = std::tan(prm->max_dip_degrees * M_PI / 180.0);
    P.taper = prm->taper_fraction;
    P.fold_d2_max = sqrt_threshold(prm->max_aperture_m);
    P.taper_f = (float)prm->taper_fraction;
    P.spreading = prm->apply_spreading ? 1 : 0;
    P.obliquity = prm->apply_obliquity ? 1 : 0;
    P.aa = prm->aa_enabled ? 1 : 0;
    const double gmax = prm->grid_dx > prm->grid_dy ? prm->grid_dx : prm->grid_dy;
    P.aa_cA = (float)(4.0 * gmax * prm->aa_dominant_freq);
    P.aa_cB = (float)(prm->aa_dominant_freq / 500.0);
    P.aa_gmax = gmax;
    P.aa_fdom = prm->aa_dominant_freq;
    P.cr_v0 = prm->curved_v0;
    P.cr_k = prm->curved_k;
    P.cr_k_zero = std::fabs(prm->curved_k) < 1e-10 ? 1 : 0;
    P.cr_inv_k_ln2 = P.cr_k_zero ? 0.f : (float)(M_LN2 / prm->curved_k);
    // VTI returns 2 t0/2 = 0 at t0 = 0; the curved leg of depth 0 is log(1) = 0 for k != 0
    P.t0_zero_exact = (prm->traveltime == PSTM_TT_VTI ||
                       ((prm->traveltime == PSTM_TT_CURVED || prm->traveltime == PSTM_TT_CURVED_VTI) &&
                        !P.cr_k_zero)) ? 1 : 0;
    P.exact_units = prm->precision == PSTM_PREC_EXACT ? 1 : 0;
    P.curved_kind = (prm->traveltime == PSTM_TT_CURVED || prm->traveltime == PSTM_TT_CURVED_VTI) ? 1 : 0;
    P.cr_B0 = 1.0 / (prm->curved_v0 * prm->curved_v0 * P.dt_s * P.dt_s);
    P.cr_k2 = prm->curved_k * prm->curved_k;
    P.cr_inv_k_dt = P.cr_k_zero ? 0.0 : kTimeScale / (prm->curved_k * P.dt_s);
    P.cr_inv_k_unit = P.cr_inv_k_dt / kSampleUnit;
    // FP32 partial sums over one chunk where the caller asks for compensated sums (an FP32
    // accumulation error of 32 instead of 128 terms, both below the pairs' own rounding:
    // images are 1.1e-7 from FP64 either way; 0.5 % of the time of offset bins)
    P.flush_mask = prm->compensated ? 0 : kFlush - 1;
    P.wait_iters = kWaitIters;
    // Fault injection for the tests of the bounded waits: PSTM_CUDA_INJECT_FAULT=wait
    // leaves the first trace chunks' copies unissued, so the kernel's bounded
    // wait for them runs out after a few polls and it reports KERR_WAIT_TIMEOUT.
    // Read when a launch is prepared (a captured batch keeps what it saw).
    if (const char *inj = std::getenv("PSTM_CUDA_INJECT_FAULT")) {
        if (std::strcmp(inj, "wait") == 0) {
            P.inject_stall = 1;
            P.wait_iters = 256;
        }
    }

    // Pillar patch: the px x py = kPillars rectangle that covers the tile with the
    // fewest patches, 2 x 4 first (the closer its pillars, the shorter the sample
    // ranges a CTA stages).
    const int shapes[4][2] = {{2, 4}, {4, 2}, {1, 8}, {8, 1}};
    int64_t best = -1;
    for (const auto &sh : shapes) {
        const int64_t nbx = (out->nx + sh[0] - 1) / sh[0], nby = (out->ny + sh[1] - 1) / sh[1];
        if (best >= 0 && nbx * nby >= best) continue;
        best = nbx * nby;
        P.px = sh[0];
        P.py = sh[1];
        P.n_pblk_x = (int32_t)nbx;
        P.n_pblk_y = (int32_t)nby;
    }
    P.n_tblk = (out->nt + kTimes - 1) / kTimes;
    P.n_pblk_fold = (int32_t)(((int64_t)out->nx * out->ny + kFoldPillars - 1) / kFoldPillars);
    P.max_chunk = kChunk;
    P.n_splits = split_traces(best * P.n_tblk, tr->n_traces);
    return P;
}

// The interface's limit on a trace row: two rows, the pillars' records and the
// partial sums of up to 4096 output times in one SM's shared memory.
inline bool row_fits(const pstm_traces_desc *tr, const pstm_params *prm, int nt, int smem_optin) {
    int R = (nt + 511) / 512;
    if (R > 8) R = 8;
    const int PB = (R <= 1 || tr->amp_dtype != PSTM_AMP_F32) ? 8 : 4;
    const bool has_c = prm->traveltime == PSTM_TT_CURVED || prm->traveltime == PSTM_TT_CURVED_VTI;
    const int64_t fixed = 4096 + (int64_t)PB * 1024 * (has_c ? 3 : 2) +
                          (int64_t)PB * R * 512 * (prm->compensated ? 6 : 4) + 3072;
    const int64_t eb = (int64_t)amp_elem_bytes(tr->amp_dtype), pitch = (tr->n_samples + 16 / eb - 1) / (16 / eb) * (16 / eb);
    return smem_optin >= fixed + 2 * pitch * eb;
}

// Grid of the gather kernel for `n_out` outputs of this tile: items x splits,
// then the fold-counting CTAs, in whole clusters.  False: too many for one launch.
inline bool plan_grid(const KParams &P, int64_t n_out, unsigned &grid) {
    const int64_t items = (int64_t)P.n_pblk_x * P.n_pblk_y * P.n_tblk * n_out * P.n_splits;
    const int64_t folds = ((int64_t)P.n_pblk_fold * n_out + P.n_splits - 1) / P.n_splits * P.n_splits;
    if (items + folds > 0x7fffffff) return false;
    grid = (unsigned)(items + folds);
    return true;
}

inline size_t gather_smem(int traveltime) {
    return (size_t)dynamic_bytes(traveltime != PSTM_TT_STRAIGHT);
}

}  // namespace plan
}  // namespace pstm
