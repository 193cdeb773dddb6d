// kparams.h -- launch parameters shared by the host side (capi.cu) and the
// migration kernels.  Plain C++ struct passed by value to every launch.
#pragma once
#include <stdint.h>
#include <vector_types.h>

namespace pstm {

enum AmpKind { AMP_F32 = 0, AMP_BF16 = 1, AMP_F16 = 2 };
enum TTKind { TT_STRAIGHT = 0, TT_CURVED = 1, TT_VTI = 2, TT_CURVED_VTI = 3 };

// error bits a kernel can raise in *err
enum KernelError { KERR_WAIT_TIMEOUT = 1, KERR_UNSORTED_AXIS = 2 };

// One output of the batched form: its traces and its image/fold.
struct BinWork {
    int64_t trace0;              // first trace in the concatenated panel
    int64_t n_traces;
    void *image;
    int32_t *fold;
    int32_t shares;              // ranks among which its traces are divided (plan::split_traces)
    int32_t pad;
};

// The scatter schedule: the panel cut into segments of seg_traces traces;
// segment s reaches the pillar blocks [pbx0, pbx1] x [pby0, pby1] (empty when
// pbx0 > pbx1).
struct SegmentBox {
    int32_t pbx0, pbx1, pby0, pby1;
};

struct KParams {
    // ---- traces ----
    const void *amps;
    const void *amps_end;        // one past the panel's last sample
    int64_t amp_stride;          // elements between rows
    int64_t n_traces;
    int32_t ns;                  // samples per trace
    int32_t elem;                // bytes per amplitude
    int32_t amp_kind;            // AmpKind
    int32_t pad0;
    const double *sx, *sy, *rx, *ry, *mx, *my, *w;   // w nullable
    double dt_s, inv_dt, tstart_s;   // input sampling (seconds), 1 / dt
    float s_scale, s_offset;     // sample index s = T * s_scale + s_offset
    float s_guard_lo, s_guard_hi;  // fast-path accept window for s
    float s_rej_lo, s_rej_hi;    // outside [s_rej_lo, s_rej_hi] the pair is rejected
    float s_max_clamp;           // largest s allowed for the interpolation read
    int32_t pad1;
    double s_magic;              // see kIndexMagic: FP64 sample index exposed in a mantissa (EXACT path)

    // ---- what the launch migrates: one panel, bins, runs or boxed segments ----
    const BinWork *bins;         // nullable: the outputs of the batched form
    const int64_t *runs;         // nullable: n_runs [begin, end) trace ranges
    const SegmentBox *boxes;     // nullable: the scatter schedule's segments
    int64_t seg_traces;
    int64_t n_run_traces;        // traces of all runs
    int32_t n_runs;
    int32_t n_bins;
    int32_t n_splits;            // CTAs of one cluster that share an item's traces
    int32_t max_chunk;           // traces staged per step (<= kChunk)
    int32_t n_pblk_x, n_pblk_y;  // pillar patches
    int32_t n_tblk;              // time blocks
    int32_t n_pblk_fold;         // CTAs that count one output's fold

    // ---- output ----
    void *image;
    int32_t *fold;
    int32_t image_f32;           // 0: f64 image, 1: f32 image
    int32_t fold3d;
    int32_t nx, ny, nt;
    int32_t px, py;              // pillar patch of one CTA (px * py pillars)
    int32_t flush_mask;          // FP32 sums go into FP64 after chunks k with k & mask == mask
    const double *xa, *ya, *xg, *yg, *ta;   // xg/yg nullable

    // ---- velocity ----
    const double *vrms;          // (nt) or (nx*ny*nt)
    int32_t vel3d;
    int32_t eta3d;
    float inv_dt_f;              // 1 / dt (s)
    int32_t exact_units;         // weights' time unit: 1 = samples (EXACT), 0 = seconds
    int32_t curved_kind;         // curved-ray traveltime (its T can be ~0 at t0 > 0)
    int32_t t0_zero_exact;       // at t0 = 0 every pair has T = 0 exactly in FP64 (VTI; curved, k != 0)
    const double *eta;           // nullable
    double eta_const;

    // ---- parameters ----
    double max_ap, min_ap, tan_dip, taper;
    double fold_d2_max;          // largest d^2 with RN(sqrt(d^2)) <= max_ap
    float taper_f;               // taper fraction
    int32_t spreading, obliquity;
    int32_t aa;
    float aa_cA, aa_cB;          // 4*max(dx,dy)*f_dom, f_dom/500
    double aa_gmax, aa_fdom;     // max(dx, dy), f_dom (FP64 paths)
    double cr_v0, cr_k;
    float cr_inv_k_ln2;          // ln2 / k (log2 based)
    int32_t cr_k_zero;           // |k| < 1e-10: straight-ray fallback with v0
    int32_t *err;                // device error word (KernelError bits)
    double cr_B0;                // 1 / (v0 dt)^2: |k| ~ 0 straight rays in v0
    double cr_k2;                // k^2
    double cr_inv_k_dt;          // kTimeScale / (k dt)
    double cr_inv_k_unit;        // the same per kSampleUnit
    int32_t wait_iters;          // polls of one bounded mbarrier wait before it gives up
    int32_t inject_stall;        // fault injection: the first chunks' copies are never issued, so the
                                 // bounded waits for them run out (host-selected, tests only)
};

}  // namespace pstm
