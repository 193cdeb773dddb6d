// migrate.cuh -- gather-form Kirchhoff PSTM kernel for sm_100a.
//
// One CTA owns a patch of 8 output pillars and 64 consecutive output times.
// Consumer warp w (of 8) owns pillar w and its lane l the times l and l + 32,
// whose state (per-time terms, partial sums) stays in registers for the whole
// trace loop.  A ninth warp, the producer, feeds them chunks of up to 32 traces
// through two shared-memory buffers (full/empty mbarriers, bounded waits):
//   producer  runs over the trace midpoints and lists the next traces inside
//             the CTA's largest aperture; bounds each trace's traveltime over
//             the patch and the block, which gives the samples it can
//             contribute; and issues a TMA bulk copy of that window -- not of
//             the whole row.  Geometry and window go into a trace table;
//   consumers turn the table into records of their own pillar (FP64
//             distances, rounded once) in three classes: PLAIN, where every
//             test of the pair loop is known to pass for every lane; MID, where
//             only the aperture's taper and the trace ends are open; and EDGE,
//             the rest.  Then they run the classes' pair loops; every four (or one)
//             chunks their FP32 sums go into FP64.  16-bit samples are first
//             widened to FP32 in shared memory.
// No warp waits for another consumer (except to widen), so uneven chunks and the
// producer's memory latency are hidden; the first form, in which the eight warps
// selected, staged and built in turn between CTA barriers, lost 12 % of its warp
// time at the barrier and spent 520 instructions per warp and chunk outside the
// pair loops, 8 per pair.
// A small output grid splits an item's traces over the 2-8 CTAs of a cluster,
// whose FP64 sums rank 0 adds in rank order through distributed shared memory,
// so results do not depend on scheduling.  The image is added into once, in the
// epilogue.  Further CTAs of the same launch count the fold.
//
// What bounds it: issue.  Dispatch costs of one warp add up (measured, cycles per
// SM sub-partition: FP64 2.1, or 3.4 with three register operands; FP32 1.15,
// packed FP32 2.3; shared-memory reads, MUFU and integer about 1), and a PLAIN
// straight-ray pair with AA is 20 of FP64, 9 of FP32, 5 integer, 3 MUFU, 3 reads and
// 2 moves: 43 cycles, which is what it takes (39 without AA, 54-70 MID), while its
// three MUFU operations occupy that pipe for 24.  Unrolling by 1 to 4, software
// pipelining, scalar instead of packed FP32, and one or three CTAs per SM instead
// of two are all within 8 % of each other or slower.  Records cost 220 cycles a warp
// and chunk.  64 x 64 pillars x 1500 times x 16,384 traces, 3-D velocity, AA: 191 ms
// with whole rows staged and state reloaded from tables per chunk, 120 ms now.
//
// Reference semantics (paths relative to the reference project):
//   loop structure, fold, aperture, taper, weights  numba_cpu_optimized.py:147-231
//   per-time terms                                   numba_cpu_optimized.py:358-401
//   triangle AA weight                               pstm_migration.metal:95-132
//   curved-ray leg                                   pstm_curved_ray.metal:50-96
//   VTI leg                                          pstm_anisotropic_vti.metal:103-148
//
// Precision.  PSTM_PREC_EXACT forms the sample index in FP64 and splits it
// into integer and fraction with bit operations (the fraction cut to
// 2^-23), so the trace-end test is an FP64 decision.  Otherwise traveltime is
// FP32; PSTM_PREC_FAST re-takes trace-end decisions inside a guard band in FP64.
#pragma once
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "kparams.h"
#include "logtab.cuh"
#include "pstm_cuda.h"

namespace pstm {

constexpr int kPillars = 8;                 // pillars per CTA, one consumer warp each
constexpr int kConsumers = 32 * kPillars;
constexpr int kThreads = kConsumers + 32;   // and the producer warp
constexpr int kTimes = 64;                  // output times per CTA, two per lane
constexpr int kChunk = 32;                  // traces per chunk, upper bound: one per lane when records are built
constexpr int kRowPitch = 256;              // staged samples per trace with 32 traces per chunk
constexpr int kPool = kChunk * kRowPitch;   // staged samples of one buffer
constexpr int kMaxSplits = 8;               // CTAs of a cluster that share an item's traces
constexpr int kFlush = 4;                   // chunks whose FP32 sums are added into FP64 together (a power of 2)
constexpr int kFoldPillars = 8;             // pillars per fold-counting CTA
// Default bound of every mbarrier wait loop (KParams::wait_iters), in polls that each may
// block for a while.  A consumer's wait covers the producer's search for the next traces too:
// one of 200 million midpoints, 2.1 s, did not exhaust it.
constexpr int kWaitIters = 1 << 20;

// EXACT path: traveltimes are carried times 2^128, so that a funnel shift turns
// them into floats, and the sample index plus 2^20, times the same scale, has the
// integer index in the high word's low bits and 32 fraction bits in the low word.
constexpr double kTimeScale = 0x1p128;
// The weights take T in units of 256 m or 128 samples, the middle of its range, so that
// 1 / T^2 moves no amplitude far (in metres and samples it is 2^-20 to 2^-28, and
// amplitudes below 2^-100 lost bits to it before the point's factor gave them back).
constexpr double kMetreUnit = 256.0, kSampleUnit = 128.0;
constexpr double kQScale = 0x1p238;         // of squares: (2^128 / 2 / kMetreUnit)^2, the legs double their roots
static_assert(kQScale == (kTimeScale / 2 / kMetreUnit / 0x1p100) * (kTimeScale / 2 / kMetreUnit) * 0x1p100, "");
// 2^20 in the sum, plus 2^-22: an index within 2^-22 below an integer counts as
// that integer (the trace-end decisions are those of an index rounded to 2^-21),
// and the fraction's float takes the 2^-22 off again
constexpr double kIndexMagic = 1048576.0 + 0x1p-22;
constexpr float kFractionBase = 1.f + 0x1p-22f;
constexpr unsigned kHiBase = 0x49300000u;   // high word of 2^20 2^128
constexpr unsigned kFloatBase = 0x4B000000u;   // FP32 paths: 2^23, whose low mantissa bits are the index

// ---------------------------------------------------------------- math helpers
__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// sqrt for q > 0: the hardware's approximate reciprocal square root
// (rsqrt.approx.f64) refined by one Newton step, accurate to ~2^-44.
__device__ __forceinline__ double sqrt_newton(double q) {
    double h;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(h) : "d"(q));
    const double u = q * h;
    const double c = fma(-u, u, q);
    return fma(c, 0.5 * h, u);
}
// 1/x for x > 0: the hardware's approximate reciprocal refined by one Newton step.
__device__ __forceinline__ double rcp_newton(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return fma(r, fma(-x, r, 1.0), r);
}
// 2 sqrt(q) for q > 0 from the same approximation and Newton step, written as
// W (3 - W h), W = q h: three FP64 operations, the factor 2 left to the caller's
// units.
__device__ __forceinline__ double sqrt_newton_x2(double q) {
    double h;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(h) : "d"(q));
    const double w = q * h;
    return w * fma(-w, h, 3.0);
}
// x 2^-128 for x 2^-128 in the float normal range, x >= 0, as a float with the
// mantissa truncated (|error| < 1 float ulp): the low 9 bits of the double's
// exponent field are then the float's, so one funnel shift does it.
__device__ __forceinline__ float scaled_double_to_float(double x) {
    return __uint_as_float(__funnelshift_l((unsigned)__double2loint(x), (unsigned)__double2hiint(x), 3));
}

// The same, rounded to the nearest float: half a unit added to the bits first, two
// more integer instructions (the hardware's conversion takes 9 issue cycles).
__device__ __forceinline__ float scaled_double_to_float_rn(double x) {
    return scaled_double_to_float(__longlong_as_double(__double_as_longlong(x) + (1ll << 28)));
}

template <int AMP>
__device__ __forceinline__ float amp_at(const unsigned char *row, int i) {
    if constexpr (AMP == AMP_F32) {
        return reinterpret_cast<const float *>(row)[i];
    } else if constexpr (AMP == AMP_BF16) {
        return __uint_as_float(((unsigned)reinterpret_cast<const unsigned short *>(row)[i]) << 16);
    } else {
        return __half2float(reinterpret_cast<const __half *>(row)[i]);
    }
}

__device__ __forceinline__ float bf16_to_f32(unsigned short h) { return __uint_as_float((unsigned)h << 16); }

// ---------------------------------------------------------------- TMA bulk copies
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait for the mbarrier phase with the given parity: at most `iters`
// polls (each a potentially blocking try_wait); false = gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int iters) {
    for (int i = 0; i < iters; ++i) {
        uint32_t done;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// ---------------------------------------------------------------- per-point state
// Quantities of one output time.
struct TimeState {
    float t0h2;            // (t0/2)^2
    float tg;              // weights apply only when T > tg ("T > 1 ms"); -1 when always
    float tguard;          // 1 ms in the unit of T's tests
    float vz, vz2, ivwc;   // curved: velocity at image depth, 1/vz
    bool tzero;
    bool tz;               // t0 = 0 with T = 0 exactly for every pair
    double A;              // (t0 / (2 dt))^2 (at least 1e-20)
    double vz64;           // curved kinds: v(z) of the image depth
};

// Quantities of one (pillar, time).
struct PtState {
    float iv2, ap, itw, tsn;
    float K;               // weight numerator
    float ivw_t;           // 1/v_w per unit of T (AA sin theta)
    float aaA;             // 4 max(dx,dy) f_dom / v_w (AA)
    float aa_k;            // aaA / v_w per unit of T
    float aa_thr;          // minf / T above which sin(theta) >= 0.01 (unit of T's tests)
    float thr_s;           // aa_thr per sample
    float t02v2, c1, e2;   // VTI: (t0/2)^2 v^2, 1+2eta, 2 eta / v^2
    float iv2r;            // 1/v_rms^2 (the curved+VTI ratio's hyperbolic leg; iv2 may be 1/v0^2)
    double v, eta;
    double iv, B;          // 1/(v dt), its square
};

// The state of output point (p, t), evaluated in FP64 as
// numba_cpu_optimized.py:378-399 does and rounded once to FP32.  `unit` is the
// weights' unit of the traveltime T, `per` of the base unit.  In metres T is v T, the sum of the legs'
// effective lengths: the spreading is 1 / (v T), the obliquity t0 v / (v T) and
// sin(theta) = minf / (v T) then need nothing of the point but t0 v.
enum TimeUnit { UNIT_SECONDS = 0, UNIT_SAMPLES = 1, UNIT_METRES = 2 };
template <int TT>
__device__ __forceinline__ void point_state(const KParams &P, int p, int t, int unit, double per, TimeState &ts,
                                            PtState &s) {
    const double t0 = P.ta[t] / 1000.0;
    const double v = P.vel3d ? P.vrms[(int64_t)p * P.nt + t] : P.vrms[t];
    double eta = P.eta_const;
    if (P.eta) eta = P.eta3d ? P.eta[(int64_t)p * P.nt + t] : P.eta[t];
    double ap = v * t0 * 0.5 * P.tan_dip;
    if (ap < P.min_ap) ap = P.min_ap;
    else if (ap > P.max_ap) ap = P.max_ap;
    const double rv = 1.0 / v, rvdt = rv * P.inv_dt;   // (divisions are what a small CTA's start waits for)
    s.v = v;
    s.eta = eta;
    s.iv = rvdt;
    // units of T per second (`per` is a power of two)
    const double ips = 1.0 / per, ut = (unit == UNIT_METRES ? v : (unit == UNIT_SAMPLES ? P.inv_dt : 1.0)) * ips;
    // the tests of T keep samples as their unit in metres too
    const double tt = unit == UNIT_SECONDS ? 1.0 : P.inv_dt;
    // straight rays and VTI have T >= t0, so only t0 < 1.1 ms can give T <= 1 ms;
    // the curved-ray leg of the reference tends to 0 at large offsets
    const bool small_t = P.curved_kind || t0 < 0.0011;
    ts.t0h2 = (float)((t0 * 0.5) * (t0 * 0.5));
    ts.tguard = (float)(0.001 * tt);
    ts.tg = small_t ? ts.tguard : -1.f;
    const double th = t0 * 0.5 * P.inv_dt;
    ts.A = fmax(th * th, 1e-20);   // keeps the FP64 legs > 0 at t0 = 0
    ts.tzero = !(t0 > 0.0);
    ts.tz = ts.tzero && P.t0_zero_exact;
    ts.vz = ts.vz2 = ts.ivwc = 0.f;
    ts.vz64 = 0.0;
    double rvw = rv;   // 1/v_w
    s.iv2 = (float)(rv * rv);
    s.iv2r = s.iv2;
    s.B = rvdt * rvdt;
    if constexpr (TT == TT_CURVED || TT == TT_CURVED_VTI) {
        const double z = P.cr_k_zero ? P.cr_v0 * (t0 * 0.5) : (P.cr_v0 / P.cr_k) * (exp(P.cr_k * (t0 * 0.5)) - 1.0);
        ts.vz64 = P.cr_v0 + P.cr_k * z;
        ts.vz = (float)ts.vz64;
        ts.vz2 = (float)(ts.vz64 * ts.vz64);
        rvw = 1.0 / ts.vz64;
        ts.ivwc = (float)rvw;
        if (P.cr_k_zero) s.iv2 = ts.ivwc * ts.ivwc;   // |k| ~ 0: straight rays in v0 (curved_ray.py:35-38)
    }
    s.ap = (float)ap;
    // x = d itw + tsn is 0 or less before the taper and 1 or more beyond the aperture; the MID
    // loop has no other test of the aperture.  Without one only d = 0 is inside (0), or nothing
    // is (below 0).  A hard cut has x = -1 throughout, and tests of its own.
    const float width = s.ap * P.taper_f;
    if (width > 1e-30f) {
        s.itw = rcp_approx(width);
        s.tsn = -(s.ap * (1.f - P.taper_f)) * s.itw;
    } else if (P.taper_f > 0.f) {
        s.itw = 1e30f;
        s.tsn = s.ap < 0.f ? 1.f : 0.f;
    } else {
        s.itw = 0.f;
        s.tsn = -1.f;
    }
    // 1/(v T_sec) = ivw_t / T
    const float ivw = (float)rvw;
    s.ivw_t = (unit == UNIT_METRES ? 1.f : (unit == UNIT_SAMPLES ? ivw * P.inv_dt_f : ivw)) * (float)ips;
    s.aaA = P.aa_cA * ivw;
    s.aa_k = s.aaA * s.ivw_t;
    s.aa_thr = 0.01f * rcp_approx(unit == UNIT_SECONDS ? ivw : ivw * P.inv_dt_f);
    s.thr_s = unit == UNIT_SECONDS ? s.aa_thr * (float)P.dt_s : s.aa_thr;
    // rounded once: an error of 1/v_w would be common to a whole image in a constant velocity
    const double Kt = P.obliquity ? t0 * ut : 1.0;   // the obliquity's numerator
    s.K = (float)(P.spreading ? Kt * ips * (unit == UNIT_METRES ? 1.0 : (unit == UNIT_SAMPLES ? rvw * P.inv_dt : rvw)) : Kt);
    s.t02v2 = 0.f;
    s.c1 = 1.f;
    s.e2 = 0.f;
    if constexpr (TT == TT_VTI || TT == TT_CURVED_VTI) {
        const float ef = (float)eta, iv2 = s.iv2r;
        s.t02v2 = ts.t0h2 * rcp_approx(iv2);   // (t0/2)^2 v^2
        s.c1 = 1.f + 2.f * ef;
        s.e2 = 2.f * ef * iv2;
    }
}

// The FP64 numbers of one point that the EXACT pair loop keeps: C = (t0 v / 2)^2
// (times kQScale, or k^2 for curved+VTI), iv = kMetreUnit / (v dt), c1 = 1 + 2 eta, e2 = 2 eta,
// 2 v(z) and v(z)^2.
struct XState {
    double A, C, iv, c1, e2, vz, vz2;
};
template <int TT, bool KZ>
__device__ __forceinline__ XState exact_state(const KParams &P, const TimeState &ts, const PtState &s) {
    constexpr bool CURVED = TT == TT_CURVED || TT == TT_CURVED_VTI;
    XState x;
    x.A = ts.A;
    const double vdt = s.v * P.dt_s;
    x.C = ts.A * vdt * vdt * (CURVED ? (KZ ? 1.0 : P.cr_k2) : kQScale);
    x.iv = s.iv * kMetreUnit;
    x.c1 = 1.0 + 2.0 * s.eta;
    x.e2 = 2.0 * s.eta;
    x.vz = 2.0 * ts.vz64;
    x.vz2 = ts.vz64 * ts.vz64;
    return x;
}
// The squared distances h^2 of an EXACT record (finite: the producer drops other
// traces): straight and VTI carry them times kQScale, the curved kinds times k^2.
template <int TT, bool KZ>
__device__ __forceinline__ double record_square(const KParams &P, double x) {
    if constexpr (TT == TT_CURVED || TT == TT_CURVED_VTI) return KZ ? x : P.cr_k2 * x;
    // x kQScale by the exponent (x = 0 becomes 2^-785: as good as 0 beside C)
    return __hiloint2double(__double2hiint(x) + (238 << 20), __double2loint(x));
}
// Twice v + sqrt(v^2 + k^2 h^2), the numerator of a curved leg's logarithm.
__device__ __forceinline__ double curved_numerator(const XState &x, double kx) {
    const double q = kx + x.vz2;
    double h;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(h) : "d"(q));
    const double w = q * h;
    return fma(w, fma(-w, h, 3.0), x.vz);
}

// FP64 traveltime (the EXACT path) of one pair from its record: B = {ds2, dr2},
// C = VTI {ds2^2, dr2^2}, curved {1/(4 bs br), 0} or curved+VTI {1/(2 bs), 1/(2 br)},
// bs = v0 + sqrt(v0^2 + k^2 ds2).  Returns T times 2^128 in the weights' unit and puts
// the sample index word into `v`: the sum of 2^20 + index, times 2^128.
// Straight and VTI work in units of kMetreUnit: a leg's effective length is sqrt(C + x) with
// x = h^2, and with the VTI correction sqrt(C + x - 2 eta x^2 / (C + (1+2eta) x)); the
// legs' sum times 1 / (v dt) is the index.  Against squares of times, A + x B,
// this needs an addition instead of a three-operand FMA per leg (2.1 instead of
// 3.4 issue cycles) and no velocity in the weights.
// CLAMP: radicands that odd parameters (eta < -0.15) can push below zero are
// kept above it.
template <int TT, bool KZ, bool CLAMP>
__device__ __forceinline__ double exact_time(const KParams &P, const LogEntry *log_tab, const XState &x, bool tz,
                                             bool tzero, const double2 &B, const double2 &C, double &v) {
    const double magic = P.s_magic;
    if constexpr (TT == TT_STRAIGHT || TT == TT_VTI) {
        double qs = B.x + x.C, qr = B.y + x.C, hs, hr;
        if constexpr (TT == TT_VTI) {
            const double Ds = fma(B.x, x.c1, x.C), Dr = fma(B.y, x.c1, x.C);
            const double rr = rcp_newton(Ds * Dr);
            qs = fma(-(x.e2 * C.x), Dr * rr, qs);
            qr = fma(-(x.e2 * C.y), Ds * rr, qr);
            if constexpr (CLAMP) {
                qs = fmax(qs, 0x1p80);
                qr = fmax(qr, 0x1p80);
            }
        }
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(hs) : "d"(qs));
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(hr) : "d"(qr));
        const double ws = qs * hs, wr = qr * hr;
        double T = fma(ws, fma(-ws, hs, 3.0), wr * fma(-wr, hr, 3.0));
        if constexpr (TT == TT_VTI && CLAMP) T = tz ? 0.0 : T;   // the reference's VTI leg is 0 at t0 = 0
        v = fma(T, x.iv, magic);
        return T;
    } else if constexpr (TT == TT_CURVED) {   // |k| ~ 0: straight rays in v0 (curved_ray.py:35-38)
        if constexpr (KZ) {
            const double T = sqrt_newton(fma(B.x, P.cr_B0, x.A)) + sqrt_newton(fma(B.y, P.cr_B0, x.A));
            v = fma(T, kTimeScale, magic);
            return T * (kTimeScale / kSampleUnit);
        } else {
            double L = log_by_table(log_tab, curved_numerator(x, B.x) * curved_numerator(x, B.y) * C.x);
            if constexpr (CLAMP) L = tz ? 0.0 : L;   // depth 0: both legs are log(1) = 0
            v = fma(L, P.cr_inv_k_dt, magic);
            return L * P.cr_inv_k_unit;
        }
    } else {
        double tcs, tcr;
        if constexpr (KZ) {
            tcs = sqrt_newton(fma(B.x, P.cr_B0, x.A));
            tcr = sqrt_newton(fma(B.y, P.cr_B0, x.A));
        } else {
            tcs = log_by_table(log_tab, curved_numerator(x, B.x) * C.x);
            tcr = log_by_table(log_tab, curved_numerator(x, B.y) * C.y);
        }
        // leg = t_curved sqrt(1 - f), f = 2 eta x^2 / ((C + (1+2eta) x)(C + x)), x and C times k^2
        const double Hs = B.x + x.C, Hr = B.y + x.C;
        const double Ds = fma(B.x, x.c1, x.C), Dr = fma(B.y, x.c1, x.C);
        const double ps = Ds * Hs, pr = Dr * Hr;
        const double rr = rcp_newton(ps * pr);
        double us = fma(-(x.e2 * B.x * B.x), pr * rr, 1.0), ur = fma(-(x.e2 * B.y * B.y), ps * rr, 1.0);
        if constexpr (CLAMP) {
            us = fmax(us, 1e-40);
            ur = fmax(ur, 1e-40);
        }
        double L = fma(tcs, sqrt_newton(us), tcr * sqrt_newton(ur));
        if constexpr (CLAMP || KZ)   // t0 = 0: nothing, or (|k| ~ 0, where no point is odd) the curved legs alone
            L = tzero ? (tz ? 0.0 : tcs + tcr) : L;
        v = fma(L, KZ ? kTimeScale : P.cr_inv_k_dt, magic);
        return L * (KZ ? kTimeScale / kSampleUnit : P.cr_inv_k_unit);
    }
}

// 0.5 (1 + cos(pi x)) = cos^2(pi x / 2) for x in [0, 1]: cos as a polynomial in x^2
// with value 1 at 0 and the least largest error on [0, 1] (2.4e-10, fitted by
// reweighted least squares), then squared; 1.3e-7 in FP32, all of it rounding.
// Taylor's series takes two more terms for 7e-9.
constexpr float kTaper1 = -1.2337005390219158f, kTaper2 = 0.25366934998483653f, kTaper3 = -0.020862751638218144f,
                kTaper4 = 9.17788771589905e-4f, kTaper5 = -2.3848339607722318e-5f;
__device__ __forceinline__ float taper_weight(float x) {
    const float u = x * x;
    float c = kTaper5;
    c = fmaf(c, u, kTaper4);
    c = fmaf(c, u, kTaper3);
    c = fmaf(c, u, kTaper2);
    c = fmaf(c, u, kTaper1);
    c = fmaf(c, u, 1.0f);
    return c * c;
}
// The same for two x in [0, 1], in packed FP32 pairs.
__device__ __forceinline__ float2 taper_weight2(float2 x) {
    auto two = [](float a) { return make_float2(a, a); };
    const float2 u = __fmul2_rn(x, x);
    float2 c = __ffma2_rn(two(kTaper5), u, two(kTaper4));
    c = __ffma2_rn(c, u, two(kTaper3));
    c = __ffma2_rn(c, u, two(kTaper2));
    c = __ffma2_rn(c, u, two(kTaper1));
    c = __ffma2_rn(c, u, two(1.0f));
    return __fmul2_rn(c, c);
}

// ---------------------------------------------------------------- FP64 exact decisions
// (rare paths: they read the launch parameters from a global copy, so the
// kernel's own parameter block never has its address taken)
// FP64 traveltime of one pair from its raw quantities: output time t0 (s),
// squared horizontal source and receiver distances, v_rms, eta and the
// curved-ray (v0, k).  The oracle's formulas; also the surrogate's target.
template <int TT>
__host__ __device__ inline double traveltime_fp64(double t0, double ds2, double dr2, double v, double eta, double v0,
                                                  double k) {
    const double t0h = t0 * 0.5;
    auto vti_corr = [&](double h2) {
        const double v2 = v * v;
        const double den = v2 * (t0h * t0h * v2 + (1.0 + 2.0 * eta) * h2);
        return fabs(den) > 1e-20 ? (2.0 * eta * h2 * h2) / den : 0.0;
    };
    auto curved_leg = [&](double h2) {
        if (fabs(k) < 1e-10) {
            const double z = v0 * t0h;
            const double r = sqrt(h2 + z * z);
            return r > 0.0 ? r / v0 : 0.0;
        }
        const double z = (v0 / k) * (exp(k * t0h) - 1.0);
        const double vz = v0 + k * z;
        const double kx2 = k * k * h2;
        const double a = vz + sqrt(vz * vz + kx2), b = v0 + sqrt(v0 * v0 + kx2);
        return b <= 0.0 ? 0.0 : (1.0 / k) * log(a / b);
    };
    if constexpr (TT == TT_STRAIGHT) {
        const double iv2 = 1.0 / (v * v);
        return sqrt(t0h * t0h + ds2 * iv2) + sqrt(t0h * t0h + dr2 * iv2);
    } else if constexpr (TT == TT_CURVED) {
        return curved_leg(ds2) + curved_leg(dr2);
    } else if constexpr (TT == TT_VTI) {
        if (v <= 0.0 || t0h <= 0.0) return 2.0 * t0h;
        auto leg = [&](double h2) {
            const double q = t0h * t0h + h2 / (v * v) - vti_corr(h2);
            return sqrt(q > 0.0 ? q : 0.0);
        };
        return leg(ds2) + leg(dr2);
    } else {
        auto leg = [&](double h2) {
            const double tc = curved_leg(h2);
            if (v <= 0.0 || t0h <= 0.0) return tc;
            const double r = 1.0 - vti_corr(h2) / (t0h * t0h + h2 / (v * v));
            return tc * sqrt(r > 0.0 ? r : 0.0);
        };
        return leg(ds2) + leg(dr2);
    }
}

template <int TT>
__device__ double exact_traveltime(const KParams *P, int64_t tr, int p, int t, double ox, double oy) {
    const double t0 = P->ta[t] / 1000.0;
    const double v = P->vel3d ? P->vrms[(int64_t)p * P->nt + t] : P->vrms[t];
    const double dxs = ox - P->sx[tr], dys = oy - P->sy[tr];
    const double dxr = ox - P->rx[tr], dyr = oy - P->ry[tr];
    double eta = P->eta_const;
    if (P->eta) eta = P->eta3d ? P->eta[(int64_t)p * P->nt + t] : P->eta[t];
    return traveltime_fp64<TT>(t0, dxs * dxs + dys * dys, dxr * dxr + dyr * dyr, v, eta, P->cr_v0, P->cr_k);
}

// Is the FP64 sample index of this pair inside [0, ns-1)?
template <int TT>
__device__ __noinline__ bool exact_sample_ok(const KParams *P, int64_t tr, int p, int t, double ox, double oy) {
    const double T = exact_traveltime<TT>(P, tr, p, t, ox, oy);
    const double s = (T - P->tstart_s) / P->dt_s;
    return s >= 0.0 && s < (double)(P->ns - 1);
}

// Is the midpoint outside the time-varying aperture, decided in FP64?
static __device__ __noinline__ bool exact_outside_aperture(const KParams *P, int64_t tr, int p, int t, double ox,
                                                           double oy) {
    const double dx = ox - P->mx[tr], dy = oy - P->my[tr];
    const double d = sqrt(dx * dx + dy * dy);
    const double v = P->vel3d ? P->vrms[(int64_t)p * P->nt + t] : P->vrms[t];
    double ap = v * (P->ta[t] / 1000.0) * 0.5 * P->tan_dip;
    if (ap < P->min_ap) ap = P->min_ap;
    else if (ap > P->max_ap) ap = P->max_ap;
    return d > ap;
}

// ---------------------------------------------------------------- traveltime (FP32)
// B = {ds2, dr2, k^2 ds2 | ds2^2, k^2 dr2 | dr2^2}; C (curved kinds) =
// {1/(bs br) | 1/bs, 1/br, ds2^2, dr2^2}.  Result in seconds.
// KZ: |k| < 1e-10, straight rays in v0 for the curved leg.  TESTS: points at t0 = 0
// are possible (the EDGE loop); without it no lane branches.
template <int TT, bool KZ, bool TESTS>
__device__ __forceinline__ float traveltime(const KParams &P, const TimeState &ts, const PtState &s,
                                            const float4 &B, const float4 &Cc) {
    if constexpr (TT == TT_STRAIGHT || (TT == TT_CURVED && KZ)) {
        return sqrt_approx(fmaf(B.x, s.iv2, ts.t0h2)) + sqrt_approx(fmaf(B.y, s.iv2, ts.t0h2));
    } else if constexpr (TT == TT_CURVED) {
        const float a = ts.vz + sqrt_approx(ts.vz2 + B.z);
        const float b = ts.vz + sqrt_approx(ts.vz2 + B.w);
        return P.cr_inv_k_ln2 * lg2_approx(a * b * Cc.x);
    } else if constexpr (TT == TT_VTI) {
        const float Ds = fmaf(s.c1, B.x, s.t02v2);
        const float Dr = fmaf(s.c1, B.y, s.t02v2);
        const float rr = rcp_approx(Ds * Dr);
        const float qs = fmaf(-(s.e2 * B.z), Dr * rr, fmaf(B.x, s.iv2, ts.t0h2));
        const float qr = fmaf(-(s.e2 * B.w), Ds * rr, fmaf(B.y, s.iv2, ts.t0h2));
        const float T = sqrt_approx(fmaxf(qs, 0.f)) + sqrt_approx(fmaxf(qr, 0.f));
        return TESTS && ts.tzero ? 0.f : T;
    } else {
        float tcs, tcr;
        if constexpr (KZ) {
            tcs = sqrt_approx(fmaf(B.x, s.iv2, ts.t0h2));
            tcr = sqrt_approx(fmaf(B.y, s.iv2, ts.t0h2));
        } else {
            const float a = ts.vz + sqrt_approx(ts.vz2 + B.z);
            const float b = ts.vz + sqrt_approx(ts.vz2 + B.w);
            tcs = P.cr_inv_k_ln2 * lg2_approx(a * Cc.x);
            tcr = P.cr_inv_k_ln2 * lg2_approx(b * Cc.y);
        }
        // leg = t_curved * sqrt(1 - corr / (t0h^2 + h^2/v^2)), corr = e2 h^4 / D, v = v_rms
        const float Hs = fmaf(B.x, s.iv2r, ts.t0h2), Hr = fmaf(B.y, s.iv2r, ts.t0h2);
        const float Ds = fmaf(s.c1, B.x, s.t02v2), Dr = fmaf(s.c1, B.y, s.t02v2);
        const float ps_ = Ds * Hs, pr_ = Dr * Hr;
        const float rr = rcp_approx(ps_ * pr_);
        const float xs = s.e2 * Cc.z * (pr_ * rr), xr = s.e2 * Cc.w * (ps_ * rr);
        const float T = tcs * sqrt_approx(fmaxf(1.f - xs, 0.f)) + tcr * sqrt_approx(fmaxf(1.f - xr, 0.f));
        return TESTS && ts.tzero ? tcs + tcr : T;
    }
}

// ---------------------------------------------------------------- sample ranges
// Ranges of the per-time numbers over one half (32 times) of a CTA's block, in
// samples; they bound the traveltime of a trace at those times.
struct HalfBounds {
    float A0, A1, B0, B1, e0, e1, vz0, vz1;
};

// Bounds of the traveltime (in samples) of one trace over a half's times and the
// patch, from the bounds [x0, x1] of its squared distances.  Each leg is monotone
// in every one of its numbers, so the corners of their ranges bound it:
//   straight   sqrt(A + x B), rising in A and B;
//   VTI        q = A + y - 2 eta y^2 / (A + (1+2eta) y), y = x B: rising in A and y
//              (dq/dy >= 1/(1+2eta)), falling in eta, for eta >= -0.15;
//   curved     (1/k) ln[(v + sqrt(v^2 + k^2 x)) / (v0 + sqrt(v0^2 + k^2 x))]: monotone in
//              v = v(z) and in x, either way round (|k| ~ 0: straight rays in v0);
//   curved+VTI the curved leg times sqrt(1 - f), f = 2 eta y^2 / ((A + (1+2eta) y)(A + y)),
//              which rises with eta, and with y/A when eta > 0 (falls when eta < 0).
// FP32: the caller's margin covers the rounding.
template <int TT>
__device__ __forceinline__ void leg_bounds(const KParams &P, const HalfBounds &h, float x0, float x1, float &l,
                                           float &u) {
    [[maybe_unused]] auto curved = [&](float x, float A, float vz) {
        if (P.cr_k_zero) return sqrt_approx(fmaf(x, (float)P.cr_B0, A));
        const float kx = (float)P.cr_k2 * x, v0 = (float)P.cr_v0;
        const float b = v0 + sqrt_approx(fmaf(v0, v0, kx));
        return P.cr_inv_k_ln2 * P.inv_dt_f * lg2_approx((vz + sqrt_approx(fmaf(vz, vz, kx))) * rcp_approx(b));
    };
    const float y0 = x0 * h.B0, y1 = x1 * h.B1;
    if constexpr (TT == TT_STRAIGHT) {
        l = sqrt_approx(h.A0 + y0);
        u = sqrt_approx(h.A1 + y1);
    } else if constexpr (TT == TT_VTI) {
        const float c0 = 1.f + 2.f * h.e0, c1 = 1.f + 2.f * h.e1;
        const float ql = h.A0 + y0 - 2.f * h.e1 * y0 * y0 * rcp_approx(fmaxf(h.A0 + c1 * y0, 1e-30f));
        const float qu = h.A1 + y1 - 2.f * h.e0 * y1 * y1 * rcp_approx(fmaxf(h.A1 + c0 * y1, 1e-30f));
        l = sqrt_approx(fmaxf(ql, 0.f));
        u = sqrt_approx(fmaxf(qu, 0.f));
    } else {
        l = fminf(fminf(curved(x0, h.A0, h.vz0), curved(x1, h.A0, h.vz0)),
                  fminf(curved(x0, h.A0, h.vz1), curved(x1, h.A0, h.vz1)));
        u = fmaxf(fmaxf(curved(x0, h.A1, h.vz0), curved(x1, h.A1, h.vz0)),
                  fmaxf(curved(x0, h.A1, h.vz1), curved(x1, h.A1, h.vz1)));
        l = fmaxf(l, 0.f);
        if constexpr (TT == TT_CURVED_VTI) {
            auto f = [&](float eta, float y, float A) {
                const float d = fmaxf(A + (1.f + 2.f * eta) * y, 1e-18f) * fmaxf(A + y, 1e-18f);
                return 2.f * eta * y * y * rcp_approx(d);
            };
            const float f1 = h.e1 >= 0.f ? f(h.e1, y1, h.A0) : f(h.e1, y0, h.A1);
            const float f0 = h.e0 >= 0.f ? f(h.e0, y0, h.A1) : f(h.e0, y1, h.A0);
            l *= sqrt_approx(fmaxf(1.f - fmaxf(f1, 0.f), 0.f));   // f = 0 where t0 = 0
            u *= sqrt_approx(fmaxf(1.f - fminf(f0, 0.f), 0.f));
        }
    }
}

// ---------------------------------------------------------------- shared memory
// Records of one warp, in arrays: distances (16 bytes), {m, w, row, d} (16),
// {first index, indices | trace << 24} (8) and, but for straight rays, C (16).
__host__ __device__ constexpr int record_bytes(bool has_c) { return kChunk * (has_c ? 56 : 40); }
// Dynamic shared memory of one CTA: staged samples (two FP32 buffers, or two
// 16-bit ones and their FP32 widening: the same bytes), a record buffer per
// warp, and per point the terms of the MID and EDGE loops and the FP64 sum.
__host__ __device__ constexpr int dynamic_bytes(bool has_c) {
    return 2 * kPool * 4 + kPillars * record_bytes(has_c) + 2 * kConsumers * 32;
}

// The producer's account of a chunk.
// DROP: adds nothing; SURE: every traveltime is known to exceed 1 ms and the weight
// is finite; INSIDE: every sample index is known to lie inside the trace.
enum TraceFlags { TRACE_DROP = 1, TRACE_SURE = 2, TRACE_INSIDE = 4 };
struct TraceTable {
    double sx[kChunk], sy[kChunk], rx[kChunk], ry[kChunk], mx[kChunk], my[kChunk], w[kChunk];
    long long id[kChunk];
    int4 row[kChunk];      // address sample indices are added to, first index, indices | lane << 24, TraceFlags
    int2 window[kChunk];   // first staged sample, staged samples
    float t_hi[kChunk];    // upper bound of the traveltime, samples
    int cnt;
    int wide;              // a window does not fit its row: read the chunk from global memory
};

struct CtaShared {
    unsigned long long full[2], empty[2];
    TraceTable tab[2];
    HalfBounds half[kPillars][2];
    struct {
        double ox, oy;
        float apw, ap_in, thr;
        int even;          // no point with T = 0, or with numbers that the bounds do not cover
    } warp[kPillars];
    float apmax[kPillars], t_lo, t_hi;
    float zero[2];
    long long selected[kChunk];   // the producer's own list
};

// ---------------------------------------------------------------- fold
// image fold += traces within the maximum aperture of each of kFoldPillars
// pillars, decided in FP64 (numba_cpu_optimized.py:166-172).
static __device__ __noinline__ void count_fold(const KParams &P, int pblk, int64_t trace0, int64_t n_traces,
                                               int32_t *fold) {
    __shared__ int s_cnt[kFoldPillars];
    const int n_p = P.nx * P.ny, p0 = pblk * kFoldPillars;
    double ox[kFoldPillars], oy[kFoldPillars];
    int cnt[kFoldPillars];
#pragma unroll
    for (int q = 0; q < kFoldPillars; ++q) {
        const int p = min(p0 + q, n_p - 1);
        ox[q] = P.xg ? P.xg[p] : P.xa[p / P.ny];
        oy[q] = P.yg ? P.yg[p] : P.ya[p % P.ny];
        cnt[q] = 0;
    }
    if (threadIdx.x < kFoldPillars) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    auto range = [&](int64_t a, int64_t b) {
#pragma unroll 2
        for (int64_t i = a + threadIdx.x; i < b; i += kThreads) {
            const double mx = P.mx[i], my = P.my[i];
#pragma unroll
            for (int q = 0; q < kFoldPillars; ++q) {
                const double dxm = ox[q] - mx, dym = oy[q] - my;
                const double d2 = dxm * dxm + dym * dym;
                cnt[q] += d2 <= P.fold_d2_max;
            }
        }
    };
    if (P.runs)
        for (int r = 0; r < P.n_runs; ++r) range(P.runs[2 * r], P.runs[2 * r + 1]);
    else
        range(trace0, trace0 + n_traces);
#pragma unroll
    for (int q = 0; q < kFoldPillars; ++q) {
        const int c = __reduce_add_sync(0xffffffffu, cnt[q]);
        if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_cnt[q], c);
    }
    __syncthreads();
    if (!P.fold3d) {
        if (threadIdx.x < kFoldPillars && p0 + (int)threadIdx.x < n_p) fold[p0 + threadIdx.x] += s_cnt[threadIdx.x];
        return;
    }
    for (int q = 0; q < kFoldPillars && p0 + q < n_p; ++q) {
        const int c = s_cnt[q];
        if (c == 0) continue;
        int32_t *f = fold + (int64_t)(p0 + q) * P.nt;
        for (int t = threadIdx.x; t < P.nt; t += kThreads) f[t] += c;
    }
}

// Barriers of the consumer warps alone (named barrier 1).
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory"); }
__device__ __forceinline__ bool consumers_or(bool x) {
    unsigned r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n"
                 " selp.u32 %0, 1, 0, q;\n}" : "=r"(r) : "r"((unsigned)x), "n"(kConsumers) : "memory");
    return r != 0;
}
__device__ __forceinline__ float lds_f32(uint32_t addr) {
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
// Amplitude i of a trace row in global memory.
__device__ __forceinline__ float amp_global(const KParams &P, long long id, int i) {
    const int64_t e = id * P.amp_stride + i;
    if (P.amp_kind == AMP_F32) return static_cast<const float *>(P.amps)[e];
    if (P.amp_kind == AMP_BF16)
        return bf16_to_f32(static_cast<const unsigned short *>(P.amps)[e]);
    return __half2float(static_cast<const __half *>(P.amps)[e]);
}

// ---------------------------------------------------------------- the kernel
// W2: spreading and obliquity both on (the common case), else the weight
// exponent is chosen at run time.  AA: the triangle antialiasing weight.
// KZ: curved kinds with |k| < 1e-10 (straight rays in v0).
template <int TT, int PREC, bool W2, bool AA, bool KZ>
__global__ void __launch_bounds__(kThreads, 2) gather_kernel(const __grid_constant__ KParams P) {
    namespace cg = cooperative_groups;
    constexpr bool EXACT = PREC == PSTM_PREC_EXACT;
    constexpr bool GUARD = PREC == PSTM_PREC_FAST;
    constexpr bool CURVED = TT == TT_CURVED || TT == TT_CURVED_VTI;
    constexpr bool HAS_C = TT != TT_STRAIGHT;
    constexpr int UNIT = !EXACT ? UNIT_SECONDS : (CURVED ? UNIT_SAMPLES : UNIT_METRES);
    constexpr double UNIT_PER = !EXACT ? 1.0 : (CURVED ? kSampleUnit : kMetreUnit);
    constexpr unsigned INDEX_BASE = EXACT ? kHiBase : kFloatBase;
    constexpr bool LOG = CURVED && EXACT && !KZ;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ CtaShared sh;
    __shared__ LogEntry log_tab[LOG ? kLogEntries : 1];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool producer = warp == kPillars;
    const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;

    // ---------------- the CTA's item: output, time block, pillar patch, traces
    const int splits = P.n_splits;
    const int64_t per_out = (int64_t)P.n_pblk_x * P.n_pblk_y * P.n_tblk;
    const int64_t n_items = P.bins ? per_out * P.n_bins : per_out;
    int64_t item = blockIdx.x / splits;
    const int rank = (int)(blockIdx.x - item * splits);
    void *image = P.image;
    int64_t trace0 = 0, n_traces = P.runs ? P.n_run_traces : P.n_traces;
    int shares = splits;   // ranks among which the item's traces are divided
    if (item >= n_items) {   // the fold-counting CTAs behind the items
        const int64_t k = (int64_t)blockIdx.x - n_items * splits;
        const int64_t out = k / P.n_pblk_fold;
        int32_t *fold = P.fold;
        if (P.bins) {
            if (out >= P.n_bins) return;
            trace0 = P.bins[out].trace0;
            n_traces = P.bins[out].n_traces;
            fold = P.bins[out].fold;
        } else if (out >= 1) {
            return;
        }
        if (fold) count_fold(P, (int)(k - out * P.n_pblk_fold), trace0, n_traces, fold);
        return;
    }
    if (P.bins) {
        const int64_t b = item / per_out;
        item -= b * per_out;
        trace0 = P.bins[b].trace0;
        n_traces = P.bins[b].n_traces;
        image = P.bins[b].image;
        shares = P.bins[b].shares;
        // a rank that a smaller bin has no use for leaves its slot at once (the
        // cluster's barriers wait for the threads that have not exited)
        if (rank >= shares) return;
    }
    // deep blocks first: their aperture is the widest; neighbours in y next to
    // each other, so that the CTAs that run together stage the same samples
    const int n_pblk = P.n_pblk_x * P.n_pblk_y;
    const int tblk = P.n_tblk - 1 - (int)(item / n_pblk);
    const int pblk = (int)(item % n_pblk);
    const int pbx = pblk / P.n_pblk_y, pby = pblk - pbx * P.n_pblk_y;

    const bool wide_type = P.elem == 4;
    unsigned char *const rec = smem + 2 * kPool * 4 + (producer ? 0 : warp) * record_bytes(HAS_C);
    float4 *const edge_a = reinterpret_cast<float4 *>(smem + 2 * kPool * 4 + kPillars * record_bytes(HAS_C));
    float2 *const edge_k = reinterpret_cast<float2 *>(edge_a + 2 * kConsumers);   // {K, tg}
    double *const sums = reinterpret_cast<double *>(edge_k + 2 * kConsumers);     // all [2][kConsumers]
    const uint32_t full0 = smem_u32(&sh.full[0]), full1 = smem_u32(&sh.full[1]);
    const uint32_t empty0 = smem_u32(&sh.empty[0]), empty1 = smem_u32(&sh.empty[1]);
    if (LOG && tid < kLogEntries) log_tab[tid] = log_entry(tid);
    if (tid == kConsumers) {
        mbar_init(full0, 1);
        mbar_init(full1, 1);
        mbar_init(empty0, kPillars);
        mbar_init(empty1, kPillars);
        fence_barrier_init();
        sh.zero[0] = sh.zero[1] = 0.f;
    }

    // ---------------- per-point state
    const int ix = pbx * P.px + warp / P.py, iy = pby * P.py + warp % P.py;
    const bool has_pillar = !producer && warp < P.px * P.py && ix < P.nx && iy < P.ny;
    const int p = has_pillar ? ix * P.ny + iy : 0;
    const double ox = P.xg ? P.xg[p] : P.xa[has_pillar ? ix : 0];
    const double oy = P.yg ? P.yg[p] : P.ya[has_pillar ? iy : 0];
    const bool hard_cut = !(P.taper_f > 0.f);
    const bool w_one = P.spreading + P.obliquity == 1, w_two = P.spreading + P.obliquity == 2;

    TimeState ts[2];
    PtState st[2];
    XState xs[2];
    float apw = -1.f;        // largest aperture of the warp's points
    float ap_in = INFINITY;  // distances below it are inside every point's aperture and taper
    float thr_w = 0.f;       // AA: minf / T(samples) above it everywhere
    bool odd = false;        // a point with T = 0
    bool unbounded = false;  // numbers that the bounds do not cover
    unsigned tz_lanes0 = 0u, tz_lanes1 = 0u;
    if (!producer) {
        float t_lo = INFINITY, t_hi = -INFINITY;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const int t = tblk * kTimes + 32 * g + lane;
            const bool valid = t < P.nt;
            point_state<TT>(P, p, valid ? t : P.nt - 1, UNIT, UNIT_PER, ts[g], st[g]);
            if (EXACT) xs[g] = exact_state<TT, KZ>(P, ts[g], st[g]);
            const float A = (float)ts[g].A, B = (float)st[g].B, e = (float)st[g].eta, vz = ts[g].vz;
            bool fine = A < 1e30f && B > 0.f && B < 1e30f && st[g].iv > 0.0;   // (also not NaN)
            if (TT == TT_VTI || TT == TT_CURVED_VTI) fine = fine && e >= -0.15f && e < 1e3f;
            if (CURVED) fine = fine && vz > 0.f && vz < 1e15f;
            if (valid) {
                unbounded |= !fine;
                odd |= ts[g].tz;
                ap_in = fminf(ap_in, st[g].ap * (1.f - P.taper_f));
                const float th = (float)(P.ta[t] * (0.001 * P.inv_dt));
                t_lo = fminf(t_lo, th);
                t_hi = fmaxf(t_hi, th);
                apw = fmaxf(apw, st[g].ap);
            }
            const bool live = valid && !ts[g].tz;
            // a point past the tile's end, or with T = 0 (summed apart), takes no part in the EDGE
            // loop: its aperture is stored below zero
            edge_a[g * kConsumers + tid] = make_float4(live ? st[g].ap : -1.f - st[g].ap, st[g].itw, st[g].tsn, st[g].aa_thr);
            edge_k[g * kConsumers + tid] = make_float2(st[g].K, ts[g].tg);
            sums[g * kConsumers + tid] = 0.0;
            if (live) thr_w = fmaxf(thr_w, st[g].thr_s);
            HalfBounds h;
            auto lo_of = [&](float x) { return __int_as_float(__reduce_min_sync(full, __float_as_int(x))); };
            auto hi_of = [&](float x) { return __int_as_float(__reduce_max_sync(full, __float_as_int(x))); };
            h.A0 = lo_of(live ? A : INFINITY);   // all of these are >= 0: their bits order them
            h.A1 = hi_of(live ? A : 0.f);
            h.B0 = lo_of(live ? B : INFINITY);
            h.B1 = hi_of(live ? B : 0.f);
            h.vz0 = lo_of(live ? vz : INFINITY);
            h.vz1 = hi_of(live ? vz : 0.f);
            h.e0 = lo_of(live ? e + 1.f : INFINITY);   // eta + 1 > 0
            h.e1 = hi_of(live ? e + 1.f : 0.f);
            if (!has_pillar) h.A0 = INFINITY;   // no live point
            if (lane == 0) sh.half[warp][g] = h;
            const unsigned z = __ballot_sync(full, ts[g].tz && valid);
            if (g == 0) tz_lanes0 = z;
            else tz_lanes1 = z;
        }
        apw = __int_as_float(__reduce_max_sync(full, __float_as_int(apw)));
        ap_in = __int_as_float(__reduce_min_sync(full, __float_as_int(ap_in)));
        thr_w = __int_as_float(__reduce_max_sync(full, __float_as_int(thr_w)));
        odd = __any_sync(full, odd);
        unbounded = __any_sync(full, unbounded);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            t_lo = fminf(t_lo, __shfl_xor_sync(full, t_lo, o));
            t_hi = fmaxf(t_hi, __shfl_xor_sync(full, t_hi, o));
        }
        if (lane == 0) {
            sh.warp[warp] = {ox, oy, apw, ap_in, thr_w, !odd && !unbounded};
            sh.apmax[warp] = has_pillar ? fmaxf(apw, 0.f) : 0.f;
            if (warp == 0) {
                sh.t_lo = t_lo;
                sh.t_hi = t_hi;
            }
        }
    }
    const bool any_unbounded = __syncthreads_or(has_pillar && unbounded);
    // traces per chunk: rows must hold the block's span of times plus the moveout
    // across the patch and the change of velocity over the block
    int C, pitch;
    {
        const float span = sh.t_hi - sh.t_lo;
        float need = any_unbounded ? (float)P.ns : span + fmaxf(96.f, 0.5f * span);
        need = fminf(need, (float)P.ns) + 24.f;
        C = max((int)fminf((float)kPool / need, (float)P.max_chunk), 1);
        pitch = kPool / C & ~7;
    }
    const int per16 = 16 / P.elem;
    bool timeout = false;

    if (producer) {
        // ------------------------------------------------------------ producer
        double x0 = INFINITY, x1 = -INFINITY, y0 = INFINITY, y1 = -INFINITY;   // the patch's box
        float apmax = 0.f;
        HalfBounds hb[2];
        if (lane < P.px * P.py) {
            const int jx = pbx * P.px + lane / P.py, jy = pby * P.py + lane % P.py;
            if (jx < P.nx && jy < P.ny) {
                x0 = x1 = P.xg ? P.xg[jx * P.ny + jy] : P.xa[jx];
                y0 = y1 = P.yg ? P.yg[jx * P.ny + jy] : P.ya[jy];
                apmax = sh.apmax[lane];
            }
        }
#pragma unroll
        for (int o = kPillars / 2; o > 0; o >>= 1) {
            x0 = fmin(x0, __shfl_xor_sync(full, x0, o));
            x1 = fmax(x1, __shfl_xor_sync(full, x1, o));
            y0 = fmin(y0, __shfl_xor_sync(full, y0, o));
            y1 = fmax(y1, __shfl_xor_sync(full, y1, o));
            apmax = fmaxf(apmax, __shfl_xor_sync(full, apmax, o));
        }
        x0 = __shfl_sync(full, x0, 0);
        x1 = __shfl_sync(full, x1, 0);
        y0 = __shfl_sync(full, y0, 0);
        y1 = __shfl_sync(full, y1, 0);
        apmax = fminf(__shfl_sync(full, apmax, 0), (float)P.max_ap);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            hb[g] = {INFINITY, 0.f, INFINITY, 0.f, INFINITY, 0.f, INFINITY, 0.f};
            for (int q = 0; q < kPillars; ++q) {
                const HalfBounds h = sh.half[q][g];
                if (h.A0 == INFINITY) continue;
                hb[g].A0 = fminf(hb[g].A0, h.A0);
                hb[g].A1 = fmaxf(hb[g].A1, h.A1);
                hb[g].B0 = fminf(hb[g].B0, h.B0);
                hb[g].B1 = fmaxf(hb[g].B1, h.B1);
                hb[g].vz0 = fminf(hb[g].vz0, h.vz0);
                hb[g].vz1 = fmaxf(hb[g].vz1, h.vz1);
                hb[g].e0 = fminf(hb[g].e0, h.e0);
                hb[g].e1 = fmaxf(hb[g].e1, h.e1);
            }
            hb[g].e0 -= 1.f;
            hb[g].e1 -= 1.f;
        }
        // A trace outside this radius of the pillars' box is outside every aperture.
        const double reach = (double)apmax * (1.0 + 1e-6) + 1e-3;
        const double reach2 = reach * reach;
        // this rank's share of the traces, in whole chunks
        const long long per = ((n_traces + shares - 1) / shares + kChunk - 1) / kChunk * kChunk;
        const long long v0 = min((long long)n_traces, rank * per), v1 = min((long long)n_traces, v0 + per);
        long long pos, end, left = 0;   // next trace, end of its range, (runs) traces of later ranges
        const long long stop = trace0 + v1;
        int run = 0;
        if (P.runs) {
            long long skip = v0;
            while (run < P.n_runs && skip >= P.runs[2 * run + 1] - P.runs[2 * run]) {
                skip -= P.runs[2 * run + 1] - P.runs[2 * run];
                ++run;
            }
            left = v1 - v0;
            pos = end = 0;
            if (run < P.n_runs && left > 0) {
                pos = P.runs[2 * run] + skip;
                end = min((long long)P.runs[2 * run + 1], pos + left);
                left -= end - pos;
            }
        } else {
            pos = trace0 + v0;
            end = P.boxes ? pos : stop;
        }
        auto next_range = [&]() -> bool {
            if (P.runs) {
                if (left <= 0 || run + 1 >= P.n_runs) return false;
                ++run;
                pos = P.runs[2 * run];
                end = min((long long)P.runs[2 * run + 1], pos + left);
                left -= end - pos;
                return true;
            }
            if (P.boxes) {   // the next segment whose box holds this patch, 32 boxes at a time
                while (pos < stop) {
                    const long long s0 = pos / P.seg_traces, s = s0 + lane;
                    bool hit = false;
                    if (s * P.seg_traces < stop) {
                        const SegmentBox b = P.boxes[s];
                        hit = pbx >= b.pbx0 && pbx <= b.pbx1 && pby >= b.pby0 && pby <= b.pby1;
                    }
                    const unsigned m = __ballot_sync(full, hit);
                    if (m) {
                        const long long f = s0 + __ffs(m) - 1;
                        pos = max(pos, f * (long long)P.seg_traces);
                        end = min(stop, (f + 1) * (long long)P.seg_traces);
                        return true;
                    }
                    pos = (s0 + 32) * P.seg_traces;
                }
            }
            return false;
        };
        const float margin = 1.f + (CURVED && !P.cr_k_zero ? 4e-6f * fabsf(P.cr_inv_k_ln2) * P.inv_dt_f : 0.f);
        const float start_s = (float)(P.tstart_s / P.dt_s), last = (float)(P.ns - 1);
        const float t_min = 1.01f * 0.001f * P.inv_dt_f;
        int j = 0;
        for (;; ++j) {
            // ---- select: up to C traces near the patch, one per lane
            int cnt = 0;
            int batches = 1;   // 32 traces first: enough in a dense panel
            __syncwarp();
            while (cnt < C) {
                if (pos >= end) {
                    if (!next_range()) break;
                    continue;
                }
                double mx[4], my[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const long long i = pos + 32 * u + lane;
                    const bool in = u < batches && i < end;
                    mx[u] = in ? P.mx[i] : NAN;
                    my[u] = in ? P.my[i] : NAN;
                }
                const long long base = pos;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (u >= batches || cnt >= C || base + 32 * u >= end) break;
                    const double dx = fmax(fmax(x0 - mx[u], mx[u] - x1), 0.0);
                    const double dy = fmax(fmax(y0 - my[u], my[u] - y1), 0.0);
                    // (fmax drops a NaN midpoint, so ask the midpoint itself)
                    const bool in = dx * dx + dy * dy <= reach2 && mx[u] == mx[u] && my[u] == my[u];
                    const unsigned b = __ballot_sync(full, in);
                    const int r = __popc(b & below), room = C - cnt;
                    if (in && r < room) sh.selected[cnt + r] = base + 32 * u + lane;
                    const unsigned over = __ballot_sync(full, in && r == room);   // the first one left for the next chunk
                    pos = over ? base + 32 * u + __ffs(over) - 1 : min(end, base + 32 * (u + 1));
                    cnt += min(__popc(b), room);
                }
                batches = 4;
            }
            // ---- geometry, window and copy of this lane's trace
            const bool have = lane < cnt;
            __syncwarp();
            const long long id = have ? sh.selected[lane] : 0;
            double sx = 0, sy = 0, rx = 0, ry = 0, mx = 0, my = 0, w = 1.0;
            if (have) {
                sx = P.sx[id]; sy = P.sy[id];
                rx = P.rx[id]; ry = P.ry[id];
                mx = P.mx[id]; my = P.my[id];
                if (P.w) w = P.w[id];
            }
            float lo = INFINITY, hi = -INFINITY;
            bool finite;
            {
                auto near2 = [&](double x, double y) {
                    const float a = (float)fmax(fmax(x0 - x, x - x1), 0.0), b = (float)fmax(fmax(y0 - y, y - y1), 0.0);
                    return (a * a + b * b) * (1.f - 1e-6f);
                };
                auto far2 = [&](double x, double y) {
                    const float a = (float)fmax(fabs(x0 - x), fabs(x - x1)), b = (float)fmax(fabs(y0 - y), fabs(y - y1));
                    return (a * a + b * b) * (1.f + 1e-6f);
                };
                const float s0 = near2(sx, sy), s1 = far2(sx, sy), r0 = near2(rx, ry), r1 = far2(rx, ry);
                // A coordinate that is not finite, or farther than 1.8e19 m: the trace has no sample
                // for any pair.  Asked here, because the bounds' fminf and fmaxf lose a NaN, and a
                // trace that they wrongly call PLAIN is read without a test of its index.
                finite = s1 < INFINITY && r1 < INFINITY;
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    if (hb[g].A0 == INFINITY) continue;   // no live time in this half
                    float ls, us, lr, ur;
                    leg_bounds<TT>(P, hb[g], s0, s1, ls, us);
                    leg_bounds<TT>(P, hb[g], r0, r1, lr, ur);
                    lo = ls + lr >= lo ? lo : ls + lr;   // a NaN stays
                    hi = us + ur <= hi ? hi : us + ur;
                }
            }
            const float s_lo = lo * (1.f - 2e-6f) - start_s - margin;
            const float s_hi = hi * (1.f + 2e-6f) - start_s + margin;
            const bool none = lo == INFINITY && hi == -INFINITY;      // only T = 0 times
            const bool known = !any_unbounded && s_lo <= s_hi;        // (not NaN)
            int flags = !finite || (!any_unbounded && none) || (known && (s_hi < 0.f || s_lo >= last)) ? TRACE_DROP : 0;
            if (known && lo > t_min && fabs(w) < 1e30) flags |= TRACE_SURE;
            if (known && s_lo >= 0.f && s_hi < last) flags |= TRACE_INSIDE;
            int a = 0, e = P.ns - 1;   // samples the pairs can read
            if (known) {
                a = max(0, (int)floorf(s_lo));
                e = s_hi < last ? min(P.ns - 1, (int)s_hi + 2) : P.ns - 1;
            }
            const bool wanted = have && !(flags & TRACE_DROP);
            const bool too_wide = wanted && e - a + 1 + 2 * per16 > pitch;
            const uintptr_t row = reinterpret_cast<uintptr_t>(P.amps) + (uint64_t)(id * P.amp_stride) * (unsigned)P.elem;
            const uintptr_t first = row + (uint64_t)a * (unsigned)P.elem;
            const uintptr_t src = first & ~(uintptr_t)15;   // bulk copies start on 16 bytes
            const uintptr_t last_byte = row + (uint64_t)(e + 1) * (unsigned)P.elem;
            uintptr_t src_end = (last_byte + 15) & ~(uintptr_t)15;
            const bool at_end = src_end > reinterpret_cast<uintptr_t>(P.amps_end);   // not past the panel's end
            if (at_end) src_end = last_byte & ~(uintptr_t)15;
            const unsigned bytes = wanted && !too_wide && src_end > src ? (unsigned)(src_end - src) : 0u;
            const int al = a - (int)((first & 15u) / (unsigned)P.elem);   // sample at the row's start

            // ---- into the buffer, once every consumer is done with its last chunk
            const int b = j & 1;
            TraceTable &tab = sh.tab[b];
            if (j >= 2) timeout = __any_sync(full, !mbar_wait(b ? empty1 : empty0, (uint32_t)(((j >> 1) - 1) & 1), P.wait_iters));
            if (timeout) break;
            const unsigned dst = (unsigned)((b * kPool + lane * pitch) * P.elem);
            if (have) {
                tab.sx[lane] = sx; tab.sy[lane] = sy;
                tab.rx[lane] = rx; tab.ry[lane] = ry;
                tab.mx[lane] = mx; tab.my[lane] = my;
                tab.w[lane] = w;
                tab.id[lane] = id;
                const uint32_t buf = smem_u32(smem) + (unsigned)(wide_type ? b * kPool * 4 : 2 * kPool * 2);
                tab.row[lane] = make_int4((int)(buf + (unsigned)(lane * pitch * 4) - 4u * (INDEX_BASE + (unsigned)al)),
                                          (int)(INDEX_BASE + (unsigned)a), (e - a) | (lane << 24), flags);
                tab.window[lane] = make_int2(al, wanted && !too_wide ? e - al + 1 : 0);
                tab.t_hi[lane] = hi;
            }
            if (wanted && !too_wide && at_end) {
                for (uintptr_t q = src_end > src ? src_end : src; q < last_byte; q += (unsigned)P.elem) {
                    unsigned char *d = smem + dst + (q - src);
                    if (wide_type) *reinterpret_cast<float *>(d) = *reinterpret_cast<const float *>(q);
                    else *reinterpret_cast<unsigned short *>(d) = *reinterpret_cast<const unsigned short *>(q);
                }
            }
            const bool any_wide = __any_sync(full, too_wide);
            const unsigned total = __reduce_add_sync(full, bytes);
            if (lane == 0) {
                tab.cnt = cnt;
                tab.wide = any_wide;
            }
            fence_proxy_async();   // the buffer's last reads come before the copies
            __syncwarp();
            // (fault injection: with inject_stall the first chunks never arrive, so
            // the consumers' bounded waits for them run out)
            if (!(P.inject_stall && j < 2)) {
                if (lane == 0) mbar_expect_tx(b ? full1 : full0, total);
                __syncwarp();
                if (bytes) bulk_g2s(smem_u32(smem) + dst, reinterpret_cast<const void *>(src), bytes, b ? full1 : full0);
            }
            if (cnt == 0) break;   // the end of the traces: the consumers stop here
        }
        // The copies in flight must land before the CTA leaves.  Of the chunks whose consumers
        // are not known to be done these are, after a wait of this warp that gave up, the last
        // two; and else the last one, whose consumers may have given up themselves.
        if (lane == 0)
            for (int i = max(0, timeout ? j - 2 : j - 1); i < j; ++i)
                if (!(P.inject_stall && i < 2)) mbar_wait(i & 1 ? full1 : full0, (uint32_t)((i >> 1) & 1), P.wait_iters);
    } else {
        // ------------------------------------------------------------ consumers
        // traveltime (in the weights' unit), index word (INDEX_BASE + index when
        // inside the trace) and kFractionBase + fraction (EXACT) or fraction of one pair
        const float s_scale = P.s_scale, s_offset = P.s_offset;
        constexpr int R1 = 16 * kChunk, R2 = 32 * kChunk, RC = 40 * kChunk;
        // (T_test: T in the unit of its tests, asked for with clamp_c alone)
        auto locate = [&](int c, int g, float &T, float &f, unsigned &word, float &T_test, auto clamp_c) {
            const unsigned char *r = rec + c * 16;
            if constexpr (EXACT) {
                const double2 B = *reinterpret_cast<const double2 *>(r);
                double2 Cd = make_double2(0.0, 0.0);
                if constexpr (HAS_C) Cd = *reinterpret_cast<const double2 *>(r + RC);
                double v;
                const double T2 = exact_time<TT, KZ, decltype(clamp_c)::value>(P, log_tab, xs[g], ts[g].tz, ts[g].tzero, B, Cd, v);
                word = (unsigned)__double2hiint(v);
                f = __uint_as_float(__funnelshift_r((unsigned)__double2loint(v), 0x7Fu, 9));
                // rounded, but for straight rays truncated: 2^-24 of the weights either way round
                if constexpr (TT == TT_STRAIGHT) T = scaled_double_to_float(T2);
                else T = scaled_double_to_float_rn(T2);
                if constexpr (decltype(clamp_c)::value) {
                    if constexpr (TT == TT_STRAIGHT) T_test = scaled_double_to_float(T2 * xs[g].iv);
                    else T_test = (float)(CURVED ? T2 * (kSampleUnit / kTimeScale) : T2 * xs[g].iv * (1.0 / kTimeScale));
                }
            } else {
                const float4 B = *reinterpret_cast<const float4 *>(r);
                float4 Cf = make_float4(0.f, 0.f, 0.f, 0.f);
                if constexpr (CURVED) Cf = *reinterpret_cast<const float4 *>(r + RC);
                T = traveltime<TT, KZ, (decltype(clamp_c)::value || KZ)>(P, ts[g], st[g], B, Cf);
                const float s = fmaf(T, s_scale, s_offset);
                const float fl = __fadd_rd(s, 8388608.f);
                word = (unsigned)__float_as_int(fl);
                f = s - (fl - 8388608.f);
                if constexpr (decltype(clamp_c)::value) T_test = T;
            }
        };
        // A PLAIN or MID record at both of the lane's times: locate and read each,
        // then the interpolation and weights of both.  The point's factor K is
        // left to the flush.  The AA weight max(0, 1 - max(min(u aa_k,
        // aaA), f_dom/500)) is clamp(1 - u aa_k, L, H) with L = max(0, 1 - aaA), H =
        // max(0, 1 - f_dom/500).  MID adds the taper and the test of the index;
        // what is outside reads two zeros.  WEIGHT: the traces have weights.
        const float aa_hi = fmaxf(0.f, 1.f - P.aa_cB);
        const float2 aa_lo = make_float2(fmaxf(0.f, 1.f - st[0].aaA), fmaxf(0.f, 1.f - st[1].aaA));
        const float2 aa_nk = make_float2(-st[0].aa_k, -st[1].aa_k);
        const float2 m1 = make_float2(-1.f, -1.f), p1 = make_float2(1.f, 1.f);
        const uint32_t zero_addr = smem_u32(&sh.zero[0]);
        auto fast_record = [&](int c, float2 &acc, const float4 &e0, const float4 &e1, auto mid_c, auto weight_c) {
            constexpr bool MID = decltype(mid_c)::value;
            constexpr bool WEIGHT = decltype(weight_c)::value;
            const float4 q = *reinterpret_cast<const float4 *>(rec + R1 + c * 16);   // m, w, row, d
            const unsigned row = __float_as_uint(q.z);
            float2 T, f, a0, a1;
            unsigned w0, w1;
            float unused;
            locate(c, 0, T.x, f.x, w0, unused, std::false_type{});
            locate(c, 1, T.y, f.y, w1, unused, std::false_type{});
            uint32_t r0 = row + 4u * w0, r1 = row + 4u * w1;
            float2 x = make_float2(0.f, 0.f);   // 0 at the taper's inner edge, 1 at the aperture
            if constexpr (MID) {
                const uint2 h = *reinterpret_cast<const uint2 *>(rec + R2 + c * 8);
                const unsigned len = h.y & 0xffffffu;
                x = make_float2(__saturatef(fmaf(q.w, e0.y, e0.z)), __saturatef(fmaf(q.w, e1.y, e1.z)));
                r0 = w0 - h.x < len && x.x < 1.f ? r0 : zero_addr;
                r1 = w1 - h.x < len && x.y < 1.f ? r1 : zero_addr;
            }
            a0.x = lds_f32(r0);
            a1.x = lds_f32(r0 + 4u);
            a0.y = lds_f32(r1);
            a1.y = lds_f32(r1 + 4u);
            if constexpr (EXACT) f = __fadd2_rn(f, make_float2(-kFractionBase, -kFractionBase));
            float2 amp = __ffma2_rn(f, __ffma2_rn(a0, m1, a1), a0);
            const float2 rT = make_float2(rcp_approx(T.x), rcp_approx(T.y));
            if constexpr (WEIGHT) amp = make_float2(amp.x * q.y, amp.y * q.y);
            if (W2 || w_two) amp = __fmul2_rn(amp, __fmul2_rn(rT, rT));
            else if (w_one) amp = __fmul2_rn(amp, rT);
            float2 g = p1;
            if constexpr (AA) {
                g = __ffma2_rn(make_float2(q.x * rT.x, q.x * rT.y), aa_nk, p1);
                g.x = fminf(fmaxf(g.x, aa_lo.x), aa_hi);
                g.y = fminf(fmaxf(g.y, aa_lo.y), aa_hi);
                if constexpr (MID) g = __fmul2_rn(g, taper_weight2(x));
            } else if constexpr (MID) {
                g = taper_weight2(x);
            }
            if constexpr (AA || MID) acc = __ffma2_rn(amp, g, acc);
            else acc = __fadd2_rn(amp, acc);
        };
        // one EDGE record at one of the lane's times.  SLOW: only pairs in a
        // trace-end guard band, re-decided in FP64.  GLOBAL: the amplitudes come
        // from global memory (a window that does not fit its row).
        unsigned band_mask = 0u;
        const float g_mid = 0.5f * (P.s_guard_lo + P.s_guard_hi);
        const float g_in = P.s_guard_hi - g_mid, g_out = P.s_rej_hi - g_mid;
        auto edge_pair = [&](int c, int g, const TraceTable &tab, const float4 &ea, const float2 &ek, auto slow_c,
                             auto global_c) -> float {
            [[maybe_unused]] constexpr bool SLOW = decltype(slow_c)::value;
            constexpr bool GLOBAL = decltype(global_c)::value;
            const float4 q = *reinterpret_cast<const float4 *>(rec + R1 + c * 16);   // m, w, row, d
            const uint2 h = *reinterpret_cast<const uint2 *>(rec + R2 + c * 8);
            const float d = q.w;
            const int t = tblk * kTimes + 32 * g + lane;
            bool act = d <= ea.x;
            if (PREC != PSTM_PREC_FP32 && hard_cut && d == ea.x)   // FP32 tie of distance and aperture: decide in FP64
                act = !exact_outside_aperture(&P, tab.id[h.y >> 24], p, t, sh.warp[warp].ox, sh.warp[warp].oy);
            float T, f, T_test;
            unsigned word;
            locate(c, g, T, f, word, T_test, std::true_type{});
            bool ok;
            if constexpr (EXACT) {
                ok = act && word - INDEX_BASE < (unsigned)(P.ns - 1);
                f -= kFractionBase;
            } else {
                const float s = fmaf(T, s_scale, s_offset);
                if constexpr (GUARD) {
                    const float x = fabsf(s - g_mid);
                    const bool in = x <= g_in;
                    const bool band = act && !in && x <= g_out;
                    if constexpr (SLOW) {
                        ok = band && exact_sample_ok<TT>(&P, tab.id[h.y >> 24], p, t, sh.warp[warp].ox, sh.warp[warp].oy);
                        const float sc = fminf(fmaxf(s, 0.f), P.s_max_clamp);
                        const float fl = __fadd_rd(sc, 8388608.f);
                        word = (unsigned)__float_as_int(fl);
                        f = sc - (fl - 8388608.f);
                    } else {
                        ok = act && in;
                        band_mask |= band ? (1u << c) : 0u;
                    }
                } else {   // inside iff clamping leaves the index unchanged (NaN: outside)
                    ok = act && fminf(fmaxf(s, 0.f), P.s_max_clamp) == s;
                }
            }
            float a0, a1;
            if constexpr (GLOBAL) {
                const long long id = tab.id[h.y >> 24];
                const int i0 = (int)(word - INDEX_BASE);
                a0 = ok ? amp_global(P, id, i0) : 0.f;
                a1 = ok ? amp_global(P, id, i0 + 1) : 0.f;
            } else {
                ok = ok && word - h.x < (h.y & 0xffffffu);
                const uint32_t addr = ok ? __float_as_uint(q.z) + 4u * word : zero_addr;
                a0 = lds_f32(addr);
                a1 = lds_f32(addr + 4);
            }
            const float amp = fmaf(f, a1 - a0, a0);
            float w = q.y * taper_weight2(make_float2(__saturatef(fmaf(d, ea.y, ea.z)), 0.f)).x;
            const float rT = rcp_approx(T);
            const float tg = ek.y;
            float gw = ek.x;
            if (W2 || w_two) gw *= rT * rT;
            else if (w_one) gw *= rT;
            gw = T_test > tg ? gw : 1.f;   // the reference applies them only for T > 1 ms
            if constexpr (AA) {
                // sin(theta) = min(minf / (v_w T), 1); aaA sin(theta) = min(u aaA / v_w, aaA)
                const float u = q.x * rT;
                const float y = fminf(fmaxf(fmaf(u, g ? aa_nk.y : aa_nk.x, 1.f), g ? aa_lo.y : aa_lo.x), aa_hi);
                gw *= (q.x * rcp_approx(T_test) >= ea.w && T_test >= tg) ? y : 1.f;
            }
            const float v = amp * (w * gw);
            return ok ? v : 0.f;
        };
        using F = std::false_type;
        using Tr = std::true_type;
        float2 acc = make_float2(0.f, 0.f), acc_e = acc;   // PLAIN and MID records' sums (without K), EDGE records'
        auto flush = [&]() {
            sums[tid] += (double)fmaf(acc.x, edge_k[tid].x, acc_e.x);
            sums[kConsumers + tid] += (double)fmaf(acc.y, edge_k[kConsumers + tid].x, acc_e.y);
            acc = acc_e = make_float2(0.f, 0.f);
        };
        for (int k = 0;; ++k) {
            const int b = k & 1;
            timeout = __any_sync(full, !mbar_wait(b ? full1 : full0, (uint32_t)((k >> 1) & 1), P.wait_iters));
            const TraceTable &tab = sh.tab[b];
            if (!wide_type) {
                // every consumer has its chunk, and is done with the widened samples of the last
                timeout = consumers_or(timeout);
                if (timeout) break;
                const int cnt = tab.cnt;
                if (cnt == 0) break;
                const unsigned short *src = reinterpret_cast<const unsigned short *>(smem) + b * kPool;
                float *dst = reinterpret_cast<float *>(smem + 2 * kPool * 2);
                for (int c = warp; c < cnt; c += kPillars) {
                    const int n8 = min((tab.window[c].y + 7) / 8, pitch / 8);
                    for (int v = lane; v < n8; v += 32) {
                        const uint4 q = *reinterpret_cast<const uint4 *>(src + c * pitch + 8 * v);
                        const unsigned u[4] = {q.x, q.y, q.z, q.w};
                        float o[8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if (P.amp_kind == AMP_BF16) {
                                o[2 * i] = __uint_as_float(u[i] << 16);
                                o[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
                            } else {
                                const float2 h = __half22float2(*reinterpret_cast<const __half2 *>(&u[i]));
                                o[2 * i] = h.x;
                                o[2 * i + 1] = h.y;
                            }
                        }
                        float4 *d = reinterpret_cast<float4 *>(dst + c * pitch + 8 * v);
                        d[0] = make_float4(o[0], o[1], o[2], o[3]);
                        d[1] = make_float4(o[4], o[5], o[6], o[7]);
                    }
                }
                consumers_sync();
            }
            if (timeout) break;
            const int cnt = tab.cnt;
            if (cnt == 0) break;

            // ---- records of this warp's pillar: PLAIN, then MID, then EDGE
            bool plain = false, mid = false, edge = false;
            float d = 0.f, wt = 0.f, mz = 0.f, tz_term = 0.f;
            double ds2 = 0.0, dr2 = 0.0;
            int4 row = make_int4(0, 0, 0, 0);
            if (has_pillar && lane < cnt) {
                const double ox = sh.warp[warp].ox, oy = sh.warp[warp].oy;
                const double dxm = ox - tab.mx[lane], dym = oy - tab.my[lane];
                const double d2 = dxm * dxm + dym * dym;
                // the FP64 sqrt is needed only where the aperture cut is hard
                d = hard_cut ? (float)sqrt(d2) : sqrt_approx((float)d2);
                row = tab.row[lane];
                // the maximum aperture cuts for itself: a minimum above it raises every time's own
                if (d <= sh.warp[warp].apw && d2 <= P.fold_d2_max) {
                    const double dxs = ox - tab.sx[lane], dys = oy - tab.sy[lane];
                    const double dxr = ox - tab.rx[lane], dyr = oy - tab.ry[lane];
                    ds2 = dxs * dxs + dys * dys;
                    dr2 = dxr * dxr + dyr * dyr;
                    wt = P.w ? (float)tab.w[lane] : 1.f;
                    mz = (float)fmax(fabs(dxm), fabs(dym));
                    if (!(row.w & TRACE_DROP)) {
                        // T > 1 ms and sin(theta) >= 0.01 at every point of the warp
                        const float ap_in = sh.warp[warp].ap_in;
                        const bool sure = (row.w & TRACE_SURE) && sh.warp[warp].even &&
                                          (!AA || mz >= 1.0001f * sh.warp[warp].thr * tab.t_hi[lane]);
                        const bool in = hard_cut ? d < ap_in : d <= ap_in;
                        const bool inside = row.w & TRACE_INSIDE;
                        plain = sure && in && inside;
                        mid = sure && !plain && (in || !hard_cut) && (inside || !GUARD);
                        edge = !plain && !mid;
                    }
                    if (tz_lanes0 | tz_lanes1) {   // T = 0: the trace's amplitude at time zero
                        const double s0 = (0.0 - P.tstart_s) / P.dt_s;
                        if (s0 >= 0.0 && s0 < (double)(P.ns - 1)) {
                            const int i0 = (int)s0;
                            const float f = (float)(s0 - (double)i0);
                            const float a0 = amp_global(P, tab.id[lane], i0), a1 = amp_global(P, tab.id[lane], i0 + 1);
                            tz_term = fmaf(f, a1 - a0, a0) * wt;
                        }
                    }
                }
            }
            if (tz_lanes0 | tz_lanes1) {   // weights do not apply at T = 0; aperture and taper do
#pragma unroll 1
                for (int g = 0; g < 2; ++g) {
                    unsigned m = g ? tz_lanes1 : tz_lanes0;
                    while (m) {
                        const int l = __ffs(m) - 1;
                        m &= m - 1u;
                        const float4 ea = edge_a[32 * warp + l + g * kConsumers];
                        const float ap = -1.f - ea.x, itw = ea.y, tsn = ea.z;
                        bool act = has_pillar && lane < cnt && d <= ap;
                        if (PREC != PSTM_PREC_FP32 && hard_cut && act && d == ap)
                            act = !exact_outside_aperture(&P, tab.id[lane], p, tblk * kTimes + 32 * g + l,
                                                          sh.warp[warp].ox, sh.warp[warp].oy);
                        const float x = fmaf(d, itw, tsn);
                        float v = act ? tz_term * (x > 0.f ? taper_weight(x) : 1.f) : 0.f;
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(full, v, o);
                        if (lane == l) sums[g * kConsumers + tid] += (double)v;
                    }
                }
            }
            const unsigned mp = __ballot_sync(full, plain), mt = __ballot_sync(full, mid);
            const unsigned me = __ballot_sync(full, edge);
            const int np = __popc(mp), nm = np + __popc(mt), n = nm + __popc(me);
            if (plain || mid || edge) {
                const int slot = plain ? __popc(mp & below) : (mid ? np + __popc(mt & below) : nm + __popc(me & below));
                unsigned char *r = rec + slot * 16;
                *reinterpret_cast<float4 *>(r + R1) = make_float4(mz, wt, __int_as_float(row.x), d);
                *reinterpret_cast<int2 *>(rec + R2 + slot * 8) = make_int2(row.y, row.z);
                if constexpr (EXACT) {
                    const double xs2 = record_square<TT, KZ>(P, ds2), xr2 = record_square<TT, KZ>(P, dr2);
                    *reinterpret_cast<double2 *>(r) = make_double2(xs2, xr2);
                    if constexpr (TT == TT_VTI)
                        *reinterpret_cast<double2 *>(r + RC) = make_double2(xs2 * xs2, xr2 * xr2);
                }
                float4 Bf = make_float4((float)ds2, (float)dr2, 0.f, 0.f);
                if constexpr (CURVED) {
                    const double k2 = P.cr_k2, v0 = P.cr_v0;
                    const double bs = v0 + sqrt(v0 * v0 + k2 * ds2), br = v0 + sqrt(v0 * v0 + k2 * dr2);
                    const double2 Cd = TT == TT_CURVED ? make_double2(1.0 / (bs * br), 0.0)
                                                       : make_double2(1.0 / bs, 1.0 / br);
                    if constexpr (EXACT) {
                        *reinterpret_cast<double2 *>(r + RC) =
                            TT == TT_CURVED ? make_double2(0.25 * Cd.x, 0.0) : make_double2(0.5 * Cd.x, 0.5 * Cd.y);
                    } else {
                        Bf.z = (float)(k2 * ds2);
                        Bf.w = (float)(k2 * dr2);
                        *reinterpret_cast<float4 *>(r + RC) =
                            TT == TT_CURVED ? make_float4((float)Cd.x, 0.f, 0.f, 0.f)
                                            : make_float4((float)Cd.x, (float)Cd.y, (float)(ds2 * ds2), (float)(dr2 * dr2));
                    }
                } else if constexpr (TT == TT_VTI) {
                    Bf.z = (float)(ds2 * ds2);
                    Bf.w = (float)(dr2 * dr2);
                }
                if constexpr (!EXACT) *reinterpret_cast<float4 *>(r) = Bf;
            }
            __syncwarp();

            // ---- pairs
            const bool wide = tab.wide != 0;   // rare: a window of this chunk is too long to stage
            const bool weighted = P.w != nullptr;
            if (!wide) {
                const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
                if (weighted) {
#pragma unroll 4
                    for (int c = 0; c < np; ++c) fast_record(c, acc, none, none, F{}, Tr{});
                } else {
#pragma unroll 4
                    for (int c = 0; c < np; ++c) fast_record(c, acc, none, none, F{}, F{});
                }
                if (np < nm) {
                    const float4 e0 = edge_a[tid], e1 = edge_a[kConsumers + tid];
                    if (weighted) {
#pragma unroll 2
                        for (int c = np; c < nm; ++c) fast_record(c, acc, e0, e1, Tr{}, Tr{});
                    } else {
#pragma unroll 2
                        for (int c = np; c < nm; ++c) fast_record(c, acc, e0, e1, Tr{}, F{});
                    }
                }
            }
            if (wide || nm < n || GUARD) {
                const float4 e0 = edge_a[tid], e1 = edge_a[kConsumers + tid];
                const float2 k0 = edge_k[tid], k1 = edge_k[kConsumers + tid];
                if (wide) {
#pragma unroll 1
                    for (int c = 0; c < n; ++c) {
                        acc_e.x += edge_pair(c, 0, tab, e0, k0, F{}, Tr{});
                        acc_e.y += edge_pair(c, 1, tab, e1, k1, F{}, Tr{});
                    }
                } else {
#pragma unroll 1
                    for (int c = nm; c < n; ++c) {
                        acc_e.x += edge_pair(c, 0, tab, e0, k0, F{}, F{});
                        acc_e.y += edge_pair(c, 1, tab, e1, k1, F{}, F{});
                    }
                }
                if constexpr (GUARD) {   // pairs in a trace-end guard band, re-decided in FP64
                    unsigned m = __reduce_or_sync(full, band_mask);
                    band_mask = 0u;
                    while (m) {
                        const int c = __ffs(m) - 1;
                        m &= m - 1u;
                        acc_e.x += edge_pair(c, 0, tab, e0, k0, Tr{}, Tr{});
                        acc_e.y += edge_pair(c, 1, tab, e1, k1, Tr{}, Tr{});
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(b ? empty1 : empty0);
            if ((k & P.flush_mask) == P.flush_mask) flush();
        }
        flush();
    }
    if (timeout && lane == 0) atomicOr(P.err, (int)KERR_WAIT_TIMEOUT);

    // ---------------- epilogue: image += the sums (of every rank, in rank order)
    __syncthreads();
    if (shares > 1) {
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        if (rank == 0 && !producer) {
            for (int r = 1; r < shares; ++r) {
                const double *other = cl.map_shared_rank(sums, r);
                sums[tid] += other[tid];
                sums[kConsumers + tid] += other[kConsumers + tid];
            }
        }
        cl.sync();
    }
    if (rank == 0 && has_pillar) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const int t = tblk * kTimes + 32 * g + lane;
            const double a = sums[g * kConsumers + tid];
            if (t < P.nt && a != 0.0) {
                const int64_t idx = (int64_t)p * P.nt + t;
                if (P.image_f32) {
                    float &o = static_cast<float *>(image)[idx];
                    o = (float)((double)o + a);
                } else {
                    static_cast<double *>(image)[idx] += a;
                }
            }
        }
    }
}

}  // namespace pstm
