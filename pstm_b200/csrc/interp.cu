// interp.cu -- migration with a higher-order trace interpolator.
//
// The reference's NumbaKernel takes KernelConfig.interpolation_method and
// interpolates every sample with interpolate_sample (pstm/kernels/
// numba_cpu.py:341, pstm/kernels/interpolation.py:254-301): nearest,
// Catmull-Rom cubic, Hanning-windowed sinc of 4/8/16 points and Lanczos 3/5,
// the wide ones falling back to linear within their half-width of a trace end
// and normalising by the sum of their weights.  Linear interpolation stays on
// the tiled gather kernel; the other methods run here -- in FP64 (traveltime,
// sample index, interpolation weights and accumulation) on the exact path, with
// FP32 taps, interpolation and weights after the FP64 sample index on the fast
// path -- with one CTA of 128
// threads per (pillar, block of 128 output times) and the traces read from
// the caller's geometry and panel.  Each warp stages the traces 32
// at a time in a shared-memory slice of its own: each lane takes one trace's
// pillar distances, counts it for the fold and keeps it if it lies inside the
// largest aperture of the warp's times; the kept traces, in trace order, go to
// the slice and every lane then runs them against its own output time.  Warps
// synchronise only with themselves, so none waits for a warp whose times
// keep more traces.  Aperture, taper, weights, AA and
// fold are those of the gather kernel.
#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

#include "pstm_cuda.h"
#include "kparams.h"
#include "launch.h"
#include "migrate.cuh"
#include "ctx.h"

using namespace pstm;
using namespace pstm::ctx;

namespace {

constexpr int kInterpThreads = 128;
// CTAs per SM the register budget is sized for: the kernel is bound by
// dependent FP64 latency, so more resident warps beat the few values that
// spill to L1 at this budget.
#ifndef PSTM_INTERP_MIN_CTAS
#define PSTM_INTERP_MIN_CTAS 8
#endif

template <int AMP, typename R = double>
__device__ inline R sample_at(const unsigned char *row, int64_t i) {
    return (R)amp_at<AMP>(row, (int)i);
}

// 1/x in the interpolation arithmetic: the hardware approximation refined by
// one Newton step in FP64 (~1 ulp), the approximation itself in FP32.
__device__ inline double rcp_r(double x) { return rcp_newton(x); }
__device__ inline float rcp_r(float x) { return rcp_approx(x); }

// Nearest, Catmull-Rom cubic and linear interpolation at the fractional index i +
// f, 0 <= f < 1 (0 <= i + f < ns - 1 is checked by the caller); linear also serves
// the wide methods within their half-width of a trace end.
// R is the arithmetic of the weights and taps: double (exact path) or float
// (fast path); index and fraction are FP64 in both, and so is which sample is nearest.
template <int AMP, typename R>
__device__ R interpolate_narrow(const unsigned char *row, int ns, int i, double fr, int method) {
    if (method == PSTM_INTERP_NEAREST) return sample_at<AMP, R>(row, fr < 0.5 ? i : i + 1);
    const R f = (R)fr;
    if (method == PSTM_INTERP_CUBIC && i >= 1 && i < ns - 2) {   // Catmull-Rom
        const R p0 = sample_at<AMP, R>(row, i - 1), p1 = sample_at<AMP, R>(row, i);
        const R p2 = sample_at<AMP, R>(row, i + 1), p3 = sample_at<AMP, R>(row, i + 2);
        const R c3 = R(-0.5) * p0 + R(1.5) * p1 - R(1.5) * p2 + R(0.5) * p3;
        const R c2 = p0 - R(2.5) * p1 + R(2.0) * p2 - R(0.5) * p3;
        const R c1 = R(-0.5) * p0 + R(0.5) * p2;
        return ((c3 * f + c2) * f + c1) * f + p1;
    }
    return sample_at<AMP, R>(row, i) * (R(1) - f) + sample_at<AMP, R>(row, i + 1) * f;
}

// cos(pi K / HW) and sin(pi K / HW) at compile time: the angle folded into
// [0, pi / 2], then the Taylor series.
constexpr double kPi = 3.14159265358979323846;
constexpr double cx_cos(double x) {
    double t = 1.0, s = 1.0;
    for (int n = 1; n < 16; ++n) {
        t *= -x * x / ((2.0 * n - 1.0) * (2.0 * n));
        s += t;
    }
    return s;
}
constexpr double cx_fold(int k, int hw) {   // cos(pi k / hw), |k| <= 2 hw
    if (k < 0) k = -k;
    if (k > hw) k = 2 * hw - k;
    if (2 * k == hw) return 0.0;
    return 2 * k > hw ? -cx_cos(kPi * (hw - k) / hw) : cx_cos(kPi * k / hw);
}
template <int HW, int K>
constexpr double win_cos = cx_fold(K, HW);
template <int HW, int K>
constexpr double win_sin = cx_fold(2 * K - HW, 2 * HW);   // cos of the angle less pi / 2
constexpr double cx_inv_factorial(int n) {
    double f = 1.0;
    for (int i = 2; i <= n; ++i) f /= i;
    return f;
}
template <int N>
constexpr double taylor = (N / 2 % 2 ? -1.0 : 1.0) * cx_inv_factorial(N);   // of y^N in cos (even N) or sin
// Taylor polynomial in u = y^2 from y^N on, up to the power LAST.
template <int N, int LAST, typename R>
__device__ __forceinline__ R taylor_from(R u) {
    if constexpr (N + 2 > LAST) return (R)taylor<N>;
    else return taylor_from<N + 2, LAST, R>(u) * u + (R)taylor<N>;
}
// Last power of y that matters in cos and sin up to y <= pi / 2: the next term is below
// 2^-54, half a unit in the last place of a double below 1.
constexpr int taylor_last(double y) {
    int n = 1;
    double next = y * y / 2;
    while (next > 0x1p-54) next *= y / (++n + 1);
    return n;
}
static_assert(taylor_last(kPi / 8) == 13 && taylor_last(kPi / 3) == 18 && taylor_last(kPi / 2) == 21, "sinc8, Lanczos-3, taper");

// Windowed sinc (LANCZOS false) or Lanczos (true) of half-width HW at the
// fractional index i + f (0 <= f < 1), normalised by the sum of the weights; linear
// within HW samples of a trace end.
//
// The direct weights are, at the 2 HW taps x_k = f - k, k = -HW+1 .. HW, sinc(x) =
// sin(pi x) / (pi x) times a Hann window 0.5 (1 + cos(pi x / HW)) that is 0 for |x| >=
// HW, or (Lanczos) times sinc(x / HW).  sin(pi x_k) is (-1)^k sin(pi f), so every
// factor common to the taps cancels in the normalisation and what is left is
//   sinc     (-1)^k (1 + cos(pi x_k / HW)) / x_k
//   Lanczos  (-1)^k sin(pi x_k / HW) / x_k^2.
// cos and sin of pi (f - k) / HW are combinations of C, S = cos, sin(pi f / HW) with
// compile-time factors: two Taylor polynomials serve all taps.  The divisions go
// too: taps k and 1 - k are the roots of D_k = f^2 - f - k (k - 1), so 1 / x_k = x_{1-k} /
// D_k, and multiplying all weights by the product of the D's (again common)
// leaves x_{1-k} E_k, E_k the product of the other D's.  Nothing is divided but the
// final sum; on a sample (f = 0), where the Lanczos weights all vanish and the sinc
// weights of the other taps do, the sample is returned.
//
// The fraction comes in FP64: it decides which sample is nearest, and f - 1 is rounded
// from it, not from f.  Next to a fraction of 1 the Lanczos tap there needs x_1 = f - 1
// and sin(pi x_1 / HW) to their own size: its sine is a polynomial of x_1, since the
// rotation of C and S leaves an absolute error.
//
// The form before this one took a Newton-refined reciprocal, a rotation of the
// window angle and a libm sincospi per sample: 1160 issue cycles a pair for sinc8
// in FP64 (FP64 instructions take 2.1-3.4 cycles to issue).
template <int AMP, int HW, bool LANCZOS, typename R>
struct Wide {
    static constexpr int kLast = taylor_last(kPi * (LANCZOS ? 1.0 : 0.5) / HW);

    const unsigned char *row;
    int i, i_max;
    R f, f1, C, S, S1, acc, norm;   // f1 = f - 1, S1 = sin(pi f1 / HW) (Lanczos)
    R centre;                       // the sample at f = 0 (sinc)
    R E[HW], FE[HW];   // E[k - 1]: product of the D's but D_k; f E

    // C cos + S sin with compile-time factors; 0 and 1 cost nothing
    static __device__ __forceinline__ R rotate(R a, R b, double ca, double sb) {
        if (ca == 0.0) return sb == 1.0 ? b : (sb == -1.0 ? -b : b * (R)sb);
        if (sb == 0.0) return ca == 1.0 ? a : (ca == -1.0 ? -a : a * (R)ca);
        return a * (R)ca + b * (R)sb;
    }
    // taps J and J - HW, whose window angles differ by pi: the Hann window's cosine
    // (and the Lanczos sine) changes its sign from one to the other
    template <int J>
    __device__ __forceinline__ void tap_pair(bool live) {
        if constexpr (LANCZOS) {
            const R sn = J == 1 ? S1 : rotate(S, C, win_cos<HW, J>, -win_sin<HW, J>);
            const R ea = x_over<J>(), eb = x_over<J - HW>();
            const R wa = (J & 1 ? -sn : sn) * ea * ea, wb = ((J - HW) & 1 ? sn : -sn) * eb * eb;
            add(wa, i + J);
            add(wb, i + J - HW);
        } else {
            const R cs = rotate(C, S, win_cos<HW, J>, win_sin<HW, J>);
            R wa = (J & 1 ? R(-1) - cs : R(1) + cs) * x_over<J>();
            const R wb = (J & 1 ? cs - R(1) : R(1) - cs) * x_over<J - HW>();
            int ja = i + J;
            if constexpr (J == HW) {   // beyond the window (and possibly the trace) for f < 0
                wa = live ? wa : R(0);
                ja = min(ja, i_max);
            }
            add(wa, ja);
            const R sample = add(wb, i + J - HW);
            if constexpr (J == HW) centre = sample;
        }
    }
    template <int K>   // E / x_K = x_{1-K} E_k
    __device__ __forceinline__ R x_over() const {
        constexpr int k = K > 0 ? K : 1 - K;
        if constexpr (K == 0) return f1 * E[0];
        else return FE[k - 1] + (R)(K - 1) * E[k - 1];
    }
    __device__ __forceinline__ R add(R w, int j) {
        const R sample = sample_at<AMP, R>(row, j);
        acc += sample * w;
        norm += w;
        return sample;
    }
    template <int... J>
    __device__ __forceinline__ void taps(std::integer_sequence<int, J...>, bool live) {
        (tap_pair<J + 1>(live), ...);
    }
    __device__ __forceinline__ R run(const unsigned char *r, int ns, int i0, double fr) {
        if (i0 < HW || i0 >= ns - HW) {
            const R fl = (R)fr;
            return sample_at<AMP, R>(r, i0) * (R(1) - fl) + sample_at<AMP, R>(r, i0 + 1) * fl;
        }
        row = r;
        i_max = ns - 1;
        i = i0;
        if (!LANCZOS && fr >= 0.5) {   // sinc counts from the nearest sample: -0.5 <= f < 0.5
            i += 1;
            fr -= 1.0;
        }
        if constexpr (LANCZOS) {
            if (fr < 1e-10) return sample_at<AMP, R>(row, i);
            if (1.0 - fr < 1e-10) return sample_at<AMP, R>(row, i + 1);
        }
        f = (R)fr;
        f1 = (R)(fr - 1.0);
        const R y = f * (R)(kPi / HW), u = y * y;
        C = taylor_from<0, kLast, R>(u);
        S = taylor_from<1, kLast, R>(u) * y;
        if constexpr (LANCZOS) {
            const R y1 = f1 * (R)(kPi / HW);
            S1 = taylor_from<1, kLast, R>(y1 * y1) * y1;
        }
        const R g = f * f1;
        R D[HW];
#pragma unroll
        for (int k = 1; k <= HW; ++k) D[k - 1] = g - (R)(k * (k - 1));
        // E by prefix and suffix products
        R pre = R(1);
#pragma unroll
        for (int k = 0; k < HW; ++k) {
            E[k] = pre;
            pre *= D[k];
        }
        R suf = R(1);
#pragma unroll
        for (int k = HW - 1; k >= 0; --k) {
            E[k] *= suf;
            suf *= D[k];
            FE[k] = f * E[k];
        }
        acc = norm = R(0);
        taps(std::make_integer_sequence<int, HW>{}, f >= R(0));
        const R value = norm != R(0) ? acc * rcp_r(norm) : R(0);
        // on a sample nothing but it counts, not even 0 times a NaN beside it (a return
        // before the taps costs 5 %)
        return !LANCZOS && fabs(f) < R(1e-10) ? centre : value;
    }
};

// 0.5 (1 + cos(pi x)) = cos^2(pi x / 2), 0 <= x <= 1, from cos's Taylor polynomial.
template <typename R>
__device__ __forceinline__ R taper_weight_r(R x) {
    const R y = x * (R)(0.5 * kPi);
    const R c = taylor_from<0, taylor_last(0.5 * kPi), R>(y * y);
    return c * c;
}

template <int TT>
__device__ inline double tt_of(double t0, double ds2, double dr2, double v, double eta, double v0, double k) {
    return traveltime_fp64<TT>(t0, ds2, dr2, v, eta, v0, k);
}

// Per-trace values a warp stages in shared memory for the CTA's pillar.
struct Staged {
    double ds2[32], dr2[32], d[32], w[32], m[32];
    const unsigned char *row[32];
};

// R: double on the exact path (FP64 end to end); float on the fast path,
// where only the traveltime, the sample index and the accumulation stay FP64
// and the taps, the interpolation and the weights are FP32.
template <int AMP, int HW, bool LANCZOS, typename R>
__global__ void __launch_bounds__(kInterpThreads, PSTM_INTERP_MIN_CTAS) migrate_interp_kernel(const KParams P, int tt, int method) {
    __shared__ Staged S_all[kInterpThreads / 32];
    const int p = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ix = p / P.ny, iy = p - ix * P.ny;
    const double ox = P.xg ? P.xg[p] : P.xa[ix], oy = P.yg ? P.yg[p] : P.ya[iy];
    const int t = blockIdx.y * kInterpThreads + threadIdx.x;
    const bool tv = t < P.nt;
    const int tc = tv ? t : P.nt - 1;
    const double t0 = P.ta[tc] / 1000.0;
    const double v = P.vel3d ? P.vrms[(int64_t)p * P.nt + tc] : P.vrms[tc];
    double eta = P.eta_const;
    if (P.eta) eta = P.eta3d ? P.eta[(int64_t)p * P.nt + tc] : P.eta[tc];
    double ap = v * t0 * 0.5 * P.tan_dip;
    ap = ap < P.min_ap ? P.min_ap : (ap > P.max_ap ? P.max_ap : ap);
    double vw = v;   // weights use v_rms, or v(z) at the image depth for curved rays
    if (P.curved_kind) {
        const double z = P.cr_k_zero ? P.cr_v0 * (t0 * 0.5) : (P.cr_v0 / P.cr_k) * (exp(P.cr_k * (t0 * 0.5)) - 1.0);
        vw = P.cr_v0 + P.cr_k * z;
    }
    const double taper_start = ap * (1.0 - P.taper);
    const double inv_taper_w = ap > taper_start ? 1.0 / (ap - taper_start) : 0.0;
    const double inv_dt = 1.0 / P.dt_s;
    // The weights need L = v_w T alone: spreading 1 / L, obliquity (t0 v_w) / L,
    // sin(theta) = m / L.  The sample index is formed in seconds with one Newton step:
    // a windowed sinc jumps by 0.4 % of a sample where its nearest sample changes, so
    // another rounding of the index (in metres, or a third-order step; neither faster: 32.1
    // against 31.8-32.1 ms for 40 x 40 x 500 points and 6,000 traces) moves a
    // few pairs of 10^9 across a jump and an FP64 image by 2e-9.
    const double iv2 = 1.0 / (v * v);
    // (at t0 = 0 above 0, so that a leg of length 0 has a root)
    const double t0h2 = fmax((t0 * 0.5) * (t0 * 0.5), 1e-30), vw2 = 2.0 * vw;
    const R K = P.obliquity ? (R)(t0 * vw) : R(1);
    const int n_inv = (P.spreading ? 1 : 0) + (P.obliquity ? 1 : 0);
    const R aa_A = (R)(4.0 * P.aa_gmax * P.aa_fdom / vw);
    const R aa_lo = fmax(R(0), R(1) - aa_A), aa_hi = fmax(R(0), (R)(1.0 - P.aa_fdom / 500.0));
    // T <= 1 ms, where the weights do not apply, needs t0 < 1.1 ms or curved rays
    const bool small_t = P.curved_kind || t0 < 0.0011;
    const double L2_min = small_t ? 0.002 * vw : -1.0;

    Staged &S = S_all[warp];
    // Largest aperture over the warp's output times: a trace farther than it
    // from the pillar adds nothing at any of them.
    double ap_w = tv ? ap : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ap_w = fmax(ap_w, __shfl_xor_sync(0xffffffffu, ap_w, o));

    double acc = 0.0;
    int cnt = 0;   // traces within the fold radius; the same in every lane
    for (int64_t c0 = 0; c0 < P.n_traces; c0 += 32) {
        const int64_t tr = c0 + lane;
        bool keep = false, in_fold = false;
        double dxm = 0.0, dym = 0.0, d = 0.0;
        if (tr < P.n_traces) {
            dxm = ox - P.mx[tr];
            dym = oy - P.my[tr];
            const double d2 = dxm * dxm + dym * dym;
            in_fold = d2 <= P.fold_d2_max;
            d = sqrt(d2);
            keep = in_fold && !(d > ap_w);   // the maximum cuts for itself, also below the minimum
        }
        const unsigned kb = __ballot_sync(0xffffffffu, keep);
        cnt += __popc(__ballot_sync(0xffffffffu, in_fold));
        const int n_kept = __popc(kb);
        if (keep) {
            const int j = __popc(kb & ((1u << lane) - 1u));
            const double dxs = ox - P.sx[tr], dys = oy - P.sy[tr], dxr = ox - P.rx[tr], dyr = oy - P.ry[tr];
            S.ds2[j] = dxs * dxs + dys * dys;
            S.dr2[j] = dxr * dxr + dyr * dyr;
            S.d[j] = d;
            S.w[j] = P.w ? P.w[tr] : 1.0;
            S.m[j] = fmax(fabs(dxm), fabs(dym));
            S.row[j] = reinterpret_cast<const unsigned char *>(P.amps) + tr * P.amp_stride * (int64_t)P.elem;
        }
        __syncwarp();
        for (int j = 0; j < n_kept; ++j) {
            const double dj = S.d[j];
            if (!tv || dj > ap) continue;
            const double ds2 = S.ds2[j], dr2 = S.dr2[j];
            double T;
            switch (tt) {
            case TT_CURVED: T = tt_of<TT_CURVED>(t0, ds2, dr2, v, eta, P.cr_v0, P.cr_k); break;
            case TT_VTI: T = tt_of<TT_VTI>(t0, ds2, dr2, v, eta, P.cr_v0, P.cr_k); break;
            case TT_CURVED_VTI: T = tt_of<TT_CURVED_VTI>(t0, ds2, dr2, v, eta, P.cr_v0, P.cr_k); break;
            default: T = sqrt_newton(fma(ds2, iv2, t0h2)) + sqrt_newton(fma(dr2, iv2, t0h2)); break;
            }
            const double s = (T - P.tstart_s) * inv_dt, L2 = vw2 * T;
            if (!(s >= 0.0 && s < (double)(P.ns - 1))) continue;
            const unsigned char *row = S.row[j];
            // integer and fraction without conversions: s + 1.5 2^52 has the nearest
            // integer in its low word
            const double near = s + 6755399441055744.0;
            int i0 = __double2loint(near);
            double fr = s - (near - 6755399441055744.0);
            if (fr < 0.0) {
                i0 -= 1;
                fr += 1.0;
            }
            R amp;
            if constexpr (HW > 0) amp = Wide<AMP, HW, LANCZOS, R>().run(row, P.ns, i0, fr);
            else amp = interpolate_narrow<AMP, R>(row, P.ns, i0, fr, method);
            R w = (R)S.w[j];
            if (dj > taper_start) w *= taper_weight_r((R)((dj - taper_start) * inv_taper_w));
            const R inv = R(2) * rcp_r((R)L2);
            R g = R(1);
            if (n_inv == 2) g = K * inv * inv;
            else if (n_inv == 1) g = K * inv;
            g = L2 > L2_min ? g : R(1);
            if (P.aa && L2 >= L2_min) {
                const R sn = (R)S.m[j] * inv;
                R y = R(1) - aa_A * sn;
                y = y > aa_hi ? aa_hi : y;
                y = y < aa_lo ? aa_lo : y;
                g = sn >= R(0.01) ? g * y : g;
            }
            acc += (double)(amp * (w * g));
        }
        __syncwarp();   // the next batch overwrites the staged values
    }
    if (tv) {
        const int64_t idx = (int64_t)p * P.nt + t;
        if (P.image_f32) reinterpret_cast<float *>(P.image)[idx] += (float)acc;
        else reinterpret_cast<double *>(P.image)[idx] += acc;
        if (P.fold && P.fold3d) P.fold[idx] += cnt;
    }
    if (P.fold && !P.fold3d && blockIdx.y == 0 && threadIdx.x == 0) P.fold[p] += cnt;
}

template <int AMP, int HW, bool LANCZOS>
void launch_one(const TilePlan &tp, dim3 grid, int method) {
    if (tp.exact)
        migrate_interp_kernel<AMP, HW, LANCZOS, double><<<grid, kInterpThreads, 0, tp.L.stream>>>(tp.P, tp.tt, method);
    else
        migrate_interp_kernel<AMP, HW, LANCZOS, float><<<grid, kInterpThreads, 0, tp.L.stream>>>(tp.P, tp.tt, method);
}

template <int AMP>
void launch_method(const TilePlan &tp, dim3 grid, int method) {
    switch (method) {
    case PSTM_INTERP_SINC4: launch_one<AMP, 2, false>(tp, grid, method); break;
    case PSTM_INTERP_SINC8: launch_one<AMP, 4, false>(tp, grid, method); break;
    case PSTM_INTERP_SINC16: launch_one<AMP, 8, false>(tp, grid, method); break;
    case PSTM_INTERP_LANCZOS3: launch_one<AMP, 3, true>(tp, grid, method); break;
    case PSTM_INTERP_LANCZOS5: launch_one<AMP, 5, true>(tp, grid, method); break;
    default: launch_one<AMP, 0, false>(tp, grid, method); break;   // nearest, cubic, linear
    }
}

}  // namespace

namespace pstm {
namespace ctx {
// Launch of the higher-order-interpolation kernel on a prepared tile.
int32_t launch_interp(Ctx *c, const TilePlan &tp, int method, const pstm_output_desc *out) {
    if (tp.P.n_traces > INT32_MAX) return fail(c, PSTM_ERR_INVALID_ARGUMENT, "interpolation kernel takes at most 2^31 - 1 traces");
    const dim3 grid((unsigned)((int64_t)out->nx * out->ny), (unsigned)((out->nt + kInterpThreads - 1) / kInterpThreads));
    switch (tp.amp) {
    case PSTM_AMP_F32: launch_method<AMP_F32>(tp, grid, method); break;
    case PSTM_AMP_BF16: launch_method<AMP_BF16>(tp, grid, method); break;
    default: launch_method<AMP_F16>(tp, grid, method); break;
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PSTM_OK : cuda_fail(c, e, "interpolation migrate kernel launch");
}
}  // namespace ctx
}  // namespace pstm
