// Mixed-precision path (GCV_MIXED), and the sampling of FP64 tables: the
// integrand and the panel sums run on the FP32 pipes in float-float arithmetic
// (gcv_ff.cuh, ~48-bit significand);
// FP64 is kept for the steps whose stability needs it:
//   * the compensated prefix sum of interval lengths (k_scan, shared with the
//     FP64 path),
//   * the panel error test when the FP32 test lands near the tolerance,
//   * a sample's target, its place among the intervals and leaves, and its
//     parameter (the local one, final Newton update included, in 64-bit fixed
//     point).
// Plain FP32 integrands (rounding ~3e-8 per evaluation, plus the systematic
// rounding of each interval's polynomial coefficients) cannot hold a 1e-8
// relative length on curves of one or a few knot intervals; float-float can,
// at a fraction of the FP64 cost on GB300 (FP32:FP64 throughput ~75:1).
//
// Ellipse integrands are evaluated by angle addition from one float-float sine
// and cosine per panel or leaf side (gcv_ff_eval.cuh).
#pragma once

#include <type_traits>

#include "gcv_ff_eval.cuh"
#include "gcv_kernels.cuh"

namespace gcv {

// ------------------------------------------------------------- sampling
// Newton on one leaf in float-float, in the local offset w = v - va in
// [0, dv]: F(w) = S(va + w) - S(va) - rl with the partial integral taken by
// 8-point Gauss over the shorter side of the leaf, bracketed by bisection.
// From F and the speed f0 at w, the Newton point w - dn; with the speed f1 there
// the second-order step d = 2 F / (f0 + f1), and the stopping test of leaf_newton
// (gcv_kernels.cuh): dn^2 (|f'(w - dn) - f'(w)| / 3 + |f'|^2 |dn| / (4 f)) <= eps_s.
// Where that is not enough, the speed half way (fm, in FP32 like f1) gives the
// length of the step by a rule of order seven (Simpson's and the end-corrected
// trapezoidal rule combined, their difference E the error's measure), and what of
// F that leaves its own second-order step: taken when its residual is below eps_t,
// which stands for what another iteration would leave.  Without it 9 % of the
// samples of 50,000 spatial curves took another iteration, so most warps did; now
// 6 %: 10.2 -> 9.58 ms, the uneven batch of 100,000 curves 11.3 -> 10.6, 4,096
// ellipses 0.45 -> 0.42, 10,000 cubics at rtol 1e-10 0.82 -> 0.80.  (Taken wherever
// its residual is below eps_s itself: 8.5, 9.9, 0.41, 0.77 ms, but with samples off by
// eps_s where an iteration left rounding.)
// Returns the final offset in units of 2^-60.
// 8-point Gauss nodes (-x0..-x3, x0..x3) then weights w0..w3, float-float
#define GCV_FFC(x) {split_const(x).hi, split_const(x).lo}
static __constant__ float2 c_gl8_ff[12] = {
    GCV_FFC(-gl8_x(0)), GCV_FFC(-gl8_x(1)), GCV_FFC(-gl8_x(2)), GCV_FFC(-gl8_x(3)),
    GCV_FFC(gl8_x(0)),  GCV_FFC(gl8_x(1)),  GCV_FFC(gl8_x(2)),  GCV_FFC(gl8_x(3)),
    GCV_FFC(gl8_w(0)),  GCV_FFC(gl8_w(1)),  GCV_FFC(gl8_w(2)),  GCV_FFC(gl8_w(3))};
#undef GCV_FFC

// Whether the sampler of curve code C takes its Gauss sums by node pairs
// (gl8_pairs) rather than by evaluating each node: the B-spline codes of
// degree x dimension below 10.  The larger codes hold more coefficients than
// their register cap leaves room for beside the pairs' temporaries: sampling of
// 50,000 spatial cubics and quintics took 10.4 ms with pairs below 8, 10.2
// below 10, 11.1 for every code.
__host__ __device__ constexpr bool sample_node_pairs(int code)
{
    return code > 0 && code_degree(code) * code_dim(code) < 10;
}

// The 8-point Gauss sum over [m - h, m + h] of a B-spline code by symmetric
// node pairs, as the length walk's panels take theirs: b, the interval's
// speed coefficients, is shifted in place to m (b[j] = p^(j)(m) / j!), then
// pair k evaluates the even and odd parts at X = h x_k and returns
// w_k (f(m - X) + f(m + X)) into the sum (the caller scales it by h).  For
// degree 5 in 3D that is 30 float-float multiply-adds of shift plus 4 pairs
// instead of 8 Horner evaluations of 12.
template <int C>
__device__ __forceinline__ ff gl8_pairs(ff* b, ff m, ff h)
{
    constexpr int P = code_degree(C), D = code_dim(C);
#pragma unroll
    for (int i = 0; i < P - 1; ++i)
#pragma unroll
        for (int j = P - 2; j >= i; --j)
#pragma unroll
            for (int d = 0; d < D; ++d) b[j * D + d] = ff_fma_open(b[(j + 1) * D + d], m, b[j * D + d]);
    // pairs (0, 1) and (2, 3) in packed lanes
    const ff2 h2 = splat(h);
    ff2 I2{};
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
        const ff2 X = ff2_mul(h2, pack(to_ff(split_const(gl8_x(k))), to_ff(split_const(gl8_x(k + 1)))));
        ff2 fm, fp;
        ff_node_pair2<P, D>(b, X, ff2_mul(X, X), fm, fp);
        I2 = ff2_fma(pack(to_ff(split_const(gl8_w(k))), to_ff(split_const(gl8_w(k + 1)))), ff2_add_open(fm, fp), I2);
    }
    return ff_add(lane0(I2), lane1(I2));
}

// The 8-point Gauss sum over [m - h, m + h] of an ellipse piece by symmetric
// node pairs: with sm, cm the sine and cosine at m, a pair's are sm cos(d) -+
// cm sin(d) for its small angle d, whose series needs six terms instead of the
// eleven of each node's own.
struct EllipseMid {
    ff sm, cm;
};
__device__ __forceinline__ ff gl8_ellipse(const ff* r, const EllipseMid& e, ff h)
{
    const ff2 A = splat(r[0]), B = splat(r[1]);
    const ff h8 = ff_scale(h, (float)ELLIPSE_PIECE_SCALE);
    ff I{0.0f, 0.0f};
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
        ff sd, cd;
        ff_sincospi_small(ff_mul(h8, ff{c_gl8_ff[4 + k].x, c_gl8_ff[4 + k].y}), sd, cd);
        const ff q = ff_mul_open(e.cm, sd);
        const ff2 s = ff2_add(splat(ff_mul_open(e.sm, cd)), pack(ff_neg(q), q));
        const ff2 f = ff2_sqrt_open(ff2_fma(A, ff2_mul_open(s, s), B));
        I = ff_fma(ff{c_gl8_ff[8 + k].x, c_gl8_ff[8 + k].y}, ff_add(lane0(f), lane1(f)), I);
    }
    return I;
}
// speed to FP32 accuracy and q = f f' at the offset x from the midpoint (the
// square of the speed in float-float: on a thin ellipse's tips it cancels)
// near: A, f^2, and the sine and cosine of the doubled angle there, for
// speed_slope_near
__device__ __forceinline__ float speed_slope_ellipse(const ff* r, const EllipseMid& e, ff x, float& q, float* near)
{
    ff sd, cd;
    ff_sincospi_small(ff_scale(x, (float)ELLIPSE_PIECE_SCALE), sd, cd);
    const ff s = ff_fma(e.cm, sd, ff_mul(e.sm, cd));
    const float c = fmaf(e.cm.hi, cd.hi, -e.sm.hi * sd.hi);
    q = (float)(PI * ELLIPSE_PIECE_SCALE) * r[0].hi * s.hi * c;
    near[0] = r[0].hi;
    near[1] = ff_fma(r[0], ff_mul(s, s), r[1]).hi;
    near[2] = 2.0f * s.hi * c;
    near[3] = 1.0f - 2.0f * s.hi * s.hi;
    return sqrtf(near[1]);
}
// the same at the distance x from there: A (sin^2(a + d) - sin^2 a) = A sin(2 a +
// d) sin d, all in FP32
__device__ __forceinline__ float speed_slope_near_ellipse(const float* near, float x, float& q)
{
    const float d = (float)(PI * ELLIPSE_PIECE_SCALE) * x, d2 = d * d;
    const float sd = d * fmaf(d2, fmaf(d2, 1.0f / 120.0f, -1.0f / 6.0f), 1.0f);
    const float vd = d2 * fmaf(d2, -1.0f / 24.0f, 0.5f);  // 1 - cos d
    const float s1 = near[2] + (near[3] * sd - near[2] * vd);  // sin(2 a + d)
    const float c1 = near[3] - (near[2] * sd + near[3] * vd);
    q = (float)(0.5 * PI * ELLIPSE_PIECE_SCALE) * near[0] * (s1 + (c1 * sd - s1 * vd));
    return sqrtf(fmaf(near[0] * s1, sd, near[1]));
}

// TAB: the coefficient table's element: float2 (float-float, mixed tables) or
// double (FP64 tables; lengths then come scaled by 2^-sexp, see k_sample_ff).
template <int C, typename TAB>
__device__ __forceinline__ long long ff_leaf_newton(const TAB* __restrict__ seg, int sexp, ff vaf, float dv, ff rl, ff dS,
                                                 float dvg, float eps_s, float eps_t, unsigned long long& newton)
{
    constexpr bool FROM64 = std::is_same<TAB, double>::value;
    constexpr bool PAIRS = sample_node_pairs(C);
    float blo = 0.0f, bhi = dv;
    ff w{dvg, 0.0f};
    float last = 0.0f;  // the converged Newton step
    for (int it = 0; it < NEWTON_MAXIT; ++it) {
        ++newton;
        ff r[MAX_COEF];
        // every iteration: the node-pair Gauss sum shifts r
        if constexpr (FROM64)
            EvalFF<C>::load(seg, r, sexp);
        else
            EvalFF<C>::load(seg, r);
        const bool from_left = w.hi <= 0.5f * dv;
        // [a0, a1] in local offsets: [0, w] or [w, dv]
        const ff a0 = from_left ? ff{0.0f, 0.0f} : w;
        const ff a1 = from_left ? w : ff{dv, 0.0f};
        const ff h2 = ff_scale(ff_add(a1, ff_neg(a0)), 0.5f);
        const ff m2 = ff_add(ff_add(vaf, a0), h2);
        ff I{0.0f, 0.0f};
        EllipseMid em;
        if constexpr (C == 0) {
            ff_sincospi(ff_add_f(ff_scale(m2, (float)ELLIPSE_PIECE_SCALE), r[2].hi), em.sm, em.cm);
            I = gl8_ellipse(r, em, h2);
        } else if constexpr (PAIRS) {
            I = gl8_pairs<C>(r, m2, h2);  // r now holds the coefficients about m2
        } else {
            // nodes -x_k and +x_k in packed lanes
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                const ff xk = ff_mul(h2, ff{c_gl8_ff[4 + k].x, c_gl8_ff[4 + k].y});
                const ff2 f = EvalFF<C>::speed2(r, pack(ff_add(m2, ff_neg(xk)), ff_add(m2, xk)));
                I = ff_fma(ff{c_gl8_ff[8 + k].x, c_gl8_ff[8 + k].y}, ff_add(lane0(f), lane1(f)), I);
            }
        }
        I = ff_mul(I, h2);
        // F = S(v) - target inside the leaf
        const ff F = from_left ? ff_add(I, ff_neg(rl)) : ff_add(ff_add(dS, ff_neg(I)), ff_neg(rl));
        const float Fh = F.hi + F.lo;
        if (Fh == 0.0f) break;
        if (Fh < 0.0f)
            blo = w.hi;
        else
            bhi = w.hi;
        // speed at w: after the node-pair sums from the midpoint m2, at the end
        // +-h2 of the summed side that is w
        float q0, f0, near_w[MAX_COEF];
        if constexpr (C == 0)
            f0 = speed_slope_ellipse(r, em, from_left ? h2 : ff_neg(h2), q0, near_w);
        else if constexpr (PAIRS)
            f0 = EvalFF<C>::speed_slope_f(r, from_left ? h2 : ff_neg(h2), q0, near_w);
        else
            f0 = EvalFF<C>::speed_slope_f(r, ff_add(vaf, w), q0, near_w);
        const float r0 = rcp_approx(f0), dn = Fh * r0;
        float step = dn;
        // the higher-order step only from a Newton point inside the closed
        // bracket (a step below one FP32 ulp of w leaves w.hi - dn == w.hi,
        // which must still converge); a Newton point outside it would take
        // f1 from the polynomial extrapolated past the leaf
        const float wn = w.hi - dn;
        if (wn >= blo && wn <= bhi) {
            // the speed at w - dn in FP32 from what is known at w
            float q1, f1;
            if constexpr (C == 0)
                f1 = speed_slope_near_ellipse(near_w, -dn, q1);
            else
                f1 = EvalFF<C>::speed_slope_near(near_w, -dn, q1);
            float d = 2.0f * Fh * rcp_approx(f0 + f1);
            const float r1 = rcp_approx(f1), s1 = q1 * r1, ds = s1 - q0 * r0;  // f'(w - dn), less f'(w)
            float res = dn * dn * (fabsf(ds) * (1.0f / 3.0f) + s1 * s1 * fabsf(dn) * 0.25f * r1);
            // at tight tolerances the FP32 rounding of the step itself counts:
            // the speeds and the quotients are good to a few 2^-24 of F (at most
            // 1.3e-7 was seen; with 3.5e-7 the errors at rtol 1e-11 came out a
            // tenth above the FP64 kernel's)
            const float noise = 5e-7f * fabsf(Fh);
            // FP64 tables at every tolerance: without it samples at rtol 1e-9 were
            // up to 1.4e-10 of the length off, where the FP64 kernel kept 1e-10
            bool ok = (!FROM64 && eps_t < eps_s ? res : res + noise) <= eps_s;
            // only where the speed changes little over the step: past a cusp E can be
            // small by accident
            if (!ok && fabsf(f1 - f0) + fabsf(ds * dn) <= 0.3f * f0) {
                // the speed half way; the length between w - dn and w less dn f0
                // by Simpson's rule, and the trapezoidal rule with end correction
                // less that; their errors are as -1 to 4
                float qm, fm;
                if constexpr (C == 0)
                    fm = speed_slope_near_ellipse(near_w, -0.5f * dn, qm);
                else
                    fm = EvalFF<C>::speed_slope_near(near_w, -0.5f * dn, qm);
                const float simpson = dn * (1.0f / 6.0f) * (4.0f * (fm - f0) + (f1 - f0));
                const float E = dn * (0.5f * (f1 - f0) + dn * (1.0f / 12.0f) * ds) - simpson;
                const float rest = fmaf(-dn, f0, Fh) - simpson - 0.2f * E;
                const float d0 = rest * r1;
                d = dn + fmaf(0.5f * s1 * r1, d0 * d0, d0);
                res = 0.2f * fabsf(E) + d0 * d0 * (0.5f * s1 * s1 * r1 * fabsf(d0) + (0.25f / 6.0f) * fabsf(ds));
                ok = res + noise <= eps_t && fabsf(d0) <= 0.25f * fabsf(dn);
            }
            const float wd = w.hi - d;
            if (ok && wd >= 0.0f && wd <= dv) {
                last = d;  // converged with this step
                break;
            }
            step = d;
        }
        const float ws = w.hi - step;
        if (ws > blo && ws < bhi)
            w = ff_add_f(w, -step);
        else
            w = ff{0.5f * (blo + bhi), 0.0f};  // safeguard (also NaN)
    }
    // the final update, exact in fixed point
    return fix_of_float(w.hi) + fix_of_float(w.lo) - fix_of_float(last);
}

// Mixed-precision sampling: table lookups and the target in FP64, the
// quintic-Hermite guess in FP32, Newton on the leaf in float-float
// (G8 partial integral on the shorter side, local to the leaf), and the
// final update of v exactly, in 64-bit fixed point.  Samples per lane stay 32
// apart: neighbours in neighbouring lanes share table lines and need the same
// number of Newton steps.  (Consecutive samples per lane, searched for from the
// last one's interval: 14.5 ms against 11.9 on 50,000 spatial curves; lanes that
// take their next sample while others iterate: 14.9.)
// Registers per thread are capped (blocks of up to SAMPLE_THREADS_MAX threads
// still fit) at 64, 8 blocks of 128 threads per SM, at the price of spills: the
// kernel waits on fixed latencies and table loads more than on any
// pipe.  Sampling of the uneven batch of 100,000 curves took 11.76 ms at 80
// registers, 11.40 at 72, 11.24 at 64; unnormalised inner steps (gcv_ff.cuh)
// were worth 0.47 ms of it.
constexpr int SAMPLE_FF_REGS = 64;
static_assert(SAMPLE_FF_REGS * SAMPLE_THREADS_MAX <= 65536, "a block of SAMPLE_THREADS_MAX must fit one SM");
// residual, of the curve's length, that counts as an iterate's (at most eps_frac)
constexpr float SAMPLE_TIGHT = 4e-11f;
//
// TAB = double runs the same kernel on an FP64 table (GCV_PLAIN_FP64 at
// tolerances down to PLAIN_SPLIT_RTOL).  What it computes in float-float is
// the offset inside one leaf: the sums over a curve, the target and the
// parameter stay FP64, so a float-float rounding (2^-45) enters a sample's
// position only times the leaf's share of the curve, below FP64's own
// rounding of the target on curves of some tens of leaves and at most 2.8e-14
// of the curve's length otherwise, far under the stopping threshold
// SAMPLE_EPS_FRAC * rtol * L >= 1e-13 L.  Lengths inside the leaf are scaled by
// 2^-sexp, the binary exponent of its mean speed, so that curves of any
// double magnitude fit FP32's exponent range.  The FP64 kernel was bound by
// the FP64 pipe (91 % busy, one warp instruction per 64 issue slots); this one
// by issue.  4,096 ellipses x 1,000 samples: 4.15 -> 0.42 ms; 10,000 planar
// cubics x 1,024: 8.51 -> 0.80 ms.  Position errors at rtol 1e-10 .. 1e-12 on
// ellipses, cubics and an uneven batch, rms and worst, are at or below the FP64
// kernel's: the extra term of its stopping test makes it iterate further.
template <int CODE, typename TAB>
__global__ void __maxnreg__(SAMPLE_FF_REGS) k_sample_ff(SampleParams P, const TAB* __restrict__ coef)
{
    constexpr bool FROM64 = std::is_same<TAB, double>::value;
    const Batch& b = P.b;
    const Table& t = P.t;
    unsigned long long newton = 0;
    int64_t i0, i1;
    sample_range(P, i0, i1);
    // each warp takes runs of up to SAMPLE_RUN consecutive samples, 32 at a
    // time: a lane's samples then mostly share their curve (see CurveHint).
    // Small launches shorten the runs to 32 so that no lane places 8 samples
    // one after another while most of the GPU idles (6,400 ellipse samples:
    // 120 us with runs of 256, 34 us with 32; the uneven batch of 301 curves,
    // nine launches: 750 us and 185 us)
    const int64_t per = (i1 - i0) / P.min_runs & ~(int64_t)31;
    const int run_len = per >= SAMPLE_RUN ? SAMPLE_RUN : (per < 32 ? 32 : (int)per);
    const float tight = fminf(1.0f, SAMPLE_TIGHT / P.eps_frac);
    CurveHint hint;
    const int lane = threadIdx.x & 31;
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t run = i0 + wid * run_len; run < i1; run += n_warps * run_len)
    for (int64_t ii = run + lane; ii < run + run_len && ii < i1; ii += 32) {
        int64_t i;
        const int c = sample_curve_hint(P, ii, i, hint);
        const int s0 = (int)b.seg_off[c], s1 = (int)b.seg_off[c + 1];
        int s;
        long long v;  // local parameter, fixed point
        if (s1 == s0) {
            s = -1;
            v = -FIX_ONE;
        } else {
            const double L = t.curve_len[c];
            const double pos = P.pos[i];
            const double target = P.is_relative ? pos * L : pos;
            // target <= 0 / target >= L on the bit patterns (L >= 0; a negative
            // target has a negative pattern): integer compares, off the FP64 pipe
            const long long tb = __double_as_longlong(target), lb = __double_as_longlong(L);
            // (FP64 tables: a NaN target is the curve's start, as !(target > 0) in k_sample)
            if (tb <= 0 || (FROM64 && tb > 0x7FF0000000000000ll)) {
                s = s0;
                v = -FIX_ONE;
            } else if (tb >= lb && (!FROM64 || lb >= 0)) {  // (a NaN length with its sign bit set is no end)
                s = s1 - 1;
                v = FIX_ONE;
            } else {
                s = s0 + lower_bound_key32(t.seg_cum + s0, s1 - s0, dkey(target));
                if (s == s1) s = s1 - 1;
                const double prev = s > s0 ? t.seg_cum[s - 1] : 0.0;
                const double rr = target - prev;
                const int64_t lo = t.leaf_off[s];
                const int cnt = t.leaf_cnt[s];
                int j = lower_bound_key32(t.leaf_cum + lo, cnt, dkey(rr));
                if (j >= cnt) j = cnt - 1;
                double base = 0.0, va = -1.0;
                float fa, qa;
                if (j) {
                    base = t.leaf_cum[lo + j - 1];
                    va = t.leaf_v[lo + j - 1];
                    fa = t.leaf_f[lo + j - 1];
                    qa = t.leaf_q[lo + j - 1];
                } else {  // the interval's start: its end values, by their bits
                    fa = f32_of_f64_trunc(t.seg_f0[s]);
                    qa = f32_of_f64_trunc(t.seg_q0[s]);
                }
                const double vb = t.leaf_v[lo + j];
                const double cb = t.leaf_cum[lo + j];
                float fb = t.leaf_f[lo + j];
                float qb = t.leaf_q[lo + j];
                const double rd = rr - base, dSd = cb - base;  // target inside the leaf, leaf length
                const long long vfix = fix_of_double(va), dfix = fix_of_double(vb) - vfix;
                const int dexp = 3 - __clzll(dfix);             // leaf width 2^dexp
                int sexp = 0;
                ff rl, dS;
                if constexpr (FROM64) {
                    sexp = exponent_of(dSd) - dexp;
                    rl = ff_from_double_scaled(rd, sexp);
                    dS = ff_from_double_scaled(dSd, sexp);
                    fa = scale_down(fa, sexp);
                    fb = scale_down(fb, sexp);
                    qa = scale_down(qa, 2 * sexp);
                    qb = scale_down(qb, 2 * sexp);
                } else {
                    rl = ff_from_double(rd);
                    dS = ff_from_double(dSd);
                }
                const float dv = __int_as_float((dexp + 127) << 23);
                const ff vaf = ff_from_double(va);
                // quintic Hermite guess of v(S) on the leaf (FP32)
                float sig = dS.hi > 0.0f ? rl.hi * rcp_approx(dS.hi) : 0.0f;
                sig = fminf(fmaxf(sig, 0.0f), 1.0f);
                float dvg = sig * dv;
                const float fm = dS.hi * rcp_approx(dv);
                if (fa > 0.1f * fm && fb > 0.1f * fm) {
                    const float s2 = sig * sig, s3 = s2 * sig, s4 = s3 * sig, s5 = s4 * sig;
                    const float h5 = 10.0f * s3 - 15.0f * s4 + 6.0f * s5;
                    const float h1 = sig - 6.0f * s3 + 8.0f * s4 - 3.0f * s5;
                    const float h4 = -4.0f * s3 + 7.0f * s4 - 3.0f * s5;
                    const float h2 = 0.5f * (s2 - 3.0f * s3 + 3.0f * s4 - s5);
                    const float h3 = 0.5f * (s3 - 2.0f * s4 + s5);
                    const float ia = rcp_approx(fa), ib = rcp_approx(fb);
                    const float ka = -qa * (ia * ia) * (ia * ia), kb = -qb * (ib * ib) * (ib * ib);
                    dvg = h5 * dv + dS.hi * (h1 * ia + h4 * ib) + dS.hi * dS.hi * (h2 * ka + h3 * kb);
                    dvg = fminf(fmaxf(dvg, 0.0f), dv);
                }
                const TAB* seg = coef + b.coef_off[c] + (int64_t)(s - s0) * code_stride(CODE);
                const float Ls = FROM64 ? ff_from_double_scaled(L, sexp).hi : f32_of_f64_trunc(L);
                const float eps_s = P.eps_frac * (Ls == Ls ? Ls : dS.hi);
                const long long w = ff_leaf_newton<CODE>(seg, sexp, vaf, dv, rl, dS, dvg, eps_s, tight * eps_s, newton);
                v = vfix + (w < 0 ? 0 : w > dfix ? dfix : w);
            }
        }
        if (P.what == 2) {
            double u;
            if (s < 0) {
                u = b.kind[c] == 0 ? 0.0 : b.knots[b.knot_off[c] + b.degree[c]];
            } else {
                // (v + 1) hw + t0 up to v = 0, (v - 1) hw + t1 above: exact at
                // both ends, the operands chosen so that one side is evaluated
                const double t0 = t.seg_t0[s], t1 = t.seg_t1[s];
                const bool low = v <= 0;
                u = fma(double_of_fix(v + (low ? FIX_ONE : -FIX_ONE)), 0.5 * (t1 - t0), low ? t0 : t1);
            }
            P.out[i] = u;
        } else {
            double p3[3] = {0.0, 0.0, 0.0};
            if (s >= 0) {
                const TAB* seg = coef + b.coef_off[c] + (int64_t)(s - s0) * code_stride(CODE);
                const double vd = double_of_fix(v);
                double cd[MAX_COEF];
                const double* pc = cd;
                if constexpr (FROM64) {
                    pc = seg;
                } else {
                    // points from the float-float coefficients, evaluated in FP64
                    // (a B-spline stores a[0] and then b[k - 1] = k a[k])
                    constexpr int n = code_stride(CODE), dim = code_dim(CODE);
#pragma unroll
                    for (int k = 0; k < n; ++k) {
                        cd[k] = (double)seg[k].x + (double)seg[k].y;
                        if (CODE != 0 && k >= 2 * dim) cd[k] *= 1.0 / (double)(k / dim);
                    }
                }
                Eval<CODE>::point(pc, vd, p3);
            }
            for (int k = 0; k < P.pdim; ++k) P.out[i * P.pdim + k] = p3[k];
        }
    }
    if (P.collect) {
        for (int o = 16; o > 0; o >>= 1) newton += __shfl_xor_sync(0xffffffffu, newton, o);
        if ((threadIdx.x & 31) == 0 && newton) atomicAdd(t.ctr + C_NEWTON, newton);
    }
}

}  // namespace gcv
