// Set-up of a B-spline knot interval: the power-basis coefficients in the local
// variable v of the piece on knot span `span` (k[span] < k[span + 1]), u = m +
// w v with m the span's midpoint and w its half width.  The reference runs its
// basis recursion at every evaluated point (samples/sample2_bspline/BSpline.h:26-96,
// b_spline_func_value / b_spline_derv_o1 / to_point); here each interval is
// expanded once.
//
// The derivative's control points over the knots, Q_j = (P_{j+1} - P_j) /
// (t_{j+P} - t_j), are values of its polar form g at P - 1 consecutive knots.  Two
// of them that share all knots but one, t_lo and t_hi, give
//   g(m, ..) by interpolation   T_j + (m - t_lo) / (t_hi - t_lo) (T_{j+1} - T_j)
//   g(1, ..) by difference      (T_{j+1} - T_j) / (t_hi - t_lo)
// and the coefficient of (u - m)^l is binomial(P - 1, l) g(m^(P-1-l), 1^l).  The
// values needed, l = 0 .. P - 1, share most of their steps (polar_tree), and both
// kinds of step share the difference.  The position at m follows from the same
// interpolated values: replacing the knots of P_0 by m one after another,
//   C(m) = P_0 + sum_r (m - t_r) g(m^r, t_{r+2} ..).
// g is carried times w and (m - t_r) over w, so that nothing has the units of a
// control point over a knot: with Q_j itself, knots in units of 1e-30 under
// coordinates of 1e9 overflowed in float-float.
// For degree 5 in 3D that is about 3,200 instructions in float-float, against
// 5,600 of the basis recursion on polynomials it replaces (whose code also missed
// the instruction cache); planar cubics take about 95 instead of 190 FP64
// instructions.  Measured before and now: 50,000
// spatial quintics in float-float 1.29 -> 1.02 ms, the uneven batch of 301,000 curves
// 7.42 -> 5.52 ms (coefficient stores included), 10,000 planar cubics in FP64
// 193 -> 140 us; the FP64 lengths' largest relative error fell from 6.1e-13 to 2.7e-15
// (uneven batch, rtol 1e-11).
#pragma once

#include "gcv_ff.cuh"
#include "gcv_table.cuh"

namespace gcv {

__device__ __forceinline__ double n_add(double a, double b) { return a + b; }
__device__ __forceinline__ double n_sub(double a, double b) { return a - b; }
__device__ __forceinline__ double n_mul(double a, double b) { return a * b; }
__device__ __forceinline__ double n_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double n_times(double a, int k) { return a * (double)k; }
__device__ __forceinline__ ff n_add(ff a, ff b) { return ff_add(a, b); }
__device__ __forceinline__ ff n_sub(ff a, ff b) { return ff_add(a, ff_neg(b)); }
__device__ __forceinline__ ff n_mul(ff a, ff b) { return ff_mul(a, b); }
__device__ __forceinline__ ff n_fma(ff a, ff b, ff c) { return ff_fma(a, b, c); }
__device__ __forceinline__ ff n_times(ff a, int k) { return ff_mul_f(a, (float)k); }
__device__ __forceinline__ void n_from(double x, double& y) { y = x; }
__device__ __forceinline__ void n_from(double x, ff& y) { y = ff_from_double(x); }
__device__ __forceinline__ ff n_recip(ff x) { return ff_recip(x); }
// 1 / x, x > 0, to a unit in the last place: FP32 reciprocal of the
// significand, two Newton steps in FP64 (four FP64 instructions)
__device__ __forceinline__ double n_recip(double x)
{
    const int hi = __double2hiint(x), raw = (hi >> 20) & 0x7FF;
    if (raw < 2 || raw > 2044) return 1.0 / x;
    const double s = __hiloint2double((hi & 0xFFFFF) | 0x3FF00000, __double2loint(x));  // [1, 2)
    const float f = __int_as_float(0x3F800000 | ((hi & 0xFFFFF) << 3) | (int)((unsigned)__double2loint(x) >> 29));
    const int b = __float_as_int(__fdividef(1.0f, f));
    double y = __longlong_as_double(((long long)b << 29) + (896ll << 52));
    y = fma(y, fma(-s, y, 1.0), y);
    y = fma(y, fma(-s, y, 1.0), y);
    return __hiloint2double(__double2hiint(y) + ((1023 - raw) << 20), __double2loint(y));
}

__host__ __device__ constexpr int binomial(int n, int k)
{
    int b = 1;
    for (int i = 0; i < k; ++i) b = b * (n - i) / (i + 1);
    return b;
}

// What the steps need of the knots, relative to the midpoint.
template <int P, typename T>
struct SpanKnots {
    static constexpr int N = P - 1;
    T w;                     // half width
    T t[2 * P];              // knots span - P + 1 .. span + P
    T rq[P];                 // w / (t[j + P] - t[j]): w times the derivative's control points
    T tw[P > 1 ? P - 1 : 1];  // (m - t[r]) / w; 1 for r = P - 1
    T alpha[N * P / 2 + 1];  // step s, pair j: (m - t_lo) / (t_hi - t_lo)
    T beta[N * P / 2 + 1];   // w / (t_hi - t_lo)
    // pairs of the steps before s (step s has N - s)
    __host__ __device__ static constexpr int first(int s) { return s * N - s * (s - 1) / 2; }

    // width = k[span + 1] - k[span] > 0
    __device__ __forceinline__ void set(const double* __restrict__ kv, int span, double width)
    {
        n_from(width, w);
        w = half(w);
        // each knot by its distance from the nearer end of the span: no
        // cancellation against the midpoint
#pragma unroll
        for (int i = 0; i < 2 * P; ++i) {
            if (i == P - 1) {
                t[i] = neg(w);
            } else if (i == P) {
                t[i] = w;
            } else {
                T d;
                n_from(kv[span - P + 1 + i] - kv[i < P ? span : span + 1], d);
                t[i] = i < P ? n_sub(d, w) : n_add(d, w);
            }
        }
#pragma unroll
        for (int j = 0; j < P; ++j) rq[j] = n_mul(w, n_recip(n_sub(t[j + P], t[j])));
        if constexpr (P > 1) {
            const T rw = n_recip(w);
#pragma unroll
            for (int r = 0; r < P - 1; ++r) tw[r] = n_mul(neg(t[r]), rw);
        }
#pragma unroll
        for (int s = 0; s < N; ++s)
#pragma unroll
            for (int j = 0; j < N - s; ++j) {
                const T lo = t[j + 1 + s], r = n_recip(n_sub(t[j + P], lo));
                alpha[first(s) + j] = n_mul(neg(lo), r);
                beta[first(s) + j] = n_mul(w, r);
            }
    }
    __device__ __forceinline__ static double neg(double a) { return -a; }
    __device__ __forceinline__ static ff neg(ff a) { return ff_neg(a); }
    __device__ __forceinline__ static double half(double a) { return 0.5 * a; }
    __device__ __forceinline__ static ff half(ff a) { return ff_scale(a, 0.5f); }
};

// step s from its N - s + 1 values: interpolated, differences (times w), or both
template <int S, int P, typename T>
__device__ __forceinline__ void polar_lerp(const SpanKnots<P, T>& k, const T* in, T* out)
{
#pragma unroll
    for (int j = 0; j < P - 1 - S; ++j) out[j] = n_fma(k.alpha[k.first(S) + j], n_sub(in[j + 1], in[j]), in[j]);
}
template <int S, int P, typename T>
__device__ __forceinline__ void polar_diff(const SpanKnots<P, T>& k, const T* in, T* out)
{
#pragma unroll
    for (int j = 0; j < P - 1 - S; ++j) out[j] = n_mul(k.beta[k.first(S) + j], n_sub(in[j + 1], in[j]));
}
template <int S, int P, typename T>
__device__ __forceinline__ void polar_both(const SpanKnots<P, T>& k, const T* in, T* lerp, T* diff)
{
#pragma unroll
    for (int j = 0; j < P - 1 - S; ++j) {
        const T d = n_sub(in[j + 1], in[j]);
        lerp[j] = n_fma(k.alpha[k.first(S) + j], d, in[j]);
        diff[j] = n_mul(k.beta[k.first(S) + j], d);
    }
}

// q: the P control points times w; out[l] = w g(m^(N-l), w^l); lead[r] = w g(m^r, t_{r+2} ..), the
// first of the values interpolated r times
template <int P, typename T>
__device__ __forceinline__ void polar_tree(const SpanKnots<P, T>& k, const T* q, T* out, T* lead)
{
    constexpr int N = P - 1;
    lead[0] = q[0];
    if constexpr (N == 0) {
        out[0] = q[0];
    } else if constexpr (N == 1) {
        polar_both<0, P>(k, q, out, out + 1);
    } else {
        T a[N], b[N];  // one interpolation; one difference
        polar_both<0, P>(k, q, a, b);
        lead[1] = a[0];
        if constexpr (N == 2) {
            polar_both<1, P>(k, a, out, out + 1);
            polar_diff<1, P>(k, b, out + 2);
        } else {
            T c[N - 1], e[N - 1];  // two interpolations; two differences
            polar_lerp<1, P>(k, a, c);
            polar_diff<1, P>(k, b, e);
            lead[2] = c[0];
            if constexpr (N == 3) {
                polar_both<2, P>(k, c, out, out + 1);
                polar_both<2, P>(k, e, out + 2, out + 3);
            } else {
                T f[N - 2], h[N - 2], i[N - 2];  // three; one and two; three differences
                polar_lerp<2, P>(k, c, f);
                polar_both<2, P>(k, e, h, i);
                lead[3] = f[0];
                polar_both<3, P>(k, f, out, out + 1);
                polar_both<3, P>(k, h, out + 2, out + 3);
                polar_diff<3, P>(k, i, out + 4);
            }
        }
    }
    lead[N] = out[0];
}

// one dimension: the position at the midpoint, less P_0, and the tree's values
template <int P, int D, typename T>
__device__ __forceinline__ T expand_dim(const SpanKnots<P, T>& k, const double* __restrict__ c0, int d, T* out)
{
    T q[P], lead[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
        n_from(c0[(j + 1) * D + d] - c0[j * D + d], q[j]);
        q[j] = n_mul(q[j], k.rq[j]);
    }
    polar_tree<P>(k, q, out, lead);
    T a = lead[P - 1];
#pragma unroll
    for (int r = 0; r < P - 1; ++r) a = n_fma(k.tw[r], lead[r], a);
    return a;
}

// FP64 table: the position polynomial a[k][d], k = 0 .. P; dC/dv is b[k][d] =
// (k + 1) a[k + 1][d] (Eval::load_speed)
template <int P, int D>
__device__ __forceinline__ void bspline_setup(const double* __restrict__ kv, const double* __restrict__ cp, int span,
                                              double* out)
{
    SpanKnots<P, double> k;
    k.set(kv, span, kv[span + 1] - kv[span]);
    const double* c0 = cp + (size_t)(span - P) * D;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        double g[P];
        out[d] = c0[d] + expand_dim<P, D>(k, c0, d, g);
#pragma unroll
        for (int l = 0; l < P; ++l) out[(l + 1) * D + d] = n_times(g[l], binomial(P, l + 1));
    }
}

// Mixed table: the position at the midpoint (it only enters points), then the
// derivative's coefficients b[k][d], which the walk and the sampler read
// without rescaling.  FP64 only centres the data (differences of knots and of
// control points, which carry the cancellation), each converted once.
template <int P, int D>
__device__ __forceinline__ void bspline_setup_ff(const double* __restrict__ kv, const double* __restrict__ cp, int span,
                                                 double width, float2* out)
{
    SpanKnots<P, ff> k;
    k.set(kv, span, width);
    const double* c0 = cp + (size_t)(span - P) * D;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        ff g[P];
        const ff a = ff_add(ff_from_double(c0[d]), expand_dim<P, D>(k, c0, d, g));
        out[d] = make_float2(a.hi, a.lo);
#pragma unroll
        for (int l = 0; l < P; ++l) {
            const ff b = n_times(g[l], P * binomial(P - 1, l));
            out[(l + 1) * D + d] = make_float2(b.hi, b.lo);
        }
    }
}

}  // namespace gcv
