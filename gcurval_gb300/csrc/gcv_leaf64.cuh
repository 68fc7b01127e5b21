// K15 of one accepted panel of an FP64 table with as few FP64 instructions as
// its accuracy allows (leaf_k15).
//
// The FP64 pipe takes one warp instruction per 64 issue slots, so FP64 is
// kept for what carries the result's accuracy:
//   * B-splines: the speed polynomials shifted to the panel's midpoint and
//     scaled to it, their squared norm as one polynomial q in x on [-1, 1],
//     and its even and odd parts, E(x^2) -+ x O(x^2), shared by each Kronrod
//     pair: 2 P - 1 multiply-adds a pair instead of two Horner evaluations per
//     dimension;
//   * ellipses: angle addition from one sine and cosine (AngleTable);
//   * square roots (kronrod_root): the root S to ~44 bits on the FP32 and
//     integer pipes, one FP64 residual x - S^2, its correction
//     (x - S^2) / 2 S summed in FP32 beside the FP64 sum of w S.  Two FP64
//     instructions per node, the sum good to FP64 rounding.
// A planar cubic's panel takes about 90 FP64 instructions, against about 300 of
// panel_k15; an ellipse's about 145 against about 650.
//
// The polynomial q is good to a rounding of its largest coefficients, so where the
// speed at a node is a small part of the panel's largest (LEAF_LOW) its root is
// not: next to a zero of even order, whose speeds are smooth and whose panel is
// accepted whole, lengths were off by up to 4e-10.  Such panels are summed once more
// by leaf_k15_nodes, from the speeds' components (none of the 44,000 leaves of random
// planar and spatial cubics and uneven curves).
#pragma once

#include "gcv_ff_eval.cuh"

namespace gcv {

// the seven positive Kronrod nodes, their squares and weights
static __constant__ double c_gk_x[7] = {gk_x(0), gk_x(1), gk_x(2), gk_x(3), gk_x(4), gk_x(5), gk_x(6)};
static __constant__ double c_gk_z[7] = {gk_x(0) * gk_x(0), gk_x(1) * gk_x(1), gk_x(2) * gk_x(2), gk_x(3) * gk_x(3),
                                        gk_x(4) * gk_x(4), gk_x(5) * gk_x(5), gk_x(6) * gk_x(6)};
static __constant__ double c_gk_w[7] = {gk_wk(0), gk_wk(1), gk_wk(2), gk_wk(3), gk_wk(4), gk_wk(5), gk_wk(6)};
static __constant__ float c_gk_wf[7] = {(float)gk_wk(0), (float)gk_wk(1), (float)gk_wk(2), (float)gk_wk(3),
                                        (float)gk_wk(4), (float)gk_wk(5), (float)gk_wk(6)};

// x 2^-s for any s by the exponent bits (0 below the normal range)
__device__ __forceinline__ double scale_exp(double x, int s)
{
    const int hi = __double2hiint(x), raw = (hi >> 20) & 0x7FF, e = raw - s;
    if (raw == 0x7FF) return x;
    if (raw == 0 || e <= 0) return 0.0;
    if (e >= 0x7FF) return __hiloint2double((hi & 0x80000000) | 0x7FF00000, 0);
    return __hiloint2double(hi - (s << 20), __double2loint(x));
}

// S ~ sqrt(x) to ~44 bits, and corr += wf (x - S^2) / 2 S: S from a FP32 root
// s0 of x's leading 24 bits and one FP32 Newton correction c that sees the
// next 24, put together as a double's bit pattern (s0's bits plus c as an
// integer in units of its last place).  x below 2^-70 of the interval's scale
// (its square root below 2^-35, where x is rounding) or negative counts as 0.
__device__ __forceinline__ double kronrod_root(double x, float wf, float& corr)
{
    const int hx = __double2hiint(x);
    const unsigned lx = (unsigned)__double2loint(x);
    const bool live = hx >= (1023 - 70) << 20;
    const float xh = __int_as_float(((hx - (896 << 20)) << 3) | (int)(lx >> 29));
    const int e = (hx >> 20) - 1023;
    const float xl = __uint2float_rn(lx & 0x1FFFFFFFu) * __int_as_float((e - 52 + 127) << 23);
    const float y = rsqrtf(xh), s0 = xh * y, hy = 0.5f * y;
    const float c = (fmaf(-s0, s0, xh) + xl) * hy;
    // c in units of 2^-51 of s0's binade (at most 2^31 / 2), then of 2^-52
    const int b0 = __float_as_int(s0), e0 = (b0 >> 23) - 127;
    const int ci = __float2int_rn(c * __int_as_float((51 - e0 + 127) << 23));
    const long long bits = (((long long)b0 << 29) + (896ll << 52)) + ((long long)ci << 1);
    const double S = live ? __longlong_as_double(bits) : 0.0;
    const double r = fma(-S, S, x);
    // the residual as a float by its bit pattern (0 below 2^-126)
    const int hr = __double2hiint(r), er = (hr >> 20) & 0x7FF;
    const float rf = er > 897 ? __int_as_float((hr & 0x80000000) | (((hr & 0x7FFFFFFF) - (896 << 20)) << 3) |
                                               (int)((unsigned)__double2loint(r) >> 29))
                              : 0.0f;
    corr = live ? fmaf(wf * hy, rf, corr) : corr;
    return S;
}
// the Kronrod pair i with squared speeds x0, x1; low: the smallest one's leading bits
__device__ __forceinline__ void kronrod_pair(double x0, double x1, int i, double& acc, float& corr, int& low)
{
    const float wf = c_gk_wf[i];
    low = min(low, min(__double2hiint(x0), __double2hiint(x1)));
    const double S0 = kronrod_root(x0, wf, corr), S1 = kronrod_root(x1, wf, corr);
    acc = fma(c_gk_w[i], S0 + S1, acc);
}

// A squared speed below 2^-LEAF_LOW of q's largest coefficient (or below
// kronrod_root's range) is taken from its components.  Above it q's rounding
// moves a speed by at most 2^(LEAF_LOW / 2 - 1) units of q's, and a node's weight is a
// fifth of the panel or less: a few units of the panel's sum.
constexpr int LEAF_LOW = 8;

// seg: the interval's FP64 table entry; sexp: the binary exponent that brings
// its speeds near 1; panel (k, depth).  The integral over the panel of v;
// `again`: leaf_k15_nodes has to give it.
template <int CODE>
__device__ __forceinline__ double leaf_k15(const double* __restrict__ seg, int sexp, unsigned long long k, int depth,
                                           bool& again)
{
    const double hw = pow2_neg(depth);
    const double mid = fma(__ull2double_rn(k), 2.0 * hw, -1.0) + hw;
    double acc = 0.0, centre;
    float corr = 0.0f;
    int low = 0x7FFFFFFF;
    again = false;
    if constexpr (CODE == 0) {
        double A = seg[0], B = seg[1], sm, cm;
        int sA = 2 * sexp, sB = 2 * sexp;
        lift_denormal(A, sA);
        lift_denormal(B, sB);
        A = scale_exp(A, sA);
        B = scale_exp(B, sB);
        sincospi(fma(mid, ELLIPSE_PIECE_SCALE, seg[2]), &sm, &cm);
        // the pair's rounding enters all 15 nodes alike: its length error is
        // taken back through A (its angle error shifts the panel's nodes
        // by 1e-16, which leaves the integral)
        A = fma(A, fma(-cm, cm, fma(-sm, sm, 1.0)), A);
        const double(*tab)[2] = c_angle.sc[depth];
#pragma unroll 1
        for (int i = 0; i < 7; ++i) {
            const double sd = __ldg(&tab[i][0]), p = fma(-sm, __ldg(&tab[i][1]), sm);
            const double up = fma(cm, sd, p), dn = fma(-cm, sd, p);
            kronrod_pair(fma(A * up, up, B), fma(A * dn, dn, B), i, acc, corr, low);
        }
        centre = fma(A * sm, sm, B);
    } else {
        constexpr int P = code_degree(CODE), D = code_dim(CODE), N = P - 1;
        double q[2 * N + 1];
#pragma unroll
        for (int d = 0; d < D; ++d) {
            // derivative polynomial (k + 1) a[k + 1], shifted to the midpoint
            double b[P];
#pragma unroll
            for (int j = 0; j < P; ++j) {
                b[j] = scale_exp(seg[(j + 1) * D + d], sexp - (j == 1 ? 1 : j == 3 ? 2 : 0));
                if (j == 2 || j == 4) b[j] *= double(j + 1);
            }
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = N - 1; j >= i; --j) b[j] = fma(b[j + 1], mid, b[j]);
#pragma unroll
            for (int j = 1; j < P; ++j) b[j] = scale_exp(b[j], j * depth);
            // its square, added to the others'
#pragma unroll
            for (int m = 0; m <= 2 * N; ++m) {
                double s = 0.0;
                bool any = false;
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    const int j = m - i;
                    if (j > i && j < P) {
                        s = any ? fma(b[i], b[j], s) : b[i] * b[j];
                        any = true;
                    }
                }
                double v = any ? scale_exp(s, -1) : 0.0;
                if (m % 2 == 0) v = any ? fma(b[m / 2], b[m / 2], v) : b[m / 2] * b[m / 2];
                q[m] = d == 0 ? v : q[m] + v;
            }
        }
#pragma unroll(P <= 3 ? 7 : 1)
        for (int i = 0; i < 7; ++i) {
            const double x = c_gk_x[i], z = c_gk_z[i];
            double E = q[2 * N], O = 0.0;
#pragma unroll
            for (int m = 2 * N - 2; m >= 0; m -= 2) E = fma(E, z, q[m]);
            if constexpr (N > 0) {
                O = q[2 * N - 1];
#pragma unroll
                for (int m = 2 * N - 3; m >= 1; m -= 2) O = fma(O, z, q[m]);
            }
            kronrod_pair(N > 0 ? fma(x, O, E) : E, N > 0 ? fma(-x, O, E) : E, i, acc, corr, low);
        }
        centre = q[0];
        int top = 0;
#pragma unroll
        for (int m = 0; m <= 2 * N; ++m) top = max(top, __double2hiint(q[m]) & 0x7FFFFFFF);
        low = min(low, __double2hiint(centre));
        again = top != 0 && low < max(top - (LEAF_LOW << 20), (1023 - 70) << 20);
    }
    acc = fma(gk_wk(7), kronrod_root(centre, (float)gk_wk(7), corr), acc);
    return scale_exp((acc + (double)corr) * hw, -sexp);
}

// The same panel of a B-spline piece by 16 lanes, one node each (the centre twice,
// with half its weight), every speed from its components in FP64 throughout: its
// error is a rounding of the interval's largest speed.  Every lane of the warp takes
// part; the result is the same in the 16.
template <int CODE>
__device__ __noinline__ double leaf_k15_nodes(const double* __restrict__ seg, int sexp, unsigned long long k, int depth)
{
    constexpr int P = code_degree(CODE), D = code_dim(CODE);
    const int i = threadIdx.x & 7;
    const double hw = pow2_neg(depth), x = i < 7 ? c_gk_x[i] : 0.0, w = i < 7 ? c_gk_w[i] : 0.5 * gk_wk(7);
    const double v = fma(threadIdx.x & 8 ? hw : -hw, x, fma(__ull2double_rn(k), 2.0 * hw, -1.0) + hw);
    double s = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        double p = scale_exp(seg[P * D + d], sexp) * double(P);
#pragma unroll
        for (int j = P - 2; j >= 0; --j) p = fma(p, v, scale_exp(seg[(j + 1) * D + d], sexp) * double(j + 1));
        s = fma(p, p, s);
    }
    double f = w * sqrt(s);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
    return scale_exp(f * hw, -sexp);
}

}  // namespace gcv
