// Float-float evaluators of the mixed-precision path: curve speeds in
// float-float arithmetic (gcv_ff.cuh), an own float-float sin(pi x) for
// ellipses, and the 15-node Kronrod panel built from them.
#pragma once

#include "gcv_ff.cuh"
#include "gcv_ff2.cuh"
#include "gcv_table.cuh"

namespace gcv {

// float-float constants from double literals (split at compile time)
struct ffc {
    float hi, lo;
};
__host__ __device__ constexpr ffc split_const(double x)
{
    return ffc{(float)x, (float)(x - (double)(float)x)};
}
__device__ __forceinline__ ff to_ff(ffc c) { return ff{c.hi, c.lo}; }

// sin(pi x) and cos(pi x) for small x by their Taylor series, at compile time
__host__ __device__ constexpr double series_sinpi(double x)
{
    double t = PI * x, s = 0.0;
    for (int k = 1; t > 1e-40 || t < -1e-40; k += 2) {
        s += t;
        t *= -(PI * x) * (PI * x) / ((k + 1) * (k + 2));
    }
    return s;
}
__host__ __device__ constexpr double series_cospi(double x)
{
    double t = 1.0, s = 0.0;
    for (int k = 0; t > 1e-20 || t < -1e-20; k += 2) {
        s += t;
        t *= -(PI * x) * (PI * x) / ((k + 1) * (k + 2));
    }
    return s;
}

// Ellipse panels by angle addition: with w_m the panel's midpoint and d_i =
// 2^-depth x_i / ELLIPSE_PIECES the offset of the Kronrod pair i from it,
// sin(pi (w_m -+ d_i)) = sin(pi w_m) cos(pi d_i) -+ cos(pi w_m) sin(pi d_i).
// The offsets depend on the depth alone, so their sines and cosines are a
// table, and a panel evaluates one sine and cosine instead of fifteen.
// Order of the panels' node pairs: those of the Gauss rule first (1, 3, 5, and the
// centre, 7), then the Kronrod-only ones
__host__ __device__ constexpr int gk_pair(int j) { return j < 4 ? 2 * j + 1 : 2 * j - 8; }
__host__ __device__ constexpr double gk_pair_x(int j) { return gk_pair(j) < 7 ? gk_x(gk_pair(j)) : 0.0; }

constexpr int ANGLE_DEPTHS = 49;  // 0 .. MAX_DEPTH_LIMIT
struct alignas(16) AngleTable {
    double sc[ANGLE_DEPTHS][8][2];  // pair i: sin(pi d_i), 1 - cos(pi d_i); entry 7 is the centre
    float ff[ANGLE_DEPTHS][8][4];   // float-float sine and cosine of pair gk_pair(i): sin hi, lo, cos hi, lo
    __host__ __device__ constexpr AngleTable() : sc(), ff()
    {
        double h = ELLIPSE_PIECE_SCALE;
        for (int d = 0; d < ANGLE_DEPTHS; ++d, h *= 0.5)
            for (int i = 0; i < 8; ++i) {
                const double x = i < 7 ? h * gk_x(i) : 0.0, h2 = series_sinpi(0.5 * x);
                sc[d][i][0] = series_sinpi(x);
                sc[d][i][1] = 2.0 * h2 * h2;
                const double s = series_sinpi(h * gk_pair_x(i)), c = series_cospi(h * gk_pair_x(i));
                ff[d][i][0] = split_const(s).hi;
                ff[d][i][1] = split_const(s).lo;
                ff[d][i][2] = split_const(c).hi;
                ff[d][i][3] = split_const(c).lo;
            }
    }
};
static __device__ const AngleTable c_angle{};

// sin(pi u) and cos(pi u) for |u| <= 1/4 in the two lanes of one packed series
// in u^2 (nine terms: the next are below 1e-17 relative); the sine's lane
// is then multiplied by u
constexpr int SINCOS_TERMS = 9;
__host__ __device__ constexpr double sinpi_coef(int k)
{
    double c = PI;
    for (int i = 1; i <= k; ++i) c *= -PI * PI / ((2 * i) * (2 * i + 1));
    return c;
}
__host__ __device__ constexpr double cospi_coef(int k)
{
    double c = 1.0;
    for (int i = 1; i <= k; ++i) c *= -PI * PI / ((2 * i - 1) * (2 * i));
    return c;
}
// sin(pi x) and cos(pi x) for x in [-1, 1]
__device__ __forceinline__ void ff_sincospi(ff x, ff& s, ff& c)
{
    ff y = x.hi < 0.0f ? ff_neg(x) : x;
    const bool left = y.hi > 0.5f;
    if (left) y = ff_add_f(ff_neg(y), 1.0f);
    const bool swap = y.hi > 0.25f;
    const ff u = swap ? ff_add_f(ff_neg(y), 0.5f) : y;
    const ff2 U = splat(ff_mul(u, u));
    ff2 p = pack(to_ff(split_const(sinpi_coef(SINCOS_TERMS - 1))), to_ff(split_const(cospi_coef(SINCOS_TERMS - 1))));
#pragma unroll
    for (int k = SINCOS_TERMS - 2; k >= 1; --k)
        p = ff2_fma_open(p, U, pack(to_ff(split_const(sinpi_coef(k))), to_ff(split_const(cospi_coef(k)))));
    p = ff2_fma(p, U, pack(to_ff(split_const(sinpi_coef(0))), to_ff(split_const(cospi_coef(0)))));
    const ff a = ff_mul(lane0(p), u), b = lane1(p);
    s = swap ? b : a;
    c = swap ? a : b;
    if (x.hi < 0.0f) s = ff_neg(s);
    if (left) c = ff_neg(c);
}

// sin(pi d) and cos(pi d) for |d| <= 1/16 (half an ellipse leaf's angle): six
// terms, the next are below 2^-50 of the leading one
constexpr int SMALL_TERMS = 6;
__device__ __forceinline__ void ff_sincospi_small(ff d, ff& s, ff& c)
{
    const ff2 U = splat(ff_mul(d, d));
    ff2 p = pack(to_ff(split_const(sinpi_coef(SMALL_TERMS - 1))), to_ff(split_const(cospi_coef(SMALL_TERMS - 1))));
#pragma unroll
    for (int k = SMALL_TERMS - 2; k >= 1; --k)
        p = ff2_fma_open(p, U, pack(to_ff(split_const(sinpi_coef(k))), to_ff(split_const(cospi_coef(k)))));
    p = ff2_fma(p, U, pack(to_ff(split_const(sinpi_coef(0))), to_ff(split_const(cospi_coef(0)))));
    s = ff_mul(lane0(p), d);
    c = lane1(p);
}

// ------------------------------------------------------------- evaluators
// Ellipses whose speeds have an exponent below this may have denormal squares
// (semi-axes below 2^-511).
constexpr int ELLIPSE_TINY = -480;

template <int CODE>
struct EvalFF {
    static constexpr int P = code_degree(CODE);
    static constexpr int D = code_dim(CODE);
    // A, B, w0 (ellipse piece) or the derivative polynomial
    // b[k][d] = (k + 1) a[k + 1][d], stored after the midpoint position a[0]
    // (gcv_setup.cuh)
    __device__ __forceinline__ static void load(const float2* __restrict__ seg, ff* r)
    {
        if constexpr (CODE == 0) {
            r[0] = ff{seg[0].x, seg[0].y};
            r[1] = ff{seg[1].x, seg[1].y};
            r[2] = ff{seg[2].x, seg[2].y};  // w0 = (2 j + 1) / ELLIPSE_PIECES - 1: exact in FP32
        } else {
#pragma unroll
            for (int k = 0; k < P * D; ++k) {
                const float2 c = seg[D + k];
                r[k] = ff{c.x, c.y};
            }
        }
    }
    // the same from the FP64 table's position polynomial, all lengths times
    // 2^-s: b[k] = (k + 1) a[k + 1], or A, B (squared lengths) and w0
    __device__ __forceinline__ static void load(const double* __restrict__ seg, ff* r, int s)
    {
        if constexpr (CODE == 0) {
            if (s >= ELLIPSE_TINY) {
                r[0] = ff_from_double_scaled(seg[0], 2 * s);
                r[1] = ff_from_double_scaled(seg[1], 2 * s);
            } else {
                double A = seg[0], B = seg[1];
                int sA = 2 * s, sB = 2 * s;
                lift_denormal(A, sA);
                lift_denormal(B, sB);
                r[0] = A != 0.0 ? ff_from_double_scaled(A, sA) : ff{0.0f, 0.0f};
                r[1] = B != 0.0 ? ff_from_double_scaled(B, sB) : ff{0.0f, 0.0f};
            }
            r[2] = ff{__double2float_rn(seg[2]), 0.0f};
        } else {
#pragma unroll
            for (int k = 0; k < P; ++k)
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    const ff a = ff_from_double_scaled(seg[(k + 1) * D + d], s);
                    // exact for the powers of two
                    r[k * D + d] = (k & (k + 1)) == 0 ? ff_scale(a, float(k + 1)) : ff_mul_f(a, float(k + 1));
                }
        }
    }
    // the speeds of a B-spline piece at two points at once, in packed lanes, each
    // coefficient splat into both
    __device__ __forceinline__ static ff2 speed2(const ff* r, ff2 v)
    {
        static_assert(CODE != 0, "ellipse sums go by angle addition");
        ff2 s{};
#pragma unroll
        for (int d = 0; d < D; ++d) {
            ff2 acc = splat(r[(P - 1) * D + d]);
#pragma unroll
            for (int k = P - 2; k >= 1; --k) acc = ff2_fma_open(acc, v, splat(r[k * D + d]));
            if constexpr (P > 1) acc = ff2_fma(acc, v, splat(r[d]));
            s = d == 0 ? ff2_mul_open(acc, acc) : (d + 1 < D ? ff2_fma_open(acc, acc, s) : ff2_fma(acc, acc, s));
        }
        return ff2_sqrt_open(s);
    }
    // Speed rounded to FP32 and q at a float-float point (B-splines): the
    // components in float-float (Horner at the full point), their norm in FP32
    // (the sampler's Newton steps use f to FP32 accuracy only); t[j][d]: the
    // component's Taylor coefficients there in FP32, for speed_slope_near.
    __device__ __forceinline__ static float speed_slope_f(const ff* r, ff v, float& q, float* t)
    {
        float s = 0.0f, u = 0.0f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            ff acc = r[(P - 1) * D + d];
            float c[P];  // c[j], j >= 1: p^(j)(v) / j! by the nested Horner sums
#pragma unroll
            for (int j = 1; j < P; ++j) c[j] = 0.0f;
#pragma unroll
            for (int k = P - 2; k >= 0; --k) {
#pragma unroll
                for (int j = P - 1; j >= 2; --j)
                    if (j <= P - 1 - k) c[j] = fmaf(c[j], v.hi, c[j - 1]);
                c[1] = fmaf(c[1], v.hi, acc.hi);
                acc = ff_fma(acc, v, r[k * D + d]);
            }
            c[0] = acc.hi + acc.lo;
            s = fmaf(c[0], c[0], s);
            if constexpr (P > 1) u = fmaf(c[0], c[1], u);
#pragma unroll
            for (int j = 0; j < P; ++j) t[j * D + d] = c[j];
        }
        q = u;
        return sqrtf(s);
    }
    // speed and q at the distance x from the point of t
    __device__ __forceinline__ static float speed_slope_near(const float* t, float x, float& q)
    {
        float s = 0.0f, u = 0.0f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            float acc = t[(P - 1) * D + d], dacc = 0.0f;
#pragma unroll
            for (int k = P - 2; k >= 0; --k) {
                dacc = fmaf(dacc, x, acc);
                acc = fmaf(acc, x, t[k * D + d]);
            }
            s = fmaf(acc, acc, s);
            u = fmaf(acc, dacc, u);
        }
        q = u;
        return sqrtf(s);
    }
    // speed and q in plain FP32 from the coefficients' leading parts: for the
    // leaf table's f and q, which only shape the sampler's initial guess
    __device__ __forceinline__ static float speed_slope32(const ff* r, float v, float& q)
    {
        if constexpr (CODE == 0) {
            float sn, cs;
            sincospif(fmaf(v, (float)ELLIPSE_PIECE_SCALE, r[2].hi), &sn, &cs);
            q = (float)(PI * ELLIPSE_PIECE_SCALE) * r[0].hi * sn * cs;
            return sqrtf(fmaf(r[0].hi, sn * sn, r[1].hi));
        } else {
            float s = 0.0f, t = 0.0f;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                float acc = r[(P - 1) * D + d].hi, dacc = 0.0f;
#pragma unroll
                for (int k = P - 2; k >= 0; --k) {
                    dacc = fmaf(dacc, v, acc);
                    acc = fmaf(acc, v, r[k * D + d].hi);
                }
                s = fmaf(acc, acc, s);
                t = fmaf(acc, dacc, t);
            }
            q = t;
            return sqrtf(s);
        }
    }
};

// B-spline panels by node pairs.  The speed polynomials p_d (degree P - 1 in
// v) are shifted to the panel's midpoint m and scaled to its half width h:
// b_j = h^j p_d^(j)(m) / j!, so p_d(m + h x) = sum_j b_j x^j on x in [-1, 1]
// (Horner-form Taylor shift, (P - 1) P / 2 float-float FMAs per dimension,
// then exact power-of-two scaling; on deep panels the high terms may
// underflow, where they are below any float-float rounding of b_0).  The
// symmetric nodes m -+ h x_i then share one evaluation of the even part
// E = b_0 + b_2 x^2 + ... and the odd part O = x (b_1 + b_3 x^2 + ...):
// p(m -+ h x) = E -+ O.  Per pair of nodes this replaces two Horner passes
// in v (2 (P - 1) float-float FMAs per dimension) and the two node
// positions by about half the work.

// The speeds of two node pairs at once, in the lanes of packed FP32 pairs
// (FFMA2 / FADD2 / FMUL2): x and x2 hold the two pairs' offsets and their
// squares, the coefficients b are shared (each is splat into both lanes where
// it is used).
template <int P, int D>
__device__ __forceinline__ void ff_node_pair2(const ff* b, ff2 x, ff2 x2, ff2& fm, ff2& fp)
{
    constexpr int N = P - 1;
    constexpr int JE = (N % 2 == 0) ? N : N - 1;
    constexpr int JO = (N % 2 == 1) ? N : N - 1;
    ff2 sm{}, sp{};
#pragma unroll
    for (int d = 0; d < D; ++d) {
        ff2 e = splat(b[JE * D + d]);
#pragma unroll
        for (int j = JE - 2; j >= 0; j -= 2) e = ff2_fma_open(e, x2, splat(b[j * D + d]));
        ff2 lo_ = e, hi_ = e;
        if constexpr (JO >= 1) {
            ff2 o = splat(b[JO * D + d]);
#pragma unroll
            for (int j = JO - 2; j >= 1; j -= 2) o = ff2_fma_open(o, x2, splat(b[j * D + d]));
            o = ff2_mul_open(o, x);
            lo_ = ff2_add(e, ff2_neg(o));
            hi_ = ff2_add(e, o);
        }
        sm = d == 0 ? ff2_mul_open(lo_, lo_) : (d + 1 < D ? ff2_fma_open(lo_, lo_, sm) : ff2_fma(lo_, lo_, sm));
        sp = d == 0 ? ff2_mul_open(hi_, hi_) : (d + 1 < D ? ff2_fma_open(hi_, hi_, sp) : ff2_fma(hi_, hi_, sp));
    }
    fm = ff2_sqrt_open(sm);
    fp = ff2_sqrt_open(sp);
}

// The seven Kronrod node pairs and the centre as four packed steps.  The first
// two hold the pairs that are Gauss nodes too, so that only they add to G; the
// eighth lane is the centre node (x = 0: both of its "nodes" are the centre, so it
// carries half the centre weights).  Per step: x, x^2, the Kronrod weights and
// the Gauss weights, each as the hi / lo float pairs of both lanes.
struct GkStep2 {
    float2 xh, xl, x2h, x2l, wkh, wkl, wgh, wgl;
};
__host__ __device__ constexpr double gk_pair_wk(int j) { return gk_pair(j) < 7 ? gk_wk(gk_pair(j)) : 0.5 * gk_wk(7); }
__host__ __device__ constexpr double gk_pair_wg(int j) { return gk_pair(j) < 7 ? gk_wg(gk_pair(j)) : 0.5 * gk_wg(7); }
#define GCV_GK_STEP2(j)                                                                                          \
    {{split_const(gk_pair_x(2 * j)).hi, split_const(gk_pair_x(2 * j + 1)).hi},                                  \
     {split_const(gk_pair_x(2 * j)).lo, split_const(gk_pair_x(2 * j + 1)).lo},                                  \
     {split_const(gk_pair_x(2 * j) * gk_pair_x(2 * j)).hi, split_const(gk_pair_x(2 * j + 1) * gk_pair_x(2 * j + 1)).hi}, \
     {split_const(gk_pair_x(2 * j) * gk_pair_x(2 * j)).lo, split_const(gk_pair_x(2 * j + 1) * gk_pair_x(2 * j + 1)).lo}, \
     {split_const(gk_pair_wk(2 * j)).hi, split_const(gk_pair_wk(2 * j + 1)).hi},                                \
     {split_const(gk_pair_wk(2 * j)).lo, split_const(gk_pair_wk(2 * j + 1)).lo},                                \
     {split_const(gk_pair_wg(2 * j)).hi, split_const(gk_pair_wg(2 * j + 1)).hi},                                \
     {split_const(gk_pair_wg(2 * j)).lo, split_const(gk_pair_wg(2 * j + 1)).lo}}
static __constant__ GkStep2 c_gk_step2[4] = {GCV_GK_STEP2(0), GCV_GK_STEP2(1), GCV_GK_STEP2(2), GCV_GK_STEP2(3)};
#undef GCV_GK_STEP2
// step j's sums of node pairs into K and G
__device__ __forceinline__ void gk_add(int j, ff2 sum, ff2& kk2, ff2& gg2)
{
    const GkStep2& c = c_gk_step2[j];
    kk2 = ff2_fma(ff2{c.wkh, c.wkl}, sum, kk2);
    if (j < 2) gg2 = ff2_fma(ff2{c.wgh, c.wgl}, sum, gg2);
}

// the midpoint of panel (k, depth), built exactly from the integer k
__device__ __forceinline__ ff panel_mid(unsigned long long k, int depth)
{
    const float hw = __int_as_float((127 - depth) << 23);  // 2^-depth, exact
    const float kh = (float)(unsigned)(k >> 24), kl = (float)(unsigned)(k & 0xFFFFFFull);
    const float sh = __int_as_float((127 + 25 - depth) << 23), sl = 2.0f * hw;  // 2^(25-depth), 2^(1-depth)
    return ff_add_f(ff_add_f(two_sum(-1.0f, kh * sh), kl * sl), hw);
}

// An ellipse piece's panel by angle addition (AngleTable), two node pairs per
// packed step as in panel_k15_ff_pairs.  r: A, B, w0.
__device__ __forceinline__ void panel_k15_ff_ellipse(const ff* r, unsigned long long k, int depth, ff& K, ff& G)
{
    const float hw = __int_as_float((127 - depth) << 23);  // 2^-depth, exact
    ff sm, cm;
    ff_sincospi(ff_add_f(ff_scale(panel_mid(k, depth), (float)ELLIPSE_PIECE_SCALE), r[2].hi), sm, cm);
    const ff2 s2 = splat(sm), c2 = splat(cm), A = splat(r[0]), B = splat(r[1]);
    const float4* tab = reinterpret_cast<const float4*>(c_angle.ff[depth]);
    ff2 kk2{}, gg2{};
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
        const float4 a = __ldg(tab + 2 * j), b = __ldg(tab + 2 * j + 1);
        const ff2 sd{make_float2(a.x, b.x), make_float2(a.y, b.y)}, cd{make_float2(a.z, b.z), make_float2(a.w, b.w)};
        const ff2 p = ff2_mul_open(s2, cd);
        const ff2 up = ff2_fma(c2, sd, p), dn = ff2_fma(c2, ff2_neg(sd), p);
        const ff2 fm = ff2_sqrt_open(ff2_fma(A, ff2_mul_open(dn, dn), B));
        const ff2 fp = ff2_sqrt_open(ff2_fma(A, ff2_mul_open(up, up), B));
        gk_add(j, ff2_add_open(fm, fp), kk2, gg2);
    }
    K = ff_scale(ff_add(lane0(kk2), lane1(kk2)), hw);
    G = ff_scale(ff_add(lane0(gg2), lane1(gg2)), hw);
}

// b: the interval's speed coefficients on entry, shifted to the panel's midpoint
// and scaled to its half width in place
template <int P, int D>
__device__ __forceinline__ void panel_shift(ff* b, unsigned long long k, int depth)
{
    const ff mid = panel_mid(k, depth);
    // Taylor shift to mid: after pass i, b[i] holds p^(i)(mid) / i!
#pragma unroll
    for (int i = 0; i < P - 1; ++i)
#pragma unroll
        for (int j = P - 2; j >= i; --j)
#pragma unroll
            for (int d = 0; d < D; ++d) b[j * D + d] = ff_fma_open(b[(j + 1) * D + d], mid, b[j * D + d]);
    const float hw = __int_as_float((127 - depth) << 23);
    float sc = hw;
#pragma unroll
    for (int j = 1; j < P; ++j) {
#pragma unroll
        for (int d = 0; d < D; ++d) b[j * D + d] = ff_scale(b[j * D + d], sc);
        sc *= hw;
    }
}

template <int CODE>
__device__ __forceinline__ void panel_k15_ff_pairs(ff* b, unsigned long long k, int depth, ff& K, ff& G)
{
    constexpr int P = code_degree(CODE), D = code_dim(CODE);
    const float hw = __int_as_float((127 - depth) << 23);
    panel_shift<P, D>(b, k, depth);
    // the node pairs two at a time in packed lanes (the centre in the last
    // step's second lane); the two lanes' sums are added at the end
    ff2 kk2{}, gg2{};
    // Rolled: four inlined copies of even a planar quadratic's step missed the
    // instruction cache (k_walk of planar degree 2-3: no_instruction first
    // among the stalls after the fixed latencies; the uneven batch's walk 14.4 ms
    // unrolled, 13.0 rolled).
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
        const GkStep2& c = c_gk_step2[j];
        ff2 fm, fp;
        ff_node_pair2<P, D>(b, ff2{c.xh, c.xl}, ff2{c.x2h, c.x2l}, fm, fp);
        gk_add(j, ff2_add_open(fm, fp), kk2, gg2);
    }
    const ff kk = ff_add(lane0(kk2), lane1(kk2));
    const ff gg = ff_add(lane0(gg2), lane1(gg2));
    K = ff_scale(kk, hw);
    G = ff_scale(gg, hw);
}

// the float-float panel of a curve code, by node pairs: B-splines from the
// polynomials shifted to the midpoint, ellipses by angle addition; r (the interval's
// speed coefficients) is scratch: the B-spline panel shifts it in place
template <int CODE>
__device__ __forceinline__ void panel_ff(ff* r, unsigned long long k, int depth, ff& K, ff& G)
{
    if constexpr (CODE == 0)
        panel_k15_ff_ellipse(r, k, depth, K, G);
    else
        panel_k15_ff_pairs<CODE>(r, k, depth, K, G);
}

__device__ __forceinline__ void load_ff_dyn(int code, const float2* __restrict__ seg, ff* r)
{
    switch (code) {
#define GCV_CASE(C)                                                                                \
    case C: EvalFF<C>::load(seg, r); break;
        GCV_FOR_EACH_CODE(GCV_CASE)
#undef GCV_CASE
    default: break;
    }
}

__device__ __forceinline__ void panel_ff_dyn(int code, ff* r, unsigned long long k, int depth, ff& K, ff& G)
{
    switch (code) {
#define GCV_CASE(C)                                                                                \
    case C: panel_ff<C>(r, k, depth, K, G); break;
        GCV_FOR_EACH_CODE(GCV_CASE)
#undef GCV_CASE
    default: K = G = ff{0.0f, 0.0f}; break;
    }
}

template <int CODE>
__device__ __forceinline__ float speed_slope32_of(int code, const ff* r, float v, float& q)
{
    if constexpr (CODE >= 0) {
        return EvalFF<CODE>::speed_slope32(r, v, q);
    } else {
        switch (code) {
#define GCV_CASE(C)                                                                                \
    case C: return EvalFF<C>::speed_slope32(r, v, q);
            GCV_FOR_EACH_CODE(GCV_CASE)
#undef GCV_CASE
        default: q = 0.0f; return 0.0f;
        }
    }
}

}  // namespace gcv
