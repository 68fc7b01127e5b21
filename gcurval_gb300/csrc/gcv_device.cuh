// Device-side building blocks of the arc-length library: quadrature
// constants, curve evaluators on per-knot-interval polynomials (set up by
// gcv_setup.cuh), and warp helpers.
//
// Every knot interval ("segment") is mapped to a local variable v in [-1, 1]:
//   B-spline  t = t0 + (v + 1) * hw,  hw = (k[span+1] - k[span]) / 2
//   ellipse   piece j of ELLIPSE_PIECES equal parameter pieces of [0, 2 pi]:
//             theta = pi * (2 j + 1 + v) / ELLIPSE_PIECES
// and the integrand is f(v) = |dC/dv| = |C'(t)| * hw, so that the segment
// length is the integral of f over [-1, 1].
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gcv {

// ---------------------------------------------------------------- constants
// 15-point Kronrod rule with its embedded 7-point Gauss rule (the published
// Gauss-Kronrod G7-K15 nodes and weights), nodes descending from the right end.
__host__ __device__ constexpr double gk_x(int i)
{
    return i == 0 ? 0.991455371120812639206854697526329
         : i == 1 ? 0.949107912342758524526189684047851
         : i == 2 ? 0.864864423359769072789712788640926
         : i == 3 ? 0.741531185599394439863864773280788
         : i == 4 ? 0.586087235467691130294144845693013
         : i == 5 ? 0.405845151377397166906606412076961
         : i == 6 ? 0.207784955007898467600689403773245
                  : 0.0;
}
__host__ __device__ constexpr double gk_wk(int i)
{
    return i == 0 ? 0.022935322010529224963732008058970
         : i == 1 ? 0.063092092629978553290700663189204
         : i == 2 ? 0.104790010322250183839876322541518
         : i == 3 ? 0.140653259715525918745189590510238
         : i == 4 ? 0.169004726639267902826583426598550
         : i == 5 ? 0.190350578064785409913256402421014
         : i == 6 ? 0.204432940075298892414161999234649
                  : 0.209482141084727828012999174891714;
}
// Gauss weights of the odd Kronrod indices 1, 3, 5 and of the centre (7)
__host__ __device__ constexpr double gk_wg(int i)
{
    return i == 1 ? 0.129484966168869693270611432679082
         : i == 3 ? 0.279705391489276667901467771423780
         : i == 5 ? 0.381830050505118944950369775488975
         : i == 7 ? 0.417959183673469387755102040816327
                  : 0.0;
}

// 8-point Gauss-Legendre nodes / weights (positive half; symmetric)
__host__ __device__ constexpr double gl8_x(int i)
{
    return i == 0 ? 0.183434642495649804939476142360184
         : i == 1 ? 0.525532409916328985817739049189254
         : i == 2 ? 0.796666477413626739591553936475830
                  : 0.960289856497536231683560868569473;
}
__host__ __device__ constexpr double gl8_w(int i)
{
    return i == 0 ? 0.362683783378361982965150449277196
         : i == 1 ? 0.313706645877887287337962201986601
         : i == 2 ? 0.222381034453374470544355994426241
                  : 0.101228536290376259152531354309962;
}

constexpr double PI = 3.141592653589793238462643383279502884;

// ------------------------------------------------------------ curve codes
// 0 = ellipse; B-splines 16 + 4 p + D for degree p in 1..5 and D in {2, 3}.
constexpr int CODE_ELLIPSE = 0;
__host__ __device__ constexpr int bs_code(int p, int d) { return 16 + 4 * p + d; }
__host__ __device__ constexpr int code_degree(int code) { return code == 0 ? 0 : (code - 16) / 4; }
__host__ __device__ constexpr int code_dim(int code) { return code == 0 ? 2 : (code - 16) % 4; }
// values of coefficient data per segment: the position polynomial of a
// B-spline piece ((p + 1) D), the 9 ellipse terms
__host__ __device__ constexpr int code_stride(int code)
{
    return code == 0 ? 9 : (code_degree(code) + 1) * code_dim(code);
}
// An ellipse is integrated as this many equal parameter pieces (a power of
// two, so that v / ELLIPSE_PIECES is exact): more lanes per curve and a few
// leaves per piece instead of one long chain of panels.
constexpr int ELLIPSE_PIECES = 8;
constexpr double ELLIPSE_PIECE_SCALE = 1.0 / ELLIPSE_PIECES;
constexpr int MAX_DEGREE = 5;
constexpr int MAX_COEF = 18;  // (5 + 1) * 3

// Exact 2^-k for 0 <= k <= 1000 built from the exponent bits (no FP64 op).
__device__ __forceinline__ double pow2_neg(int k)
{
    return __longlong_as_double((long long)(1023 - k) << 52);
}

// ------------------------------------------------------------- evaluators
// Ellipse piece data (9 doubles): A = (a^2 - b^2) h^2, B = b^2 h^2 with
// h = pi / ELLIPSE_PIECES, w0 = (2 j + 1) / ELLIPSE_PIECES - 1, then a, b,
// cos(rot), sin(rot), cx, cy.  With w = w0 + v / ELLIPSE_PIECES in [-1, 1]
// (theta = pi (w + 1)): f(v) = sqrt(B + A sin^2(pi w)), because
// |C'(theta)|^2 = a^2 sin^2 + b^2 cos^2 and sin^2(pi (w + 1)) = sin^2(pi w).
__device__ __forceinline__ double ellipse_speed(double A, double B, double w0, double v)
{
    const double s = sinpi(fma(v, ELLIPSE_PIECE_SCALE, w0));
    return sqrt(fma(A * s, s, B));
}

// B-spline segment data: position polynomial a[k][d] (k = 0..P), then the
// derivative polynomial b[k][d] = (k + 1) a[k + 1][d] (k = 0..P-1), both in v.
template <int P, int D>
__device__ __forceinline__ double bs_speed(const double* b, double v)
{
    double s = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        double acc = b[(P - 1) * D + d];
#pragma unroll
        for (int k = P - 2; k >= 0; --k) acc = fma(acc, v, b[k * D + d]);
        s = d == 0 ? acc * acc : fma(acc, acc, s);
    }
    return sqrt(s);
}

// f = |g(v)| and q = g(v) . g'(v) (so df/dv = q / f): Horner for the value
// and its derivative in one pass.
template <int P, int D>
__device__ __forceinline__ double bs_speed_slope(const double* b, double v, double& q)
{
    double s = 0.0, t = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        double acc = b[(P - 1) * D + d], dacc = 0.0;
#pragma unroll
        for (int k = P - 2; k >= 0; --k) {
            dacc = fma(dacc, v, acc);
            acc = fma(acc, v, b[k * D + d]);
        }
        s = d == 0 ? acc * acc : fma(acc, acc, s);
        t = d == 0 ? acc * dacc : fma(acc, dacc, t);
    }
    q = t;
    return sqrt(s);
}

// ellipse: f^2 = B + A sin^2(pi w), dw/dv = 1 / ELLIPSE_PIECES, so
// q = f f' = A sin cos pi / ELLIPSE_PIECES
__device__ __forceinline__ double ellipse_speed_slope(double A, double B, double w0, double v, double& q)
{
    double s, c;
    sincospi(fma(v, ELLIPSE_PIECE_SCALE, w0), &s, &c);
    q = (PI * ELLIPSE_PIECE_SCALE) * A * s * c;
    return sqrt(fma(A * s, s, B));
}

template <int P, int D>
__device__ __forceinline__ void bs_point(const double* a, double v, double* out)
{
#pragma unroll
    for (int d = 0; d < D; ++d) {
        double acc = a[P * D + d];
#pragma unroll
        for (int k = P - 1; k >= 0; --k) acc = fma(acc, v, a[k * D + d]);
        out[d] = acc;
    }
}

// Register copy of one segment's evaluation data.
struct SegRegs {
    double c[MAX_COEF];
};

template <int CODE>
struct Eval {
    static constexpr int P = code_degree(CODE);
    static constexpr int D = code_dim(CODE);
    static constexpr int NL = CODE == 0 ? 3 : P * D;  // doubles the speed needs
    // loads what speed() needs: ellipse A, B, w0, or the derivative polynomial
    // b[k][d] = (k + 1) a[k + 1][d] of the stored position polynomial a
    __device__ __forceinline__ static void load_speed(const double* __restrict__ seg, double* r)
    {
        if constexpr (CODE == 0) {
            r[0] = seg[0];
            r[1] = seg[1];
            r[2] = seg[2];
        } else {
#pragma unroll
            for (int k = 0; k < P; ++k)
#pragma unroll
                for (int d = 0; d < D; ++d) r[k * D + d] = double(k + 1) * seg[(k + 1) * D + d];
        }
    }
    __device__ __forceinline__ static double speed(const double* r, double v)
    {
        if constexpr (CODE == 0)
            return ellipse_speed(r[0], r[1], r[2], v);
        else
            return bs_speed<P, D>(r, v);
    }
    // speed and q = f * df/dv
    __device__ __forceinline__ static double speed_slope(const double* r, double v, double& q)
    {
        if constexpr (CODE == 0)
            return ellipse_speed_slope(r[0], r[1], r[2], v, q);
        else
            return bs_speed_slope<P, D>(r, v, q);
    }
    // point at local v (writes D doubles; ellipses apply rotation and centre)
    __device__ __forceinline__ static void point(const double* __restrict__ seg, double v, double* out)
    {
        if constexpr (CODE == 0) {
            // theta / pi = (2 j + 1 + v) / ELLIPSE_PIECES = (w0 + 1) + v / ELLIPSE_PIECES
            double s, c;
            sincospi(fma(v, ELLIPSE_PIECE_SCALE, seg[2] + 1.0), &s, &c);
            const double x = seg[3] * c, y = seg[4] * s;
            out[0] = seg[5] * x - seg[6] * y + seg[7];
            out[1] = seg[6] * x + seg[5] * y + seg[8];
        } else {
            double a[(P + 1) * D];
#pragma unroll
            for (int i = 0; i < (P + 1) * D; ++i) a[i] = seg[i];
            bs_point<P, D>(a, v, out);
        }
    }
};

// Runtime dispatch over every built-in code, for batches that mix curve kinds.
#define GCV_FOR_EACH_CODE(X)                                                                       \
    X(0) X(bs_code(1, 2)) X(bs_code(2, 2)) X(bs_code(3, 2)) X(bs_code(4, 2)) X(bs_code(5, 2))      \
        X(bs_code(1, 3)) X(bs_code(2, 3)) X(bs_code(3, 3)) X(bs_code(4, 3)) X(bs_code(5, 3))

__device__ __forceinline__ void load_speed_dyn(int code, const double* __restrict__ seg, double* r)
{
    switch (code) {
#define GCV_CASE(C)                                                                                \
    case C: Eval<C>::load_speed(seg, r); break;
        GCV_FOR_EACH_CODE(GCV_CASE)
#undef GCV_CASE
    default: break;
    }
}

__device__ __forceinline__ void point_dyn(int code, const double* __restrict__ seg, double v, double* out)
{
    switch (code) {
#define GCV_CASE(C)                                                                                \
    case C: Eval<C>::point(seg, v, out); break;
        GCV_FOR_EACH_CODE(GCV_CASE)
#undef GCV_CASE
    default: break;
    }
}

// ------------------------------------------------------------ warp helpers
// Non-negative doubles order like their bit patterns: binary searches on
// cumulative lengths compare 64-bit integers instead of using the FP64 pipe.
__device__ __forceinline__ long long dkey(double x) { return __double_as_longlong(x); }

// first index in [lo, hi) with a[i] >= key (a non-decreasing, non-negative)
__device__ __forceinline__ int64_t lower_bound_key(const double* __restrict__ a, int64_t lo, int64_t hi,
                                                   long long key)
{
    int64_t n = hi - lo;
    while (n > 0) {
        const int64_t h = n >> 1;
        if (dkey(__ldg(a + lo + h)) < key) {
            lo += h + 1;
            n -= h + 1;
        } else {
            n = h;
        }
    }
    return lo;
}

// the same over n entries from a, as an offset in 32 bits
__device__ __forceinline__ int lower_bound_key32(const double* __restrict__ a, int n, long long key)
{
    int lo = 0;
    while (n > 0) {
        const int h = n >> 1;
        const bool less = dkey(__ldg(a + lo + h)) < key;
        lo = less ? lo + h + 1 : lo;
        n = less ? n - h - 1 : h;
    }
    return lo;
}

// last index i in [0, n) with off[i] <= x (off non-decreasing, off[0] <= x)
__device__ __forceinline__ int upper_bound_i64(const int64_t* __restrict__ off, int n, int64_t x)
{
    int lo = 0, cnt = n;
    while (cnt > 0) {
        const int h = cnt >> 1;
        if (__ldg(off + lo + h) <= x) {
            lo += h + 1;
            cnt -= h + 1;
        } else {
            cnt = h;
        }
    }
    return lo - 1;
}

}  // namespace gcv
