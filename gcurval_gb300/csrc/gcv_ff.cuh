// Float-float ("double-float") arithmetic on the FP32 pipes.
//
// A value is an unevaluated sum hi + lo of two floats with |lo| <= ulp(hi)/2,
// about 48 significant bits.  The building blocks are the published
// error-free transformations: Knuth's TwoSum, Dekker's Fast2Sum, and the
// FMA-based exact product (TwoProd).  Every operation below is a handful of
// FP32 instructions; on GB300 an FP32 instruction costs 1/75 of an FP64 one,
// so a float-float polynomial evaluation is several times cheaper than the
// same evaluation in FP64 while keeping ~1e-14 relative accuracy.
//
// Nothing here may be compiled with fast-math (it relies on IEEE rounding and
// on the compiler not reassociating additions; the files are built without
// --use_fast_math and multiply-adds are written as explicit fmaf).
#pragma once

#include <cuda_runtime.h>

namespace gcv {

struct ff {
    float hi, lo;
};

// Dekker Fast2Sum (|a| >= |b|)
__device__ __forceinline__ ff fast_two_sum(float a, float b);

// double -> float-float from the bit pattern (integer and FP32 operations
// only: on GB300 every FP64-pipe instruction, conversions included, costs as
// much issue time as dozens of FP32 ones).  hi = the leading 24 significand
// bits, lo = the remaining 29 bits scaled by 2^(e-52) (rounded to 24 bits),
// then renormalised.  Outside 2^-100 <= |x| < 2^127 (and for 0, NaN, Inf) the
// FP64 conversions are used.
__device__ __forceinline__ ff ff_from_double(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned top = (unsigned)(b >> 32);
    const int e = (int)((top >> 20) & 0x7FFu) - 1023;
    if (e < -100 || e > 126) {
        const float h = __double2float_rn(x);
        return ff{h, __double2float_rn(x - (double)h)};
    }
    const unsigned sign = top & 0x80000000u;
    const unsigned long long m = b & 0xFFFFFFFFFFFFFull;  // 52 significand bits
    const float hi = __uint_as_float(sign | ((unsigned)(e + 127) << 23) | (unsigned)(m >> 29));
    const int sc = e - 52, s1 = sc / 2, s2 = sc - s1;   // two factors inside the float range
    float lo = __uint2float_rn((unsigned)(m & 0x1FFFFFFFull));
    lo = lo * __int_as_float((s1 + 127) << 23) * __int_as_float((s2 + 127) << 23);
    return fast_two_sum(hi, sign ? -lo : lo);
}

// x 2^-s -> float-float from the bit pattern, for data of any double range:
// the caller's s brings the values it works with near 1, and what falls below
// 2^-70 there is 0 (far under any float-float rounding of them), what rises
// above 2^126 is infinite.  NaN and infinities pass through (s above -1150: a
// zero's exponent counts as 2^-1023).  Selects, no
// branches: the samplers convert up to 15 coefficients per Newton step.
__device__ __forceinline__ ff ff_from_double_scaled(double x, int s)
{
    const unsigned top = (unsigned)__double2hiint(x), low = (unsigned)__double2loint(x);
    const unsigned sign = top & 0x80000000u, raw = (top >> 20) & 0x7FFu;
    const int e = (int)raw - 1023 - s;
    const bool tiny = raw == 0u || e < -70, huge = raw == 0x7FFu || e > 126;
    const unsigned m = ((top & 0xFFFFFu) << 3) | (low >> 29);
    const unsigned special = raw == 0x7FFu && ((top & 0xFFFFFu) | low) != 0u ? 0x7FC00000u : 0x7F800000u;
    const float hi = __uint_as_float(sign | (huge ? special : tiny ? 0u : ((unsigned)(e + 127) << 23) | m));
    const float lo = __uint2float_rn(low & 0x1FFFFFFFu) * __uint_as_float(((unsigned)(e - 52 + 127) << 23) | sign);
    return tiny || huge ? ff{hi, 0.0f} : fast_two_sum(hi, lo);
}

// x 2^-s as (x, s) with x out of the denormals
__device__ __forceinline__ void lift_denormal(double& x, int& s)
{
    if ((__double2hiint(x) & 0x7FF00000) == 0) {
        x *= 18446744073709551616.0;  // 2^64
        s += 64;
    }
}

// binary exponent of a double's magnitude (0 for 0, infinities and NaN)
__device__ __forceinline__ int exponent_of(double x)
{
    const int raw = (int)((unsigned)(__double2hiint(x)) >> 20) & 0x7FF;
    return raw == 0 || raw == 0x7FF ? 0 : raw - 1023;
}

// x 2^-s, s of any size (flushes to 0 / overflows to infinity)
__device__ __forceinline__ float scale_down(float x, int s)
{
    const int c = s < -252 ? -252 : (s > 252 ? 252 : s), h = c / 2;
    return x * __int_as_float((127 - h) << 23) * __int_as_float((127 - (c - h)) << 23);
}

__device__ __forceinline__ double ff_to_double(ff a) { return (double)a.hi + (double)a.lo; }

// Local parameters v in [-1, 1] and offsets in them as 64-bit integers in units
// of 2^-60: panel ends are exact, sums and differences are integer adds, and
// nothing of it occupies the FP64 pipe.
constexpr long long FIX_ONE = 1ll << 60;
// |x| < 2, from the bit pattern (truncated below 2^-60; panel ends are exact)
__device__ __forceinline__ long long fix_of_double(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int raw = (int)(b >> 52) & 0x7FF, sh = raw - 1023 + 8;
    const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const long long v = sh >= 0 ? (long long)(m << (sh & 15)) : (sh > -53 ? (long long)(m >> -sh) : 0ll);
    return (long long)b < 0 ? -v : v;
}
// back, the scaling by the exponent bits: with the unit in a factor, knot spans below
// 2^-960 became denormals and their parameters lost digits
__device__ __forceinline__ double double_of_fix(long long v)
{
    const double x = __ll2double_rn(v);
    return __hiloint2double(__double2hiint(x) - (v != 0 ? 60 << 20 : 0), __double2loint(x));
}
__device__ __forceinline__ long long fix_of_float(float x) { return __float2ll_rn(x * 1152921504606846976.0f); }

// float -> double from the bit pattern (the FP64 pipe's conversion for zeros,
// denormals, infinities and NaN)
__device__ __forceinline__ double double_of_float(float x)
{
    const unsigned b = __float_as_uint(x), e = (b >> 23) & 0xFFu;
    if (e == 0u || e == 0xFFu) return (double)x;
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + (896u << 20))), (int)(b << 29));
}

// reciprocal to an ulp, for factors that carry FP32 rounding anyway
__device__ __forceinline__ float rcp_approx(float x) { return __fdividef(1.0f, x); }

// double -> float by truncation of the significand, from the bit pattern
// (integer operations only), for scale factors that need a few digits;
// outside the normal float range (and for 0, NaN, Inf) the FP64 conversion
__device__ __forceinline__ float f32_of_f64_trunc(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned top = (unsigned)(b >> 32);
    const int e = (int)((top >> 20) & 0x7FFu) - 1023 + 127;
    if (e <= 0 || e >= 255) return __double2float_rn(x);
    return __uint_as_float((top & 0x80000000u) | ((unsigned)e << 23) | (unsigned)((b >> 29) & 0x7FFFFFull));
}

// Knuth TwoSum: s + e == a + b exactly
__device__ __forceinline__ ff two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return ff{s, e};
}

// Dekker Fast2Sum (|a| >= |b|)
__device__ __forceinline__ ff fast_two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    return ff{s, __fsub_rn(b, __fsub_rn(s, a))};
}

// a + b, "sloppy" variant: error relative to |a| + |b|
__device__ __forceinline__ ff ff_add(ff a, ff b)
{
    const ff s = two_sum(a.hi, b.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}

__device__ __forceinline__ ff ff_add_f(ff a, float b)
{
    const ff s = two_sum(a.hi, b);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, a.lo));
}

__device__ __forceinline__ ff ff_neg(ff a) { return ff{-a.hi, -a.lo}; }

// a * b with the exact product of the high parts
__device__ __forceinline__ ff ff_mul(ff a, ff b)
{
    const float p = __fmul_rn(a.hi, b.hi);
    const float e = fmaf(a.hi, b.hi, -p);
    return fast_two_sum(p, fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e)));
}

__device__ __forceinline__ ff ff_mul_f(ff a, float b)
{
    const float p = __fmul_rn(a.hi, b);
    const float e = fmaf(a.hi, b, -p);
    return fast_two_sum(p, fmaf(a.lo, b, e));
}

// exact scaling by a power of two
__device__ __forceinline__ ff ff_scale(ff a, float pow2) { return ff{a.hi * pow2, a.lo * pow2}; }

// a * b + c in one pass: the exact product of the high parts (p + e) and the
// cross terms enter the sloppy sum with c without first renormalising the
// product, 15 FP32 instructions instead of ff_add(ff_mul(a, b), c)'s 18,
// with the same error bound relative to |a b| + |c| (the unnormalised tail t
// is below 2^-22 |p| and is rounded once more, into the low-order sum).
__device__ __forceinline__ ff ff_fma(ff a, ff b, ff c)
{
    const float p = __fmul_rn(a.hi, b.hi);
    const float t = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, fmaf(a.hi, b.hi, -p)));
    const ff s = two_sum(p, c.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(t, c.lo)));
}

// ff_fma whose result is left unnormalised (|lo| up to a few ulp of hi): for the
// inner steps of sums and Horner chains, whose next operation takes it as well
// as the normalised value (compensated Horner's scheme, Langlois and Louvet:
// the low parts are one plain Horner sum beside the high ones').  Three
// instructions fewer, and the next product waits for two roundings (hi = p + c.hi)
// instead of nine.  (The panels of 50,000 spatial curves 1.97 -> 1.73 ms, their
// samples 10.8 -> 10.2.)  What is subtracted from something of its own size, squared
// or stored is normalised.
__device__ __forceinline__ ff ff_fma_open(ff a, ff b, ff c)
{
    const float p = __fmul_rn(a.hi, b.hi);
    const float t = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, fmaf(a.hi, b.hi, -p)));
    const ff s = two_sum(p, c.hi);
    return ff{s.hi, __fadd_rn(s.lo, __fadd_rn(t, c.lo))};
}
__device__ __forceinline__ ff ff_mul_open(ff a, ff b)
{
    const float p = __fmul_rn(a.hi, b.hi);
    return ff{p, fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, fmaf(a.hi, b.hi, -p)))};
}

// 1 / b: y = rcp(b.hi), then one Newton step y + y (1 - b y) with the
// residual 1 - b y formed by FMAs (b.lo enters there)
__device__ __forceinline__ ff ff_recip(ff b)
{
    const float y = __frcp_rn(b.hi);
    const float e = fmaf(-b.lo, y, fmaf(-b.hi, y, 1.0f));
    return fast_two_sum(y, __fmul_rn(y, e));
}

// sqrt: s = a y with y = rsqrt(a) (a few ulp), then the correction c = (a - s^2) y / 2
// with the residual a - s^2 formed exactly by an FMA.  With y = (1 + d) / sqrt(a),
// c is off by 3/2 d^2, i.e. by 3/2 c^2 y, which is added (without it this term,
// up to 2^-45, was the largest error of a panel's sums: K15 of random panels of
// degree 2 - 5 was off by 2.7 - 2.9e-15 rms before, 2.4 - 2.65e-15 now).
__device__ __forceinline__ ff ff_sqrt(ff a)
{
    if (!(a.hi > 0.0f)) return ff{a.hi == 0.0f ? 0.0f : __fsqrt_rn(a.hi), 0.0f};
    const float y = rsqrtf(a.hi);
    const float s = __fmul_rn(a.hi, y);
    const float r = __fadd_rn(fmaf(-s, s, a.hi), a.lo);
    const float c = __fmul_rn(r, 0.5f * y);
    return fast_two_sum(s, fmaf(__fmul_rn(1.5f, c), __fmul_rn(c, y), c));
}

}  // namespace gcv
