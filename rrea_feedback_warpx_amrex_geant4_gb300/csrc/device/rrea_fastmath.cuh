// Table-driven natural logarithm and exponential for the transport loops.
//
// GB300 issues two FP64 FMAs per clock per SM, and the library logarithm is
// one of the largest FP64 consumers of a substep (table brackets, the GS
// angle inversion, the hazard depth).  This follows the table-driven method
// of P. T. P. Tang, "Table-driven implementation of the logarithm function in
// IEEE floating-point arithmetic", ACM TOMS 16(4), 1990:
//   x = 2^e m with m in [1, 2),  F = 1 + j/256 the table point nearest m,
//   f = m - F (exact: both in [1, 2], |f| <= 2^-9),  r = f * (1/F),
//   log x = e ln2 + log F + log1p(r),
// log1p(r) by its Taylor series through r^6 (|r| <= 2^-9, so the first
// omitted term is below 2^-62 absolutely and 2^-54 relative to r).  The
// table (RREA_ARENA_LOG_TABLE_ROWS rows of {1/F, log F high, log F low},
// filled on the host in extended precision) opens the arena.  The result is
// within two ulps of the correctly rounded logarithm for every normal
// positive x; zero, negative, subnormal, infinite and NaN inputs go to the
// CUDA log.  The coefficients are the exact rationals of the series; ln 2
// is split into its double rounding and the rounding of the remainder.
#pragma once

#include "../rrea_arena.h"
#include "rrea_rate_rows.cuh"

#include <stdint.h>

namespace rrea_dev {

constexpr double kLn2Hi = 6.93147180559945286227e-01;   // RN(ln 2)
constexpr double kLn2Lo = 2.31904681384629955842e-17;   // RN(ln 2 - kLn2Hi)

static __device__ __noinline__ double log_any(double x) { return log(x); }

__device__ __forceinline__ double flog(const double* __restrict__ arena, double x)
{
#ifdef RREA_CUDA_LIBM
    // parity-study build: CUDA's logarithm everywhere
    (void)arena;
    return log(x);
#endif
    long long const bits = __double_as_longlong(x);
    // normal, positive and finite: sign clear, biased exponent in [1, 2046]
    if (bits < 0x0010000000000000LL || bits >= 0x7ff0000000000000LL) return log_any(x);
    long long const mant = bits & 0x000fffffffffffffLL;
    int const j = static_cast<int>((mant + (1LL << 43)) >> 44);  // nearest of the 257 points, 0..256
    double const m = __longlong_as_double(mant | 0x3ff0000000000000LL);
    // F = 1 + j/256 by its bits (j = 256 carries into the exponent: 2)
    double const f = m - __longlong_as_double(0x3ff0000000000000LL + (static_cast<long long>(j) << 44));
    const double* t = arena + RREA_ARENA_LOG_TABLE + 3 * j;
    double const r = f * __ldg(t);
    double const q = fma(r, fma(r, fma(r, fma(r, -1.0 / 6.0, 1.0 / 5.0), -0.25), 1.0 / 3.0), -0.5);
    double const p = fma(r * r, q, r);
    // e = biased exponent - 1023 as a double, by the low word of 2^52 + it
    double const de = __longlong_as_double(0x4330000000000000LL | (bits >> 52)) - (4503599627370496.0 + 1023.0);
    double const hi = fma(de, kLn2Hi, __ldg(t + 1));
    double const lo = fma(de, kLn2Lo, __ldg(t + 2)) + p;
    return hi + lo;
}

// Table-driven exponential after P. T. P. Tang, "Table-driven implementation
// of the exponential function in IEEE floating-point arithmetic", ACM TOMS
// 15(2), 1989: k = rint(x 128/ln2), x = k ln2/128 + r with |r| <= ln2/256
// (r from the split of ln2/128, two FMAs), exp x = 2^(k div 128) *
// 2^((k mod 128)/128) * exp(r), expm1(r) by its Taylor series through r^5
// (first omitted term below 2^-62; the r^4 and r^5 terms, below 2^-38, in
// FP32).  2^(j/128) comes from the table as two doubles.  k is read from the
// low word of a sum and 2^(k div 128) added to the exponent, so neither takes
// a conversion or a product.  Within two ulps of the correctly rounded
// exponential for |x| < 512; the rest goes to the CUDA exp.
constexpr double kInvLn2x128 = 1.84664965233787316142e+02;  // RN(128 / ln 2)
constexpr double kLn2by128Hi = 5.41521234812457272982e-03;  // RN(ln 2 / 128)
constexpr double kLn2by128Lo = 1.81175532331742157843e-19;  // RN(ln 2 / 128 - kLn2by128Hi)

static __device__ __noinline__ double exp_any(double x) { return exp(x); }

__device__ __forceinline__ double fexp(const double* __restrict__ arena, double x)
{
#ifdef RREA_CUDA_LIBM
    // parity-study build: CUDA's exponential everywhere
    (void)arena;
    return exp(x);
#endif
    // |x| >= 512, infinite or NaN
    if ((__double2hiint(x) & 0x7fffffff) >= 0x40800000) return exp_any(x);
    constexpr double magic = 6755399441055744.0;   // 1.5 2^52: the sum's low word is the nearest integer
    double const t = fma(x, kInvLn2x128, magic);
    int const k = __double2loint(t);
    double const kf = t - magic;
    double r = fma(-kf, kLn2by128Hi, x);
    r = fma(-kf, kLn2by128Lo, r);
    float const r32 = narrow_f32(r);
    double const q = fma(r, widen_f32(r32 * (1.0f / 24.0f + r32 * (1.0f / 120.0f))) + 1.0 / 6.0, 0.5);
    double const p = fma(r * r, q, r);  // expm1(r)
    double2 const tab = __ldg(reinterpret_cast<const double2*>(arena + RREA_ARENA_EXP_TABLE) + (k & 127));
    double const v = tab.x + fma(tab.x, p, tab.y);
    // 2^(k >> 7) into the exponent: |k| < 94,600, so v stays normal
    return __longlong_as_double(__double_as_longlong(v) + (static_cast<long long>(k >> 7) << 52));
}

// 1/sqrt(x) for the normalisations of the loop: an FP32 seed (relative error
// below 2^-21) and one third-order Householder step, y (1 + e/2 + 3 e^2/8)
// with e = 1 - x y^2 (the remainder 5 e^3/16 is below 2^-61), five FP64
// slots.  The square of the seed's 24 bits is exact, so e rounds once and the
// result is within 0.51 ulp (CUDA's 0.51; 0.98 with x y formed first).
// Arguments outside [2^-100, 2^100] go to CUDA's.
__device__ __forceinline__ bool root_in_range(double x)
{
    return static_cast<uint32_t>(__double2hiint(x)) - 0x39b00000u <= 0x0c800000u;
}
__device__ __forceinline__ double rsqrt_seed(double x)
{
    uint32_t const hi = static_cast<uint32_t>(__double2hiint(x)), lo = static_cast<uint32_t>(__double2loint(x));
    float const x32 = __uint_as_float(((hi - 0x38000000u) << 3) | (lo >> 29));
    float y32;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y32) : "f"(x32));
    uint32_t const u = __float_as_uint(y32);
    return __hiloint2double(static_cast<int>((u >> 3) + 0x38000000u), static_cast<int>(u << 29));
}
static __device__ __noinline__ double rsqrt_any(double x) { return rsqrt(x); }

__device__ __forceinline__ double frsqrt(double x)
{
    if (!root_in_range(x)) return rsqrt_any(x);
    double const y = rsqrt_seed(x);
    double const e = fma(-x, y * y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}
// sqrt(x) as x y (1 + e/2 + 3 e^2/8) with the rounding of x y recovered:
// within 0.51 ulp, eight FP64 slots (x times frsqrt: six, 1.32 ulps).  Zeros
// and arguments outside the range go to CUDA's.
static __device__ __noinline__ double sqrt_any(double x) { return sqrt(x); }

__device__ __forceinline__ double fsqrt(double x)
{
    if (!root_in_range(x)) return sqrt_any(x);
    double const y = rsqrt_seed(x);
    double const e = fma(-x, y * y, 1.0);
    double const s = x * y;
    return s + fma(s * e, fma(e, 0.375, 0.5), fma(x, y, -s));
}

// sin and cos of the table angle 2 pi j/256 plus r, |r| <= pi/256: sin r and
// cos r - 1 are r - r^3/6 + r^5/120 and -r^2/2 + r^4/24 - r^6/720, the last
// terms in FP32, and the table's value is added last: within 1.1 x 2^-53
// absolutely (CUDA's 1.15; 2.0 with the r^4 term in FP32 and the table's value
// added to each part).
constexpr double kTurnStep = 2.45436926061702587187e-02;     // RN(2 pi / 256)
constexpr double kTurnStepLo = 9.56755311833869693105e-19;   // RN(2 pi / 256 - kTurnStep)
constexpr double kInvTurnStep = 4.07436654315252084757e+01;  // RN(256 / (2 pi))
__device__ __forceinline__ void sincos_step(const double* __restrict__ arena, int j, double r, double& s, double& c)
{
    double2 const tab = __ldg(reinterpret_cast<const double2*>(arena + RREA_ARENA_TURN_TABLE) + (j & 255));
    double const r2 = r * r;
    float const q = narrow_f32(r2);
    double const cm = r2 * fma(r2, 1.0 / 24.0 - widen_f32(q * (1.0f / 720.0f)), -0.5);
    double const sr = fma(r * r2, widen_f32(q * (1.0f / 120.0f)) - 1.0 / 6.0, r);
    s = tab.x + fma(tab.y, sr, tab.x * cm);
    c = tab.y + fma(-tab.x, sr, tab.y * cm);
}
// sin and cos of 2 pi u for u in [0, 1): the nearest of 256 table angles and
// the remainder (exact up to the product by 2 pi/256), 17 FP64 slots against
// 31 of a reduction of 2 pi u.  It takes the angle itself, where the
// reference rounds 2 pi u (to 4e-16) first.
__device__ __forceinline__ void sincos_turn(const double* __restrict__ arena, double u, double& s, double& c)
{
    constexpr double magic = 6755399441055744.0;   // 1.5 2^52: the sum's low word is the nearest integer
    double const t = fma(u, 256.0, magic);
    sincos_step(arena, __double2loint(t), fma(u, 256.0, magic - t) * kTurnStep, s, c);
}
// sin and cos of an angle in radians, |a| < 2^10 (the rest goes to CUDA's):
// the remainder against the nearest table angle by two multiply-adds.
static __device__ __noinline__ double2 sincos_any(double a)
{
    double2 v;
    sincos(a, &v.x, &v.y);
    return v;
}
__device__ __forceinline__ void fsincos(const double* __restrict__ arena, double a, double& s, double& c)
{
    if ((__double2hiint(a) & 0x7fffffff) >= 0x40900000) {   // |a| >= 2^10, infinite or NaN
        double2 const v = sincos_any(a);
        s = v.x;
        c = v.y;
        return;
    }
    constexpr double magic = 6755399441055744.0;
    double const t = fma(a, kInvTurnStep, magic);
    double const k = t - magic;
    sincos_step(arena, __double2loint(t), fma(-k, kTurnStepLo, fma(-k, kTurnStep, a)), s, c);
}

// atan2(y, x): the FP32 angle names the nearest of 256 table angles a (0 up to
// 0.02, where the first table angle's rounding would weigh more than the
// result's), the point is turned by -a to (u, v) (v with the rounding of its
// second product recovered, so that it keeps its relative accuracy), and with
// t = v/u, |t| < 0.0201, the angle is a + t - t^3/3 + t^5/5 - t^7/7 + t^9/9
// (the last two terms in FP32; the next is below 2^-59): within two ulps (1.5
// measured, CUDA's 1.7), for 20 FP64 slots against 46.  Points nearer than
// 2^-100 to the origin or farther than 2^100 go to CUDA's.
static __device__ __noinline__ double atan2_any(double y, double x) { return atan2(y, x); }

__device__ __forceinline__ double fatan2(const double* __restrict__ arena, double y, double x)
{
    // the larger coordinate decides: past the FP32 range the seed would name
    // any angle
    uint32_t const hi = max(static_cast<uint32_t>(__double2hiint(x)) & 0x7fffffffu,
                            static_cast<uint32_t>(__double2hiint(y)) & 0x7fffffffu);
    if (hi - 0x39b00000u > 0x0c800000u) return atan2_any(y, x);
    float const a32 = atan2f(narrow_f32(y), narrow_f32(x));
    int const j = fabsf(a32) < 0.02f ? 0 : __float2int_rn(a32 * static_cast<float>(kInvTurnStep));
    double2 const tab = __ldg(reinterpret_cast<const double2*>(arena + RREA_ARENA_TURN_TABLE) + (j & 255));
    double const u = fma(x, tab.y, y * tab.x);
    double const p = x * tab.x;
    double const v = fma(y, tab.y, -p) - fma(x, tab.x, -p);
    // v / u: an FP32 reciprocal, one Newton step, the quotient's residual
    float y32;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y32) : "f"(narrow_f32(u)));
    double w = widen_f32(y32);
    w = fma(w, fma(-u, w, 1.0), w);
    double const t0 = v * w;
    double const t = fma(w, fma(-u, t0, v), t0);
    double const t2 = t * t;
    float const q = narrow_f32(t2);
    double const s = fma(t2, 0.2 - widen_f32(q * (1.0f / 7.0f - q * (1.0f / 9.0f))), -1.0 / 3.0);
    double const angle = fma(t * t2, s, t);
    if (j == 0) return copysign(angle, y);   // (-0 keeps its sign)
    double const k = __longlong_as_double(0x4338000000000000LL + j) - 6755399441055744.0;   // j as a double
    return fma(k, kTurnStep, fma(k, kTurnStepLo, angle));
}

}  // namespace rrea_dev
