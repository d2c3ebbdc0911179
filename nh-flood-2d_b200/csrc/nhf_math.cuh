// Deterministic FP64 natural logarithm and exponential for the step kernels.
//
// The friction factor needs max(wh, 1e-5) ** (7.0 / 3.0) with the exponent
// rounded to F32 as Taichi rounds Python float constants
// (solver_compact.py:456,478), and Horton capacity needs
// exp(-k * t / 3600.) (solver_compact.py:545-547). Both are evaluated here in
// FP64 from IEEE basic operations only and rounded once to F32, so that the
// result does not depend on a vendor math library and is reproduced bit for
// bit by the CPU restatement used in the tests. Build with --fmad=false.
//
// The F32 step takes friction_pow and horton_exp below: shorter evaluations of
// the same two values that give the same F32 bits (Ziv's rounding test, the
// full evaluation where the short one cannot decide the rounding).
//
// Methods (published):
//  ln  : x = m * 2^e, m in [sqrt(1/2), sqrt(2)]; ln m = 2 atanh(s) with
//        s = (m - 1) / (m + 1) and the odd Taylor series of atanh to s^25;
//        e * ln2 is added through the Cody–Waite hi/lo split of ln2 (the
//        fdlibm constants).
//  exp : Cody–Waite reduction y = n ln2 + r, |r| <= ln2 / 2; Taylor series of
//        e^r to degree 13 (Horner); 2^n applied through the exponent field.
#pragma once
#include <cstdint>

namespace nhf {

__device__ __forceinline__ double ln_f64(double x)
{
    if (x != x) return x;
    if (x <= 0.0) return x == 0.0 ? -__longlong_as_double(0x7ff0000000000000LL)
                                  : __longlong_as_double(0x7ff8000000000000LL);
    if (x == __longlong_as_double(0x7ff0000000000000LL)) return x;
    uint64_t b = (uint64_t)__double_as_longlong(x);
    int e = (int)((b >> 52) & 0x7ff);
    if (e == 0) {
        x = x * 0x1p54;
        b = (uint64_t)__double_as_longlong(x);
        e = (int)((b >> 52) & 0x7ff) - 54;
    }
    e -= 1023;
    double m = __longlong_as_double((long long)((b & 0x000fffffffffffffULL) | 0x3ff0000000000000ULL));
    if (m > 0x1.6a09e667f3bcdp+0) { m = m * 0.5; e += 1; }
    double s = (m - 1.0) / (m + 1.0);
    double z = s * s;
    double p = 0x1.47ae147ae147bp-5;
    p = p * z + 0x1.642c8590b2164p-5;
    p = p * z + 0x1.8618618618618p-5;
    p = p * z + 0x1.af286bca1af28p-5;
    p = p * z + 0x1.e1e1e1e1e1e1ep-5;
    p = p * z + 0x1.1111111111111p-4;
    p = p * z + 0x1.3b13b13b13b14p-4;
    p = p * z + 0x1.745d1745d1746p-4;
    p = p * z + 0x1.c71c71c71c71cp-4;
    p = p * z + 0x1.2492492492492p-3;
    p = p * z + 0x1.999999999999ap-3;
    p = p * z + 0x1.5555555555555p-2;
    p = p * z + 1.0;
    double lnm = 2.0 * s * p;
    double de = (double)e;
    return de * 0x1.62e42fee00000p-1 + (de * 0x1.a39ef35793c76p-33 + lnm);
}

__device__ __forceinline__ double exp_f64(double y)
{
    if (y != y) return y;
    if (y > 709.0) return __longlong_as_double(0x7ff0000000000000LL);
    if (y < -745.0) return 0.0;
    double n = floor(y * 0x1.71547652b82fep+0 + 0.5);
    double r = (y - n * 0x1.62e42fee00000p-1) - n * 0x1.a39ef35793c76p-33;
    double p = 0x1.6124613a86d09p-33;
    p = p * r + 0x1.1eed8eff8d898p-29;
    p = p * r + 0x1.ae64567f544e4p-26;
    p = p * r + 0x1.27e4fb7789f5cp-22;
    p = p * r + 0x1.71de3a556c734p-19;
    p = p * r + 0x1.a01a01a01a01ap-16;
    p = p * r + 0x1.a01a01a01a01ap-13;
    p = p * r + 0x1.6c16c16c16c17p-10;
    p = p * r + 0x1.1111111111111p-7;
    p = p * r + 0x1.5555555555555p-5;
    p = p * r + 0x1.5555555555555p-3;
    p = p * r + 0.5;
    p = p * r + 1.0;
    p = p * r + 1.0;
    int ni = (int)n;
    if (ni < -1000) { p = p * 0x1p-600; ni += 600; }
    if (ni > 1000) { p = p * 0x1p600; ni -= 600; }
    return p * __longlong_as_double((long long)((uint64_t)(ni + 1023) << 52));
}

// x ** y for the F32 friction base, rounded once from FP64.
__device__ __forceinline__ float pow_f32(float x, float y)
{
    if (x != x) return x;
    if (x == 0.0f) return 0.0f;
    return (float)exp_f64((double)y * ln_f64((double)x));
}

__device__ __forceinline__ float exp_f32(float a) { return (float)exp_f64((double)a); }

__device__ __forceinline__ float approx_lg2(float x)
{
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float approx_ex2(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float approx_rcp(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float approx_sqrt(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Whether an FP64 value lies so near the midpoint of two F32 neighbours that a
// relative error of 2^-40 (kOpenUnits FP64 units, at least) could change its
// rounding to F32.
constexpr uint32_t kOpenUnits = 8192;
__device__ __forceinline__ bool rounding_open(double v)
{
    const uint32_t below = (uint32_t)__double_as_longlong(v) & 0x1fffffffu;  // the 29 bits F32 drops
    return below - (0x10000000u - kOpenUnits) < 2 * kOpenUnits;
}

// The full evaluations behind the rounding test, out of line: about one in
// 2^15 arguments gets here.
static __device__ __noinline__ float pow73_full(float x) { return pow_f32(x, 0x1.2aaaaap+1f); }
static __device__ __noinline__ float exp_full(float a) { return exp_f32(a); }

// x ** f32(7/3) for the friction factor, x >= 1e-5: the value of
// pow_f32(x, 7/3). With the F32 exponent y = 7/3 - c (c = 7.947e-8),
// x^y = x^3 (x^(-1/3))^2 x^(-c). x^(-1/3) is an F32 estimate s (relative
// error below 2^-18) corrected by the binomial series of (1 - t)^(-1/3) at
// t = 1 - x s^3, whose third term is under 2^-50; x^(-c) is 1 + w + w^2 / 2 at
// w = -c ln x, |w| < 2^-19.7, in F32: the logarithm's 2^-22 and three roundings
// make at most 2^-40.9 of the value, at 2^20, and less than that at smaller x.
// 11 FP64 operations instead of about 85, and a shorter chain, which is what a small step's
// momentum waits for. Measured together with horton_exp, cfl_above and
// speed_not_above (nhf_common.cuh), 32 steps: 256 x 256 cells 732 to 682 us,
// 2048 x 1531 cells with Horton soil 9.34 to 7.95 ms, quadtree of 1.36 M cells
// 5.98 to 5.36 ms.
__device__ __forceinline__ float friction_pow(float x)
{
    const float lg = approx_lg2(x);
    const double xd = (double)x, s = (double)approx_ex2(lg * -0x1.555556p-2f);
    const double t = __fma_rn(-xd, s * s * s, 1.0);
    const double r = __fma_rn(s * t, __fma_rn(t, 2.0 / 9.0, 1.0 / 3.0), s);
    const double a = xd * r;
    const double v = (xd * xd) * (a * r);
    const float w = lg * (float)(-(7.0 / 3.0 - 0x1.2aaaaap+1) * 0.693147180559945309);
    const double p = __fma_rn(v, (double)fmaf(0.5f * w, w, w), v);
    if (rounding_open(p) || !(x < 0x1p20f)) return pow73_full(x);
    return (float)p;
}

// exp(a) of the Horton capacity, a <= 0: the value of exp_f32(a). One-step
// reduction by ln 2 (|a| < 80: error under 2^-46) and the Taylor series to
// degree 10 (remainder under 2^-41.5 of the value for |r| <= ln2 / 2) with fused
// multiply-adds: 14 FP64 operations instead of about 40.
__device__ __forceinline__ float horton_exp(float a)
{
    const float n = rintf(a * 0x1.715476p+0f);
    const double r = __fma_rn((double)n, -0x1.62e42fefa39efp-1, (double)a);
    double p = 1.0 / 3628800.0;
    p = __fma_rn(p, r, 1.0 / 362880.0);
    p = __fma_rn(p, r, 1.0 / 40320.0);
    p = __fma_rn(p, r, 1.0 / 5040.0);
    p = __fma_rn(p, r, 1.0 / 720.0);
    p = __fma_rn(p, r, 1.0 / 120.0);
    p = __fma_rn(p, r, 1.0 / 24.0);
    p = __fma_rn(p, r, 1.0 / 6.0);
    p = __fma_rn(p, r, 0.5);
    p = __fma_rn(p, r, 1.0);
    p = __fma_rn(p, r, 1.0);
    p *= __longlong_as_double((long long)((int)n + 1023) << 52);
    if (rounding_open(p) || !(a > -80.0f && a <= 0.0f)) return exp_full(a);
    return (float)p;
}

// The friction power x^(7/3) and the Horton exponential in the build's physics
// type: rounded once to F32 (the power with the exponent f32(7/3)), or in the FP64
// build kept in double.
#ifdef NHF_REAL_DOUBLE
__device__ __forceinline__ double friction_pow_real(double x)
{
    if (x != x) return x;
    if (x == 0.0) return 0.0;
    return exp_f64(7.0 / 3.0 * ln_f64(x));
}
__device__ __forceinline__ double exp_real(double a) { return exp_f64(a); }
#else
__device__ __forceinline__ float friction_pow_real(float x) { return friction_pow(x); }
__device__ __forceinline__ float exp_real(float a) { return horton_exp(a); }
#endif

}  // namespace nhf
