// Quotients and a power for kernels that are bound by instruction issue and divide many numerators by
// one divisor.
#pragma once

#include <cuda_runtime.h>

namespace gpx {

// a / b with y = 1 / b at hand, b > 0 (Markstein, IBM J. Res. Dev. 34, 1990): q = a y, corrected by its
// residual.  The sign of the residual is such that an exact quotient keeps the sign of its zero.  The
// result is the correctly rounded quotient if
//   float:  y is the correctly rounded reciprocal, 2^-24 <= b < 2^24, and a is zero or at least 2^-100 (the
//           residual has to be a float: its last bit is 2^-46 of a's first).  Smaller numerators may miss
//           it by one or two in the last place;
//   double: a and b hold float values (their quotient lies 2^-26 of an ulp or more from a tie, so a
//           reciprocal good to 2^-50 is enough).
// and a is finite and the quotient does not overflow.
__device__ __forceinline__ float div_by(float a, float b, float y) {
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(b, q, -a), -y, q);
}
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(b, q, -a), -y, q);
}
// The same for any a: the residual of an infinity is NaN, which the bound turns into a number, so that the
// infinity stays.  (A negative quotient that overflows comes out as NaN.)
__device__ __forceinline__ float div_by_any(float a, float b, float y) {
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(fminf(__fmaf_rn(b, q, -a), 3.402823466e38f), -y, q);
}
// The largest magnitude of three; NaN if one is.
__device__ __forceinline__ float largest(float a, float b, float c) {
    float most;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(most) : "f"(a), "f"(b), "f"(c));
    return most;
}
// Reciprocals of normal numbers: the hardware's approximation refined by Newton steps.  In float the result
// is the correctly rounded one for every mantissa (all 2^23 are compared with __frcp_rn by the tests);
// in double it is good to an ulp.
__device__ __forceinline__ float reciprocal(float b) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return __fmaf_rn(__fmaf_rn(-b, y, 1.f), y, y);
}
__device__ __forceinline__ double reciprocal(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
    return __fma_rn(__fma_rn(-b, y, 1.0), y, y);
}

// x^g for 2^-16 < x < 2^16 (|g| < 50), else pow: 2^(g log2 x), log2 from the series of artanh,
// log2 x = k + 2 / ln 2 * (s + s^3 / 3 + s^5 / 5 + ...), s = (m - 1) / (m + 1), x = 2^k m with m between
// sqrt(1/2) and sqrt 2 (|s| < 0.172, eleven terms), and the Taylor series of 2^f, |f| <= 1/2.  The product
// g k, the large part of the exponent, is kept with its rounding error, so the error does not grow
// with the exponent: 3e-16, against 2.2e-16 of pow (rounded to a float pressure both give the same for each of
// 5 million x).  pow() spends most of its instructions on cases (signs, zeros, infinities, exponents of
// any size) that take the call here.
__device__ __forceinline__ double power(double x, double g) {
    if (!(x > 1.52587890625e-05 && x < 65536.0)) return pow(x, g);
    const int hi = __double2hiint(x);
    const int k = (hi - 0x3fe6a09e) >> 20;  // the exponent that leaves the mantissa at or above sqrt(1/2)
    const double m = __hiloint2double(hi - (k << 20), __double2loint(x));
    const double below = __dsub_rn(m, 1.0), above = __dadd_rn(m, 1.0);
    const double s = __dmul_rn(below, reciprocal(above));
    const double z = __dmul_rn(s, s);
    double p = 1.0 / 21;
    p = __fma_rn(p, z, 1.0 / 19);
    p = __fma_rn(p, z, 1.0 / 17);
    p = __fma_rn(p, z, 1.0 / 15);
    p = __fma_rn(p, z, 1.0 / 13);
    p = __fma_rn(p, z, 1.0 / 11);
    p = __fma_rn(p, z, 1.0 / 9);
    p = __fma_rn(p, z, 1.0 / 7);
    p = __fma_rn(p, z, 1.0 / 5);
    p = __fma_rn(p, z, 1.0 / 3);
    const double frac = __dmul_rn(__fma_rn(__dmul_rn(p, z), s, s), 2.8853900817779268);  // 2 / ln 2
    // (integers to and from the low word of a double, by addition: the conversions are a sixteenth as fast)
    const double kd = __dsub_rn(__hiloint2double(0x43300000, k ^ (int)0x80000000), 4503601774854144.0);  // 2^52 + 2^31
    const double gk = __dmul_rn(g, kd), gk_err = __fma_rn(g, kd, -gk);
    const double shifted = __dadd_rn(__fma_rn(g, frac, gk), 6755399441055744.0);  // 1.5 * 2^52: rounds to an integer
    const double n = __dsub_rn(shifted, 6755399441055744.0);
    const double f = __dmul_rn(__dadd_rn(__dsub_rn(gk, n), __fma_rn(g, frac, gk_err)), 0.69314718055994531);
    double e = 1.0 / 6227020800.0;
    e = __fma_rn(e, f, 1.0 / 479001600.0);
    e = __fma_rn(e, f, 1.0 / 39916800.0);
    e = __fma_rn(e, f, 1.0 / 3628800.0);
    e = __fma_rn(e, f, 1.0 / 362880.0);
    e = __fma_rn(e, f, 1.0 / 40320.0);
    e = __fma_rn(e, f, 1.0 / 5040.0);
    e = __fma_rn(e, f, 1.0 / 720.0);
    e = __fma_rn(e, f, 1.0 / 120.0);
    e = __fma_rn(e, f, 1.0 / 24.0);
    e = __fma_rn(e, f, 1.0 / 6.0);
    e = __fma_rn(e, f, 0.5);
    e = __dadd_rn(1.0, __fma_rn(__dmul_rn(f, f), e, f));
    return __hiloint2double(__double2hiint(e) + (__double2loint(shifted) << 20), __double2loint(e));
}

}  // namespace gpx
