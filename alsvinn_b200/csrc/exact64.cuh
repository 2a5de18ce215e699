// Correctly rounded FP64 division and square root without branches, for
// operands in a stated range.
//
// The FP64 method has to give the reference's bits, so every quotient and
// root must be the correctly rounded one.  The compiler's operators give
// that for every operand, but each one carries its own range test and a
// branch to a slow path: about 19 instructions of which 8 are FP64, and the
// branch keeps the ~40 quotients and ~10 roots of a cell and stage from
// overlapping.  The routines below are straight-line FMA sequences that
// share a reciprocal between the quotients of one denominator; the caller
// tests the ranges of a whole face once (euler_exact64.cuh) and takes the
// compiler's operators when the test fails.
//
// Quotients.  With y = RN(1/d), q = RN(a y), r = RN(a - d q) the value
// RN(q + r y) is RN(a/d) (P. Markstein, IBM J. Res. Dev. 34 (1990) 111;
// N. Brisebarre, J.-M. Muller, S. K. Raina, IEEE Trans. Comput. 53 (2004)
// 1069: one multiplication and two FMAs when the correctly rounded
// reciprocal is at hand), as long as nothing over- or underflows.
//
// Reciprocals.  The hardware's approximation (rcp.approx.ftz.f64, relative
// error e, measured below 2^-19.9) takes one third-order step,
// y (1 + e + e^2), rounded up, and one Newton step on the exact residual
// 1 - d y, rounded to nearest.  For d in [1, 2) the first step leaves y
// above 1/d by f = d y - 1 < 2^-52 (or below by less than 2^-59), and the
// second aims at (1 - f^2)/d, just below 1/d.  That rounds wrongly only if a
// midpoint m lies between the two.  1 - m d is then a positive multiple of
// 2^-106; but y, rounded up from just above m, is m + 2^-54, so
// f^2 = (d/2)^2 2^-106 < 2^-106 and (1 - f^2)/d is still above m.
//
// Roots.  From the hardware's y ~ 1/sqrt(x): e = 1 - x y^2, the third-order
// factor 1 + e/2 + 3 e^2/8 applied to y and to x y, then one Markstein step
// RN(g + (x - g^2) / (2 sqrt x)).  g is within 1.1 units in the last place,
// so the residual is exact where the rounding is decided, at half a unit
// from g: there x = G^2 + D with integers G (g in units of its last place)
// and D, and rounding turns on D <= G or D >= G + 1.  x is a multiple of
// 2^52 of those units squared, so D = G + 1 and D = G - 1 (odd totals)
// cannot occur and D = G only for the mantissas 1 + 2^-52 and all ones;
// every other D leaves a margin of 1.5/G, above the error of y.
//
// Zero numerators keep their sign: with d > 0 the residual is formed as
// d q - a, exactly +0 when q is exact, and subtracted.
#pragma once

#include <cuda_runtime.h>

namespace als {

// 1/d for 2^-500 <= d <= 2^500.
__device__ __forceinline__ double rcp64(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    double e = __fma_rn(-d, y, 1.0);
    e = __fma_rn(e, e, e);
    y = __fma_ru(y, e, y);
    e = __fma_rn(-d, y, 1.0);
    return __fma_rn(y, e, y);
}

// a/d for d > 0 as above, y = rcp64(d), and a = +-0 or 2^-900 <= |a| with
// 2^-1000 <= |a/d| <= 2^1000.
__device__ __forceinline__ double quot64(double a, double d, double y) {
    const double q = a * y;
    const double r = __fma_rn(q, d, -a);
    return __fma_rn(-r, y, q);
}

// sqrt(x) for 2^-500 <= x <= 2^500.
__device__ __forceinline__ double sqrt64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = __fma_rn(-x, y * y, 1.0);
    const double c = e * __fma_rn(e, 0.375, 0.5);
    const double t = x * y;
    const double g = __fma_rn(t, c, t);
    y = __fma_rn(y, c, y);
    // y/2: one off the exponent
    const double h = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
    return __fma_rn(__fma_rn(-g, g, x), h, g);
}

// Range tests on the high words.  A positive double lies in [2^a, 2^b) when
// its high word, as a signed integer, lies between those of 2^a and 2^b;
// negative values, infinities and NaNs fall outside.
__host__ __device__ constexpr int hi_pow2(int e) {
    return (1023 + e) << 20;
}

// Order key of a numerator: small for tiny nonzero values, above every
// threshold for +-0.
__device__ __forceinline__ unsigned numerator_key(double a) {
    const unsigned low = min(unsigned(__double2loint(a)), 1u);
    return ((unsigned(__double2hiint(a)) & 0x7fffffffu) | low) - 1u;
}

// a with the sign bit `s` (0 or 0x80000000) flipped in.
__device__ __forceinline__ double flip_sign(double a, int s) {
    return __hiloint2double(__double2hiint(a) ^ s, __double2loint(a));
}

} // namespace als
