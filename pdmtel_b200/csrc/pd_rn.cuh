// Correctly rounded FP64 square root, reciprocal and quotient without
// branches, for kernels whose results must be those of IEEE sqrt and / bit for
// bit.  The compiler's own sequences test for special operands and branch on
// every use, so several of them in one thread do not overlap; these are
// straight lines of FMAs that interleave, one reciprocal serves several
// quotients by the same divisor, and the caller tests the operands' range once
// (rn_range, rn_quotient_ok) and takes the plain operators outside it.
//
// Square root: the coupled iteration of Goldschmidt (g -> sqrt a, h -> 1 / (2
// sqrt a)) from a hardware seed of about 20 bits, twice, then one residual
// correction g + h (a - g^2) (P. Markstein, "Software division and square
// root using Goldschmidt's algorithms", RNC 2004).  Before the last rounding
// the result is within 2^-100 of sqrt a (a in [1, 4)), so it can only round
// to the wrong neighbour if a lies within 152 * 2^-106 of the square of a
// midpoint: a finite list of operands (the solutions of m^2 = j modulo 2^54
// for small |j|).
//
// Reciprocal and quotient: Newton's y + y (1 - b y) and Markstein's q + y (a -
// b q) with q = a y (Muller et al., Handbook of Floating-Point Arithmetic,
// section on division by Newton-Raphson with an FMA).  For b in [1, 2) the
// reciprocal satisfies |y - 1/b| <= 2^-54 (1 + 2^-47).  If a/b is within reach
// of a midpoint m, then q is one of the two neighbours of m because |a y -
// a/b| < 2^-52, so |a - b q| is b 2^-53 to first order and the result before
// rounding is within b 2^-107 of a/b, while a/b != m differs from m by at
// least 2^-105 / b: it rounds to the right side for every b below 2 - 2^-46.
// For b = 2 - 2^-52 the exact step from y = 1/2 ends on a tie that rounds to
// 1/2 instead of 1/2 + 2^-53; the estimate before the last step therefore has
// its lowest bit set.  tests/test_rn.py runs the operands that these bounds
// leave open, and random ones, against IEEE results.
#pragma once

namespace pd {

__device__ __forceinline__ double rn_pow2(double v, int e) {  // v 2^e, v and the result normal
    return __hiloint2double(__double2hiint(v) + (e << 20), __double2loint(v));
}

// s = sqrt(a) and y = 1/s, both rounded to nearest (y: see above); a in
// [2^-400, 2^400]
__device__ __forceinline__ void rn_sqrt_rcp(double a, double& s, double& y) {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(a));
    double g = a * y0, h = rn_pow2(y0, -1);
    double e = fma(-g, h, 0.5);
    g = fma(g, e, g);
    h = fma(h, e, h);
    e = fma(-g, h, 0.5);
    g = fma(g, e, g);
    h = fma(h, e, h);
    s = fma(fma(-g, g, a), h, g);
    y = __hiloint2double(__double2hiint(h) + (1 << 20), __double2loint(h) | 1);
    y = fma(fma(-s, y, 1.0), y, y);
}

// y = 1/b rounded to nearest as in rn_sqrt_rcp from an estimate y0 with a
// relative error below 2^-50; b and 1/b normal
__device__ __forceinline__ double rn_rcp(double b, double y0) {
    const double y = __hiloint2double(__double2hiint(y0), __double2loint(y0) | 1);
    return fma(fma(-b, y, 1.0), y, y);
}

// 1 / sqrt(a) within half a unit in the last place and 2^-15 of one, a in
// rn_range: with e = 1 - a y^2 for the seed y, |e| below 2^-18, it is y (1 + e/2 +
// 3 e^2/8 + 5 e^3/16 + ...), where e has the rounding of a y taken out and is
// good to 2^-72, and the terms left out are below 2^-73.
__device__ __forceinline__ double rsqrt_near(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double g = a * y;
    const double e = fma(-fma(a, y, -g), y, fma(-g, y, 1.0));
    return fma(y, e * fma(e, fma(e, 0.3125, 0.375), 0.5), y);
}

// a / b with y = 1/b, b > 0; a zero or rn_quotient_ok (the quotient of a zero
// is +0)
__device__ __forceinline__ double rn_div(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}
// a / b without a reciprocal at hand, b > 0 in rn_range, within half a unit in
// the last place and 2^-49 of one (rn_div's last step on a reciprocal that is
// rounded from within 2^-59); an a outside rn_quotient_ok may end one unit off
__device__ __forceinline__ double quotient_near(double a, double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    return rn_div(a, b, fma(y, fma(e, e, e), y));
}
// the same as rn_div with the sign of a zero kept (any quotient has the sign of a)
__device__ __forceinline__ double rn_div_signed(double a, double b, double y) {
    const double q = rn_div(a, b, y);
    return __hiloint2double((__double2hiint(q) & 0x7fffffff) | (__double2hiint(a) & 0x80000000), __double2loint(q));
}

// whether a positive operand of rn_sqrt_rcp is in [2^-400, 2^400)
__device__ __forceinline__ bool rn_range(double a) {
    return (unsigned)__double2hiint(a) - (623u << 20) < (800u << 20);
}
// the same for [2^-200, 2^200), whose third powers are in range too
__device__ __forceinline__ bool rn_range_cubed(double a) {
    return (unsigned)__double2hiint(a) - (823u << 20) < (400u << 20);
}
// distance of |a| from the range [2^-500, 2^500) of dividends, as an unsigned
// number: below rn_span inside; zeros count as inside
constexpr unsigned rn_span = 1000u << 21;
__device__ __forceinline__ unsigned rn_dividend(double a) {
    const unsigned h = (unsigned)__double2hiint(a) << 1;
    return (h | (unsigned)__double2loint(a)) ? h - (523u << 21) : 0u;
}
__device__ __forceinline__ bool rn_quotient_ok(double a) { return rn_dividend(a) < rn_span; }

}  // namespace pd
