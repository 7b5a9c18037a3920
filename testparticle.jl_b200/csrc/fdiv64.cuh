// fdiv64.cuh -- float64 square roots and quotients that share a reciprocal.
//
// The float64 kernels divide several numerators by one denominator (a vector
// by its norm, the rotation vector by 1 + |t|^2, ...).  A division of its own
// per numerator made half of the float64-pipe work of a guiding-centre
// right-hand side and a third of a Multistep step.  Here one reciprocal is
// formed as an unevaluated sum hi + lo and every quotient then costs one
// multiply and one fma:
//
//   reciprocal   hi from a float estimate and one third-order step, then
//                lo = (1 - b hi) hi: hi + lo = 1/b to about 2^-102;
//   quotient     q = fma(a, hi, a * lo), the multiplication by a two-word
//                constant of N. Brisebarre, J.-M. Muller, S. Raina,
//                "Accelerating correctly rounded floating-point division when
//                the divisor is known in advance", IEEE Trans. Comput. 53
//                (2004);
//   square root  g = x y with y = 1/sqrt(x), then one Newton correction
//                fma(x - g^2, y/2, g) (P. Markstein, IBM J. Res. Dev. 34
//                (1990)).
//
// The value before the last rounding is within 2^-100 of the exact one, so
// the result equals the correctly rounded `/` and `sqrt` unless that lies
// within 2^-100 (relative) of the midpoint of two float64 numbers.  Quotients
// below 2^-900 may differ in their last bit, and a zero quotient may have the
// other sign.  Callers check the denominator (in_range64); zero, infinite,
// NaN and extreme ones take `/` and sqrt().
#pragma once

namespace tpb {

// 2^-100 <= x < 2^100 (false for negative, infinite and NaN): the exponent
// range in which the float estimates are normal and nothing below over- or
// underflows
__device__ __forceinline__ bool in_range64(double x) {
    return (unsigned)(__double2hiint(x) - 0x39B00000) < 0x0C800000u;
}

// 1/b to about one unit in the last place (b in range)
__device__ __forceinline__ double rcp64(double b) {
    const double y = (double)__frcp_rn((float)b);
    const double e = fma(-b, y, 1.0);
    return fma(fma(e, e, e), y, y);
}

// 1/sqrt(x) to about one unit in the last place (x in range)
__device__ __forceinline__ double rsqrt64(double x) {
    const double y = (double)rsqrtf((float)x);
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// sqrt(x) from y = rsqrt64(x)
__device__ __forceinline__ double sqrt64(double x, double y) {
    const double g = x * y;
    return fma(fma(-g, g, x), 0.5 * y, g);
}

// the denominator b with its reciprocal hi (about one ulp) completed to two words
struct Rec64 {
    double hi, lo;
};
__device__ __forceinline__ Rec64 rec64(double b, double hi) { return {hi, fma(-b, hi, 1.0) * hi}; }
__device__ __forceinline__ double quot64(double a, Rec64 r) { return fma(a, r.hi, a * r.lo); }

// x / 3 and x / 15 (1/3 and 1/15 as two words; x finite)
__device__ __forceinline__ double third64(double x) { return quot64(x, {1.0 / 3.0, 0x1.5555555555555p-56}); }
__device__ __forceinline__ double fifteenth64(double x) { return quot64(x, {1.0 / 15.0, 0x1.1111111111111p-60}); }

}  // namespace tpb
