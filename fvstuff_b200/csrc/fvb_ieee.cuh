// fvb_ieee.cuh -- FP64 quotients and square roots that round as IEEE division
// and sqrt do, in a form whose reciprocals are shared between the quotients
// of one denominator, for the kernels that reproduce the reference's
// arithmetic operation for operation.
//
// A quotient a / b from the rounded reciprocal y of b:
//   q = a y,  r = q b - a (exact in one fused multiply-add),  q' = q - r y,
// the remainder correction of P. Markstein ("Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990; Muller et al.,
// Handbook of Floating-Point Arithmetic, section 4.7): with y the reciprocal
// rounded to nearest, q' is the correctly rounded quotient.  frcp's y is
// rounded from a value good to 2^-60, so where 1/b lies that close to a
// midpoint it can be the other neighbour, and q' can then be the wrong one of
// two for numerators whose quotient lies within 2^-53 ulp of a midpoint itself:
// one or two significands in 2^53 for such a b.  That no such pair is met rests
// on tests, not on the theorem.  The one place where such quotients are
// ordinary numbers is a b whose significand is all ones (a density one ulp
// under a power of two: 0.25 / b), which recip() rounds as it must.  A constant
// denominator needs no reciprocal at run time.
//
// The steps hold while nothing over- or underflows on the way, the remainder
// included, so callers collect the range tests below (integer operations on the
// bits, off the FP64 pipe) and evaluate the plain operators in the rare other
// case: a denominator outside [2^-500, 2^100), a numerator that is neither zero
// nor in [2^-900, 2^500), infinities and NaN.  A caller may leave the lower
// bound out where a quotient that small cannot reach its result.  Zero quotients
// have the operator's sign for positive denominators (quot) and for zero
// numerators that are +0 (squot).
//
// On B200, 4.0e9 random pairs (exponents within 2^+-40) and 1.3e9 pairs of
// operands a few ulp around small integers and powers of two: no quotient and
// no root differs from the operator's.
#pragma once
#include "fvb_physics.cuh"

namespace fvb {

// exponent field and top mantissa bits of |x|
__device__ __forceinline__ unsigned hi_mag(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
// the same of the number below |x|, and 0x7fffffff for a zero
__device__ __forceinline__ unsigned hi_below(double x)
{
    return (unsigned)((unsigned long long)(__double_as_longlong(x) - 1) >> 32) & 0x7fffffffu;
}

// high words of 2^-900 and 2^500 (numerators), 2^-500 and 2^100 (denominators)
constexpr unsigned kNumMin = 0x07b00000u, kNumMax = 0x5f300000u, kDenMin = 0x20b00000u, kDenMax = 0x46300000u;
// |x| < 2^500 (false for infinities and NaN)
__device__ __forceinline__ bool fin_ok(double x) { return hi_mag(x) < kNumMax; }
__device__ __forceinline__ bool fin_ok(double x, double y) { return max(hi_mag(x), hi_mag(y)) < kNumMax; }
// a numerator: zero, or 2^-900 < |x| < 2^500
__device__ __forceinline__ bool num_ok(double x) { return fin_ok(x) && hi_below(x) >= kNumMin; }
__device__ __forceinline__ bool num_ok(double x, double y)
{
    return fin_ok(x, y) && min(hi_below(x), hi_below(y)) >= kNumMin;
}
// a denominator, or the argument of a root: 2^-500 <= |x| < 2^100; pos_ok: and x > 0
__device__ __forceinline__ bool den_ok(double x) { return hi_mag(x) - kDenMin < kDenMax - kDenMin; }
__device__ __forceinline__ bool pos_ok(double x) { return (unsigned)__double2hiint(x) - kDenMin < kDenMax - kDenMin; }

// 1 / b for quot() and squot(); den_ok(b).  For b = 2^k (1 - 2^-53) the reciprocal is
// 2^-k (1 + 2^-53 + ...), rounded to nearest 2^-k (1 + 2^-52): the last bit
// of the 2^-k that the iteration may give is set
__device__ __forceinline__ double recip(double b)
{
    const double y = frcp(b);
    const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
    const int ones = (lo & (hi | 0xfff00000u)) == 0xffffffffu ? 1 : 0;
    return __hiloint2double(__double2hiint(y), __double2loint(y) | ones);
}

// a / b from y = recip(b), b > 0; num_ok(a) and pos_ok(b)
__device__ __forceinline__ double quot(double a, double b, double y)
{
    const double q = a * y;
    const double r = fma(q, b, -a);
    return fma(r, -y, q);
}
// the same for b of either sign, a not -0; num_ok(a) and den_ok(b)
__device__ __forceinline__ double squot(double a, double b, double y)
{
    const double q = a * y;
    return fma(fma(-q, b, a), y, q);
}

// A numerator below num_ok's range, where remainders and quotients underflow:
// is there one among these?
__device__ __forceinline__ bool is_small(double x) { return hi_below(x) < kNumMin; }
__device__ __forceinline__ bool is_small(double x, double y) { return min(hi_below(x), hi_below(y)) < kNumMin; }
__device__ __forceinline__ bool is_small(double x, double y, double z, double w)
{
    return min(min(hi_below(x), hi_below(y)), min(hi_below(z), hi_below(w))) < kNumMin;
}
// a / b for such an a (or a zero), y = recip(b), den_ok(b): as above on 2^600 a,
// where nothing underflows.  Where the quotient itself is subnormal, its
// rounding to 53 bits is rounded again to a whole number k of 2^-1074, and the
// remainder of k (exact) says whether that is the nearest.
__device__ __forceinline__ double small_quot(double a, double b, double y)
{
    const double A = a * 0x1p600, q = squot(A, b, y);
    if (fabs(q) >= 0x1p-422) return q * 0x1p-600;
    double k = rint(q * 0x1p474);
    const double r = fma(-k, b, A * 0x1p474);
    if (2.0 * fabs(r) > fabs(b)) k += (r > 0.0) == (b > 0.0) ? 1.0 : -1.0;
    return copysign(k * 0x1p-500 * 0x1p-574, q);
}

// sqrt(x), pos_ok(x): fsqrt (fvb_physics.cuh) ends in the same
// kind of remainder correction
__device__ __forceinline__ double root(double x) { return fsqrt(x); }

}  // namespace fvb
