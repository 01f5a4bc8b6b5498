// fvb_ieee.cuh -- FP64 quotients and square roots that round as IEEE division
// and sqrt do, in a form whose reciprocals are shared between the quotients
// of one denominator, for the kernels that reproduce the reference's
// arithmetic operation for operation.
//
// A quotient a / b from the rounded reciprocal y of b:
//   q = a y,  r = a - q b (exact in one fused multiply-add),  q' = q + r y,
// the remainder correction of P. Markstein ("Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990; Muller et al.,
// Handbook of Floating-Point Arithmetic, section 4.7): with y the reciprocal
// rounded to nearest, q' is the correctly rounded quotient.  frcp's y is
// rounded from a value good to 2^-60, so it can be the other neighbour where
// 1/b lies that close to a midpoint; q' then still rounds correctly unless
// a / b lies within about 2^-52 ulp of a midpoint itself.  The one place
// where such quotients are ordinary numbers is a b whose significand is all
// ones (a density one ulp under a power of two: 0.25 / b), which recip()
// rounds as it must.  A constant denominator needs no reciprocal at run time.
//
// The steps hold while nothing over- or underflows on the way, so callers
// collect the range tests below (integer compares of the high words, off the
// FP64 pipe) and evaluate the plain operators in the rare other case, whose
// infinities and NaN are then IEEE's own.  The sign of a zero quotient of a
// negative zero is the one thing not reproduced.
//
// On B200, 4.0e9 random pairs (exponents within 2^+-40) and 1.3e9 pairs of
// operands a few ulp around small integers and powers of two: no quotient and
// no root differs from the operator's.
#pragma once
#include "fvb_physics.cuh"

namespace fvb {

// exponent field and top mantissa bits of |x|
__device__ __forceinline__ unsigned hi_mag(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }

// |x| < 2^500 (false for infinities and NaN)
constexpr unsigned kHiMax = 0x5f300000u, kHiMin = 0x20b00000u;  // high words of 2^500 and 2^-500
__device__ __forceinline__ bool num_ok(double x) { return hi_mag(x) < kHiMax; }
__device__ __forceinline__ bool num_ok(double x, double y) { return max(hi_mag(x), hi_mag(y)) < kHiMax; }
__device__ __forceinline__ bool num_ok(double x, double y, double z)
{
    return max(max(hi_mag(x), hi_mag(y)), hi_mag(z)) < kHiMax;
}
// 2^-500 <= |x| < 2^500: a denominator, or the argument of a root
__device__ __forceinline__ bool den_ok(double x) { return hi_mag(x) - kHiMin < kHiMax - kHiMin; }

// 1 / b for quot(); den_ok(b).  For b = 2^k (1 - 2^-53) the reciprocal is
// 2^-k (1 + 2^-53 + ...), rounded to nearest 2^-k (1 + 2^-52): the last bit
// of the 2^-k that the iteration may give is set
__device__ __forceinline__ double recip(double b)
{
    const double y = frcp(b);
    const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
    const int ones = (lo & (hi | 0xfff00000u)) == 0xffffffffu ? 1 : 0;
    return __hiloint2double(__double2hiint(y), __double2loint(y) | ones);
}

// a / b from y = recip(b); num_ok(a) and den_ok(b)
__device__ __forceinline__ double quot(double a, double b, double y)
{
    const double q = a * y;
    return fma(fma(-q, b, a), y, q);
}

// sqrt(x), den_ok(x) and x > 0: fsqrt (fvb_physics.cuh) ends in the same
// kind of remainder correction
__device__ __forceinline__ double root(double x) { return fsqrt(x); }

}  // namespace fvb
