// fvb_physics.cuh -- pointwise physics and face numerics of the UP-ORDER +
// Ducros-blended HLLC/HLLE finite-volume Euler step, for the device.
//
// Everything works in the face-normal frame: a state is (rho, un, ut, p)
// with un the velocity along the face normal and ut the tangential one, and
// a flux comes back as (mass, normal momentum, tangential momentum, energy).
// An x-face takes (u, v) as (un, ut); a y-face takes (v, u) and the caller
// swaps the two momentum components back.  For the unit normals the
// reference uses, (1,0) and (0,1), this relabelling is exactly its rotation
// (fv_up7_ducros_2d.cu:245-248, :287-290).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fvb {

// Literal of type R spelled as the reference spells it (1.4f in the FP32
// solver, 1.4 in the FP64 one), so constants round identically.
#define FVB_LIT(R, x) (sizeof(R) == 4 ? R(x##f) : R(x))

template <class R> __device__ __forceinline__ R dsqrt(R x);
template <> __device__ __forceinline__ float dsqrt<float>(float x) { return sqrtf(x); }
template <> __device__ __forceinline__ double dsqrt<double>(double x) { return sqrt(x); }
template <class R> __device__ __forceinline__ R dmin(R a, R b);
template <> __device__ __forceinline__ float dmin<float>(float a, float b) { return fminf(a, b); }
template <> __device__ __forceinline__ double dmin<double>(double a, double b) { return fmin(a, b); }
template <class R> __device__ __forceinline__ R dmax(R a, R b);
template <> __device__ __forceinline__ float dmax<float>(float a, float b) { return fmaxf(a, b); }
template <> __device__ __forceinline__ double dmax<double>(double a, double b) { return fmax(a, b); }
template <class R> __device__ __forceinline__ R dabs(R a);
template <> __device__ __forceinline__ float dabs<float>(float a) { return fabsf(a); }
template <> __device__ __forceinline__ double dabs<double>(double a) { return fabs(a); }

// Min / max as one compare and a select, for the FP64 throughput paths.  An
// FP64 fmin / fmax is not one instruction on sm_100: with its NaN rules it
// issues about 7.5 (a compare, selects, integer and bit operations; ncu
// op-class counters of a loop of them), a compare and a select 3.  smax(a, b)
// is a > b ? a : b, smin(a, b) is a < b ? a : b: for finite operands the
// value fmax / fmin give (up to the sign of a zero result), and with a
// constant second operand (the clamps at 0, 1e-10, 1e-14) for every first
// operand, NaN included (NaN -> the constant).  FP32 keeps fminf / fmaxf,
// one instruction.
template <class R> __device__ __forceinline__ R smin(R a, R b);
template <> __device__ __forceinline__ float smin<float>(float a, float b) { return fminf(a, b); }
template <> __device__ __forceinline__ double smin<double>(double a, double b) { return a < b ? a : b; }
template <class R> __device__ __forceinline__ R smax(R a, R b);
template <> __device__ __forceinline__ float smax<float>(float a, float b) { return fmaxf(a, b); }
template <> __device__ __forceinline__ double smax<double>(double a, double b) { return a > b ? a : b; }

// floor used on reconstructed and updated rho and p: x > c ? x : c, so a
// NaN becomes the floor (fv_up7_ducros_2d.cu:421-422, :543-544); the same
// value as fmax(x, c) for every input
template <class R> __device__ __forceinline__ R floor14(R x)
{
    return smax<R>(x, FVB_LIT(R, 1e-14));
}

// Gas constants of one solver.  gm1 is formed as gamma - 1 at run time, the
// same subtraction the reference performs on its GAMMA_V literal.
template <class R> struct Gas {
    R gam, gm1;
};

// c = sqrt(max(gamma p / rho, 1e-14))           fv_up7_ducros_2d.cu:63-68
template <class R> __device__ __forceinline__ R sound(R p, R rho, const Gas<R> &gs)
{
    R cs2 = gs.gam * p / rho;
    const R c = FVB_LIT(R, 1e-14);
    return dsqrt<R>(cs2 > c ? cs2 : c);
}

// total energy of a primitive state            fv_up7_ducros_2d.cu:77, :251
template <class R> __device__ __forceinline__ R etot(R r, R a, R b, R p, const Gas<R> &gs)
{
    return p / gs.gm1 + FVB_LIT(R, 0.5) * r * (a * a + b * b);
}

// primitive <-> conserved                      fv_up7_ducros_2d.cu:71-88
template <class R> __device__ __forceinline__ void p2c(const R w[4], R c[4], const Gas<R> &gs)
{
    c[0] = w[0];
    c[1] = w[0] * w[1];
    c[2] = w[0] * w[2];
    c[3] = etot(w[0], w[1], w[2], w[3], gs);
}
template <class R> __device__ __forceinline__ void c2p(const R c[4], R w[4], const Gas<R> &gs)
{
    w[0] = c[0];
    w[1] = c[1] / c[0];
    w[2] = c[2] / c[0];
    w[3] = gs.gm1 * (c[3] - FVB_LIT(R, 0.5) * (c[1] * c[1] + c[2] * c[2]) / c[0]);
}

// Reciprocal and square root per arithmetic type.  Every argument on these
// paths is a positive normal number (densities and pressures are floored at
// 1e-14, wave-speed spans at 1e-10, sound speeds squared at 1e-14).
//
// FP64 reciprocal: the hardware seed (rcp.approx.ftz.f64, relative error
// 2^-19.9 measured) and one third-order Newton-Raphson step,
//   e = 1 - x y,  y' = y (1 + e + e^2),
// whose error is O(e^3) ~ 2^-60 before the last rounding (a higher-order
// Newton-Raphson iteration for 1/x, as in Muller et al., Handbook of
// Floating-Point Arithmetic).  Measured on B200 against the correctly
// rounded 1/x over 4M log-uniform samples in [1e-14, 1e14]: at most 1 ulp,
// 0.03% of samples not exact.  FVB_EXACT_RCP_SQRT=1 selects the correctly
// rounded library forms instead.
//
// FP64 square root: the hardware reciprocal-root seed (rsqrt.approx.ftz.f64,
// 2^-20.0 measured), one third-order step y' = y (1 + e/2 + 3e^2/8) with
// e = 1 - x y^2, then s = x y' and the residual correction
// s' = s + (x - s^2) y'/2 (the Newton step for sqrt through the reciprocal
// root, as in Markstein, IA-64 and Elementary Functions).  Measured: equal to the correctly rounded sqrt on all 4M samples.
//
// FP32: the hardware approximations (rcp / rsqrt, about 2 ulp).
#ifndef FVB_EXACT_RCP_SQRT
#define FVB_EXACT_RCP_SQRT 0
#endif
#if FVB_EXACT_RCP_SQRT
__device__ __forceinline__ double frcp(double x) { return __drcp_rn(x); }
__device__ __forceinline__ double fsqrt(double x) { return sqrt(x); }
#else
__device__ __forceinline__ double frcp(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double fsqrt(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    y = fma(y, e * fma(e, 0.375, 0.5), y);
    const double s = x * y;
    return fma(fma(-s, s, x), 0.5 * y, s);
}
#endif
__device__ __forceinline__ float frcp(float x) { return __fdividef(1.0f, x); }
__device__ __forceinline__ float fsqrt(float x) { return x * rsqrtf(x); }

}  // namespace fvb
