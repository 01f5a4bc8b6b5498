// fvb_face32.cuh -- the face numerics of the FP32 form as shipped: the
// reference's expression order, FP32 with the reconstruction's sums in FP64,
// quotients and roots rounded as IEEE division and sqrt round them.
//
// A quotient whose denominator is a constant or shared comes from the rounded
// reciprocal and the remainder correction of fvb_ieee.cuh, which gives the
// operator's bits where neither the quotient nor the remainder underflows or
// overflows (numerators from 2^-101 on, quotients from 2^-126); elsewhere the
// operator itself is evaluated.
#pragma once
#include "fvb_ieee.cuh"

namespace fvb {
namespace f32 {

// a / b from y = 1 / b rounded to nearest, b > 0
__device__ __forceinline__ float quot(float a, float b, float y)
{
    const float q = a * y, r = __fmaf_rn(q, b, -a);
    return __fmaf_rn(r, -y, q);
}
// twice the bits of the number below |a|, in order of magnitude; a zero: the most
__device__ __forceinline__ unsigned below(float a) { return (__float_as_uint(a) << 1) - 1u; }

struct Gas {
    float gam, gm1, ygm1;  // ygm1: 1 / gm1, rounded to nearest
};

// c = sqrt(max(gamma p / rho, 1e-14))           fv_up7_ducros_2d.cu:63-68
__device__ __forceinline__ float sound(float p, float rho, const Gas &gs)
{
    const float cs2 = gs.gam * p / rho;
    return sqrtf(cs2 > 1e-14f ? cs2 : 1e-14f);
}

// p / (gamma - 1): of a cell's pressure, whatever it is (gamma - 1 is at least
// 2^-23), and of a floored one, where only the overflow needs a look
__device__ __forceinline__ float over_gm1(float p, const Gas &gs)
{
    const bool in = __float_as_uint(p) - 0x0f800000u < 0x6f800000u - 0x0f800000u;  // 2^-96 ... 2^96
    return in ? quot(p, gs.gm1, gs.ygm1) : p / gs.gm1;
}
__device__ __forceinline__ float over_gm1_floored(float p, const Gas &gs)
{
    const float q = p * gs.ygm1, r = __fmaf_rn(q, gs.gm1, -p);
    return fabsf(r) <= 3.402823466e38f ? __fmaf_rn(r, -gs.ygm1, q) : q;  // (q is infinite, or a NaN)
}

// total energy of a normal-frame state from pe = p / (gamma - 1); the rounding
// of a fused multiply-add on the normal velocity is written out, so that it is
// the same wherever the energy is formed       fv_up7_ducros_2d.cu:77, :251
__device__ __forceinline__ float energy(float r, float un, float ut, float pe)
{
    return __fmaf_rn(0.5f * r, __fmaf_rn(un, un, __fmul_rn(ut, ut)), pe);
}

// UP7 face values from the 8-point stencil s (the face lies between s[3] and
// s[4]): sums in FP64, divided by 420 there, rounded to FP32
//                                               fv_up7_ducros_2d.cu:149-186
__device__ __forceinline__ void sums7(const double *s, double &tL, double &tR)
{
    tL = -3.0 * s[0] + 25.0 * s[1] - 101.0 * s[2] + 319.0 * s[3] + 214.0 * s[4] - 38.0 * s[5] + 4.0 * s[6];
    tR = 4.0 * s[1] - 38.0 * s[2] + 214.0 * s[3] + 319.0 * s[4] - 101.0 * s[5] + 25.0 * s[6] - 3.0 * s[7];
}
__device__ __forceinline__ void upface7(const double *s, float &vL, float &vR)
{
    double tL, tR;
    sums7(s, tL, tR);
    vL = (float)fvb::quot(tL, 420.0, 1.0 / 420.0);
    vR = (float)fvb::quot(tR, 420.0, 1.0 / 420.0);
}

// floor on rho and p: x > 1e-14 ? x : 1e-14     fv_up7_ducros_2d.cu:421-422
__device__ __forceinline__ float fl14(float x) { return fmaxf(x, 1e-14f); }

// HLLC with Davis wave-speed bounds, normal frame
//                                               fv_up7_ducros_2d.cu:237-292
__device__ __forceinline__ void hllc(const float L[4], const float Rr[4], float F[4], const Gas &gs)
{
    const float rL = L[0], uL = L[1], tL = L[2], pL = L[3];
    const float rR = Rr[0], uR = Rr[1], tR = Rr[2], pR = Rr[3];
    const float cL = sound(pL, rL, gs), cR = sound(pR, rR, gs);
    const float EL = energy(rL, uL, tL, over_gm1_floored(pL, gs)), ER = energy(rR, uR, tR, over_gm1_floored(pR, gs));
    const float SL = fminf(uL - cL, uR - cR);
    const float SR = fmaxf(uL + cL, uR + cR);
    if (SL >= 0.f) {
        F[0] = rL * uL; F[1] = rL * uL * uL + pL; F[2] = rL * uL * tL; F[3] = (EL + pL) * uL;
        return;
    }
    if (SR <= 0.f) {
        F[0] = rR * uR; F[1] = rR * uR * uR + pR; F[2] = rR * uR * tR; F[3] = (ER + pR) * uR;
        return;
    }
    const float dL = rL * (SL - uL), dR = rR * (SR - uR);
    const float Ss = (pR - pL + dL * uL - dR * uR) / (dL - dR);
    const bool left = (Ss >= 0.f);
    const float rK = left ? rL : rR, uK = left ? uL : uR, tK = left ? tL : tR;
    const float pK = left ? pL : pR, EK = left ? EL : ER, SK = left ? SL : SR;
    const float fact = rK * (SK - uK) / (SK - Ss);
    const float Us1 = fact * Ss, Us2 = fact * tK;
    const float Us3 = fact * (EK / rK + (Ss - uK) * (Ss + pK / (rK * (SK - uK))));
    F[0] = rK * uK + SK * (fact - rK);
    F[1] = rK * uK * uK + pK + SK * (Us1 - rK * uK);
    F[2] = rK * uK * tK + SK * (Us2 - rK * tK);
    F[3] = (EK + pK) * uK + SK * (Us3 - EK);
}

// HLLE on the two adjacent cell averages, normal frame, with the cells' sound
// speeds and energies                           fv_up7_ducros_2d.cu:296-328
__device__ __forceinline__ void hlle(const float L[4], const float Rr[4], float cL, float cR, float EL, float ER,
                                     float F[4])
{
    const float rL = L[0], uL = L[1], tL = L[2], pL = L[3];
    const float rR = Rr[0], uR = Rr[1], tR = Rr[2], pR = Rr[3];
    const float FL0 = rL * uL, FL1 = rL * uL * uL + pL, FL2 = rL * uL * tL, FL3 = (EL + pL) * uL;
    const float FR0 = rR * uR, FR1 = rR * uR * uR + pR, FR2 = rR * uR * tR, FR3 = (ER + pR) * uR;
    const float SL = fminf(uL - cL, uR - cR);
    const float SR = fmaxf(uL + cL, uR + cR);
    if (SL >= 0.f) { F[0] = FL0; F[1] = FL1; F[2] = FL2; F[3] = FL3; return; }
    if (SR <= 0.f) { F[0] = FR0; F[1] = FR1; F[2] = FR2; F[3] = FR3; return; }
    const float dS = fmaxf(SR - SL, 1e-10f);
    const float SRL = SR * SL;
    const float a0 = SR * FL0 - SL * FR0 + SRL * (rR - rL);
    const float a1 = SR * FL1 - SL * FR1 + SRL * (rR * uR - rL * uL);
    const float a2 = SR * FL2 - SL * FR2 + SRL * (rR * tR - rL * tL);
    const float a3 = SR * FL3 - SL * FR3 + SRL * (ER - EL);
    const float y = __frcp_rn(dS);
    F[0] = quot(a0, dS, y);
    F[1] = quot(a1, dS, y);
    F[2] = quot(a2, dS, y);
    F[3] = quot(a3, dS, y);
    // the least numerator against 2^-100 and, for the quotient, 2^-124 dS
    const unsigned least = min(min(below(a0), below(a1)), min(below(a2), below(a3)));
    const unsigned bound = max(0x1b000000u, __float_as_uint(dS * 0x1p-124f) << 1);
    if (!(fabsf(F[0]) + fabsf(F[1]) + fabsf(F[2]) + fabsf(F[3]) < 1e37f)) {
        F[0] = a0 / dS;
        F[1] = a1 / dS;
        F[2] = a2 / dS;
        F[3] = a3 / dS;
    } else if (least < bound) {
        // in FP64, where nothing underflows and whose quotient's 53 bits round to
        // FP32 as the quotient itself does (53 >= 2 * 24 + 2)
        const double D = dS, Y = recip(D);
        F[0] = (float)fvb::quot(a0, D, Y);
        F[1] = (float)fvb::quot(a1, D, Y);
        F[2] = (float)fvb::quot(a2, D, Y);
        F[3] = (float)fvb::quot(a3, D, Y);
    }
}

// pressure-jump sensor s = dp^2 / (dp^2 + 0.1 (pa+pb)^2)
//                                               fv_up7_ducros_2d.cu:114-133
__device__ __forceinline__ float ducros(float pa, float pb)
{
    const float dp = pb - pa, ps = pb + pa;
    return dp * dp / (dp * dp + 0.1f * ps * ps);
}

}  // namespace f32
}  // namespace fvb
