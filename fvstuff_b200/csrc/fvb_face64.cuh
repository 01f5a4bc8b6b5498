// fvb_face64.cuh -- FP64 cell and face arithmetic of the UP-ORDER +
// Ducros-blended HLLC/HLLE path (fvb_stage64.cuh).
//
// Normal frame as in fvb_physics.cuh.  Every fused multiply-add is written
// out and the file that includes this one is compiled with -fmad=false, so
// the value of a face does not depend on which of a thread's faces it is, on
// the tile shape or on the kernel's other template arguments.
//
// Forms (each exact in real arithmetic; a few ulp from the reference's order):
//   * UP weights pre-divided by their denominator;
//   * c = gamma p rsqrt(gamma p rho), floored at 1e-7 (c^2 at 1e-14), without
//     a division;
//   * HLLC in star variables: with S the contact speed (u_K when the fan is
//     supersonic), d_K = rho_K (S_K - u_K), p* = p_K + d_K (S - u_K),
//     rho* = d_K / (S_K - S) and E* = ((S - u_K)(d_K S + p_K) + E_K (S_K - u_K)) /
//     (S_K - S), the flux is (rho* S, rho* S^2 + p*, rho* S u_K,t, (E* + p*) S);
//   * HLLE: with kL = a (uL - SL-), kR = b (uR - SR+), a = SR+/(SR+ - SL-),
//     b = -SL-/(SR+ - SL-), the average is rho_L kL + rho_R kR and so on per
//     component; the sensor's weight is folded into a and b.
// 159 FP64 operations a UP7 face, four of them compares, beside five seeds.
#pragma once
#include "fvb_physics.cuh"

namespace fvb {
namespace f64 {

struct Gas {
    double gam, igm1, gm1;  // gamma, 1/(gamma-1), gamma-1
};

// floor used on reconstructed and updated rho and p (NaN -> the floor): x > C by
// the bits, C < x <= inf as one unsigned range, on the ALU instead of the FP64
// pipe
template <unsigned long long C>  // the bits of the floor
__device__ __forceinline__ bool above(double x)
{
    constexpr unsigned long long lo = C + 1, span = 0x7ff0000000000000ull - lo;
    return (unsigned)(((unsigned long long)__double_as_longlong(x) - lo) >> 32) <= (unsigned)(span >> 32);
}
__device__ __forceinline__ double fl14(double x) { return above<0x3d06849b86a12b9bull>(x) ? x : 1e-14; }

// gp / sqrt(gp r) = sqrt(gp / r): reciprocal root from the hardware seed
// (2^-20) and one third-order step
__device__ __forceinline__ double snd_raw(double gp, double r)
{
#if FVB_EXACT_RCP_SQRT
    return sqrt(gp / r);
#else
    const double x = gp * r;
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    y = fma(y, e * fma(e, 0.375, 0.5), y);
    return gp * y;
#endif
}
__device__ __forceinline__ double snd(double gp, double r)
{
    const double c = snd_raw(gp, r);
    return above<0x3e7ad7f29abcaf48ull>(c) ? c : 1e-7;
}

__device__ __forceinline__ double energy(double r, double a, double b, double p, const Gas &gs)
{
    return fma(0.5 * r, fma(a, a, b * b), p * gs.igm1);
}

template <int N>
__device__ __forceinline__ double dot(const double (&w)[N], const double *s)
{
    double a = w[0] * s[0];
#pragma unroll
    for (int k = 1; k < N; ++k) a = fma(w[k], s[k], a);
    return a;
}

// face values from the 2g-point stencil s[0 .. 2g-1] (the face lies between
// s[g-1] and s[g])                              fv_up7_ducros_2d.cu:149-186
template <int ORDER>
__device__ __forceinline__ void upface(const double *s, double &vL, double &vR)
{
    if constexpr (ORDER == 3) {
        constexpr double l[3] = {-1. / 6., 5. / 6., 2. / 6.}, r[3] = {2. / 6., 5. / 6., -1. / 6.};
        vL = dot<3>(l, s);
        vR = dot<3>(r, s + 1);
    } else if constexpr (ORDER == 5) {
        constexpr double l[5] = {2. / 60., -13. / 60., 47. / 60., 27. / 60., -3. / 60.};
        constexpr double r[5] = {-3. / 60., 27. / 60., 47. / 60., -13. / 60., 2. / 60.};
        vL = dot<5>(l, s);
        vR = dot<5>(r, s + 1);
    } else if constexpr (ORDER == 9) {
        // the published UP9 weights, as they stand (the left-biased set sums
        // to 4217/2520, not one)                fv_up7_ducros_2d.cu:176-186
        constexpr double l[9] = {3. / 2520., -25. / 2520., 101. / 2520., -319. / 2520., 2765. / 2520.,
                                 2139. / 2520., -533. / 2520., 97. / 2520., -11. / 2520.};
        constexpr double r[9] = {-11. / 2520., 97. / 2520., -533. / 2520., 2139. / 2520., 2765. / 2520.,
                                 -319. / 2520., 101. / 2520., -25. / 2520., 3. / 2520.};
        vL = dot<9>(l, s);
        vR = dot<9>(r, s + 1);
    } else {
        static_assert(ORDER == 7, "ORDER must be 3, 5, 7 or 9");
        constexpr double l[7] = {-3. / 420., 25. / 420., -101. / 420., 319. / 420., 214. / 420., -38. / 420.,
                                 4. / 420.};
        constexpr double r[7] = {4. / 420., -38. / 420., 214. / 420., 319. / 420., -101. / 420., 25. / 420.,
                                 -3. / 420.};
        vL = dot<7>(l, s);
        vR = dot<7>(r, s + 1);
    }
}

// carb_fv's HLL on the reconstructed states (carb_fv_2d.cu:116-160), in
// Einfeldt's form
__device__ __forceinline__ void hll(const double L[4], const double R[4], const Gas &gs, double F[4])
{
    const double rL = L[0], uL = L[1], tL = L[2], pL = L[3], rR = R[0], uR = R[1], tR = R[2], pR = R[3];
    // sound speed without a floor, as carb_fv_2d.cu:60-61 (rho, p >= 1e-14)
    const double cL = snd_raw(gs.gam * pL, rL), cR = snd_raw(gs.gam * pR, rR);
    const double EL = energy(rL, uL, tL, pL, gs), ER = energy(rR, uR, tR, pR, gs);
    const double SL = smin<double>(smin<double>(uL - cL, uR - cR), 0.), SR = smax<double>(smax<double>(uL + cL, uR + cR), 0.);
    const double inv = frcp(SR - SL), SRL = SR * SL;
    const double mL = rL * uL, mR = rR * uR;
    F[0] = fma(SRL, rR - rL, fma(SR, mL, -(SL * mR))) * inv;
    F[1] = fma(SRL, mR - mL, fma(SR, fma(mL, uL, pL), -(SL * fma(mR, uR, pR)))) * inv;
    F[2] = fma(SRL, fma(rR, tR, -(rL * tL)), fma(SR, mL * tL, -(SL * (mR * tR)))) * inv;
    F[3] = fma(SRL, ER - EL, fma(SR, (EL + pL) * uL, -(SL * ((ER + pR) * uR)))) * inv;
}

// carb_fv's Roe solver with the Harten-Hyman entropy fix (carb_fv_2d.cu:161-211)
__device__ __forceinline__ void roe(const double L[4], const double R[4], const Gas &gs, double F[4])
{
    const double rL = L[0], uL = L[1], tL = L[2], pL = L[3], rR = R[0], uR = R[1], tR = R[2], pR = R[3];
    const double ip = frcp(rL * rR);
    const double irL = rR * ip, irR = rL * ip;
    const double cL = fsqrt(gs.gam * pL * irL), cR = fsqrt(gs.gam * pR * irR);
    const double sqL = fsqrt(rL), sqR = fsqrt(rR);
    const double iden = frcp(sqL + sqR);
    const double a = fma(sqL, uL, sqR * uR) * iden, b = fma(sqL, tL, sqR * tR) * iden;  // Roe velocities
    const double EL = energy(rL, uL, tL, pL, gs), ER = energy(rR, uR, tR, pR, gs);
    const double H = fma(sqL, (EL + pL) * irL, sqR * ((ER + pR) * irR)) * iden;
    const double q2 = fma(a, a, b * b);
    const double c2 = gs.gm1 * fma(-0.5, q2, H);
    const double c = fsqrt(c2 > 1e-14 ? c2 : 1e-14);
    const double ic2 = frcp(c2);
    const double drho = rR - rL, dun = uR - uL, dut = tR - tL, dp = pR - pL;
    const double rr = sqL * sqR, rcd = rr * c * dun;
    const double b1 = (dp - rcd) * (0.5 * ic2);
    const double b2 = fma(-dp, ic2, drho);
    const double b3 = rr * dut;
    const double b4 = (dp + rcd) * (0.5 * ic2);
    // Harten-Hyman: |lambda| below eps/2 replaced by (lambda^2 + eps^2/4)/eps
    const double lam1 = a - c, lam4 = a + c;
    const double eps1 = smax<double>(2. * ((uR - cR) - (uL - cL)), 0.);
    const double eps4 = smax<double>(2. * ((uR + cR) - (uL + cL)), 0.);
    double al1 = fabs(lam1), al4 = fabs(lam4);
    const double al2 = fabs(a);
    al1 = al1 < eps1 * 0.5 ? fma(lam1, lam1, eps1 * eps1 * 0.25) * frcp(eps1) : al1;
    al4 = al4 < eps4 * 0.5 ? fma(lam4, lam4, eps4 * eps4 * 0.25) * frcp(eps4) : al4;
    const double w1 = al1 * b1, w2 = al2 * b2, w3 = al2 * b3, w4 = al4 * b4;
    const double d0 = w1 + w2 + w4;
    const double d1 = fma(w4, lam4, fma(w2, a, w1 * lam1));
    const double d2 = fma(d0, b, w3);
    const double ac = a * c;
    const double d3 = fma(w4, H + ac, fma(w3, b, fma(w2 * 0.5, q2, w1 * (H - ac))));
    const double mL = rL * uL, mR = rR * uR;
    F[0] = 0.5 * (mL + mR - d0);
    F[1] = 0.5 * (fma(mL, uL, pL) + fma(mR, uR, pR) - d1);
    F[2] = 0.5 * (fma(mL, tL, mR * tR) - d2);
    F[3] = 0.5 * (fma(EL + pL, uL, (ER + pR) * uR) - d3);
}

// sign by the high word (0 counts as non-negative, -0 as negative)
__device__ __forceinline__ bool nonneg(double x) { return __double2hiint(x) >= 0; }

// HLLC with Davis wave-speed bounds                fv_up7_ducros_2d.cu:237-292
__device__ __forceinline__ void hllc(const double L[4], const double R[4], const Gas &gs, double F[4])
{
    const double rL = L[0], uL = L[1], tL = L[2], pL = L[3], rR = R[0], uR = R[1], tR = R[2], pR = R[3];
    const double cL = snd(gs.gam * pL, rL), cR = snd(gs.gam * pR, rR);
    const double SL = smin<double>(uL - cL, uR - cR), SR = smax<double>(uL + cL, uR + cR);
    const double dL = rL * (SL - uL), dR = rR * (SR - uR);
    const double Ss = fma(-dR, uR, fma(dL, uL, pR - pL)) * frcp(dL - dR);
    // side K: by the contact when subsonic, by the fan when supersonic
    const bool supL = nonneg(SL), sup = supL | !nonneg(SR);
    const bool left = sup ? supL : nonneg(Ss);
    const double rK = left ? rL : rR, uK = left ? uL : uR, tK = left ? tL : tR;
    const double pK = left ? pL : pR, SK = left ? SL : SR;
    const double EK = energy(rK, uK, tK, pK, gs);
    // star state; in a supersonic fan S = u_K with SK - u_K and SK - S taken
    // as 1, which gives K's own state (those differences could be 0 beside a
    // floored sound speed).  S - u_K is then an exact 0, so p* and E* are p_K and
    // E_K to the bit: E* formed with p* S - p_K u_K would put a term of other
    // units beside E_K there, and lose its digits as velocities grow
    const double S = sup ? uK : Ss;
    const double w = sup ? 1. : SK - uK;
    const double q = frcp(sup ? 1. : SK - Ss);
    const double dK = rK * w, du = S - uK;
    const double ps = fma(dK, du, pK);
    const double Es = fma(du, fma(dK, S, pK), EK * w) * q;
    F[0] = dK * q * S;
    F[1] = fma(F[0], S, ps);
    F[2] = F[0] * tK;
    F[3] = (Es + ps) * S;
}

// Blended flux (1 - s) Fh + s HLLE(WL, WR), s the pressure-jump sensor of the
// two cells; L, R: reconstructions, floored here; WL, WR: the cells with sound
// speeds cW* and energies EW*.  RS: Fh is 0 HLLC (fv_up7), 1 HLL, 2 Roe.
//                                               fv_up7_ducros_2d.cu:296-328, :421-433
template <int RS>
__device__ __forceinline__ void face_flux(const double Lin[4], const double Rin[4], const double WL[4],
                                          const double WR[4], double cWL, double cWR, double EWL, double EWR,
                                          const Gas &gs, double F[4])
{
    const double L[4] = {fl14(Lin[0]), Lin[1], Lin[2], fl14(Lin[3])};
    const double R[4] = {fl14(Rin[0]), Rin[1], Rin[2], fl14(Rin[3])};
    double Fh[4];
    if constexpr (RS == 1) hll(L, R, gs, Fh);
    else if constexpr (RS == 2) roe(L, R, gs, Fh);
    else hllc(L, R, gs, Fh);
    const double rL = WL[0], uL = WL[1], tL = WL[2], pL = WL[3], rR = WR[0], uR = WR[1], tR = WR[2], pR = WR[3];
    // X = 2 min(SL, 0), Y = 2 max(SR, 0); Y - X >= 4e-7, the cells' sound
    // speeds being at least 1e-7
    const double SL = smin<double>(uL - cWL, uR - cWR), SR = smax<double>(uL + cWL, uR + cWR);
    const double X = SL - fabs(SL), Y = SR + fabs(SR), dS = Y - X;
    const double dp = pR - pL, ps = pR + pL, dp2 = dp * dp;
    const double dd = fma(0.1 * ps, ps, dp2);
    // one reciprocal for the span and the sensor's denominator (dd >= 4e-29:
    // the product is normal); w = s / (Y - X)
    const double ip = frcp(dS * dd);
    const double sd = dp2 * (dS * ip), w = sd * (dd * ip), om = 1. - sd;
    const double a = Y * w, b = -(X * w);
    const double kL = a * fma(-0.5, X, uL), kR = b * fma(-0.5, Y, uR);
    const double gL = rL * kL, gR = rR * kR;
    const double aP = a * pL, bP = b * pR;
    F[0] = fma(om, Fh[0], gL + gR);
    F[1] = fma(om, Fh[1], fma(uL, gL, fma(uR, gR, aP + bP)));
    F[2] = fma(om, Fh[2], fma(tL, gL, tR * gR));
    F[3] = fma(om, Fh[3], fma(EWL, kL, fma(EWR, kR, fma(aP, uL, bP * uR))));
}

// two neighbouring faces of one thread (cells 0 | 1 and 1 | 2)
template <int RS>
__device__ __forceinline__ void face_pair(const double LA[4], const double RA[4], const double LB[4],
                                          const double RB[4], const double W0[4], const double W1[4],
                                          const double W2[4], double c0, double c1, double c2, double e0, double e1,
                                          double e2, const Gas &gs, double FA[4], double FB[4])
{
    face_flux<RS>(LA, RA, W0, W1, c0, c1, e0, e1, gs, FA);
    face_flux<RS>(LB, RB, W1, W2, c1, c2, e1, e2, gs, FB);
}

}  // namespace f64
}  // namespace fvb
