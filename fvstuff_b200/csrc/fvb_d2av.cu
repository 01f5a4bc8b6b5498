// fvb_d2av.cu -- the scheme kept in fv_up7_ducros_2d.cu.bak (the earlier
// form of fv_up7) on the device: UP-order (3, 5, 7, 9) reconstruction of the
// conserved variables, HLLC on the reconstructed states, and a D2
// artificial viscosity
//   D2 = (C2/h) S_D (sum of lam_face dU) + (Cg/h) (1 - S_D) (the same sum)
// whose Ducros weight S_D = div^2 / (div^2 + sc c^2 / h^2) comes from the
// 6th-order divergence of the velocity (compressions only).  SSP-RK3 on
// conserved variables, no floors; FP64.
//
// One launch per stage does all of it for a tile of 32 x 8 cells: the halo
// box of the stage input (g = max((order+1)/2, 3) layers, the sensor's reach)
// goes to shared memory together with each box cell's sensor velocities,
// |u|+c, |v|+c and c; every face flux is computed once; each cell then
// forms its residual, sensor and viscosity, combines the RK stage and stores
// itself with its ghost images (put_cell).  Stage 3 max-reduces |u|+|v|+c of
// the new state for the next step's dt.
//
// Every expression keeps the reference's association order and this file
// is compiled without FMA contraction (-fmad=false), so a stage reproduces
// the reference kernels' arithmetic operation for operation.
//
// What bounds it: instruction issue and the FP64 pipe, not memory (1024^2,
// UP5: 14 us of a stage at the copy bandwidth).  The operators' divisions and
// roots were most of it: 60 divisions a cell, 4970 instructions and 1530 FP64
// ones, 235 us a stage.  Rounding the same quotients from shared reciprocals
// (fvb_ieee.cuh: one reciprocal of a density for the three quotients by it,
// none for the constant denominators and h) took a stage to 105 us; step
// control once a CTA, chained launches and tiles taken as CTAs come free to 87.
#include <algorithm>

#include "fvb_aux.h"
#include "fvb_device.cuh"
#include "fvb_ieee.cuh"

namespace fvb {
namespace {

constexpr int DTX = 32, DTY = 8, DNT = 256;

// conserved -> p, c, u, v; no density floor, c^2 floored at 1e-14
//                                          fv_up7_ducros_2d.cu.bak:65-74
__device__ __forceinline__ void d2_prim(double gam, double rho, double mx, double my, double E, double &p,
                                        double &c, double &u, double &v)
{
    u = mx / rho;
    v = my / rho;
    p = (gam - 1.0) * (E - 0.5 * (mx * u + my * v));
    const double cs2 = gam * p / rho;
    c = sqrt(cs2 > 1e-14 ? cs2 : 1e-14);
}

// HLLC of conserved face states in the face-normal frame (rho, m_n, m_t, E);
// a y-face passes (rho v, rho u) as (m_n, m_t), which leaves every
// operation's operands as the reference's y-solver has them
//                                          fv_up7_ducros_2d.cu.bak:202-282
__device__ void d2_hllc(double gam, const double UL[4], const double UR[4], double F[4])
{
    double pL, cL, uL, vL, pR, cR, uR, vR;
    d2_prim(gam, UL[0], UL[1], UL[2], UL[3], pL, cL, uL, vL);
    d2_prim(gam, UR[0], UR[1], UR[2], UR[3], pR, cR, uR, vR);
    const double SL = smin<double>(uL - cL, uR - cR);
    const double SR = smax<double>(uL + cL, uR + cR);
    if (SL >= 0.0) {
        F[0] = UL[1]; F[1] = UL[1] * uL + pL; F[2] = UL[1] * vL; F[3] = (UL[3] + pL) * uL;
        return;
    }
    if (SR <= 0.0) {
        F[0] = UR[1]; F[1] = UR[1] * uR + pR; F[2] = UR[1] * vR; F[3] = (UR[3] + pR) * uR;
        return;
    }
    const double dL = UL[0] * (SL - uL), dR = UR[0] * (SR - uR);
    const double Ss = (pR - pL + dL * uL - dR * uR) / (dL - dR);
    const bool left = Ss >= 0.0;
    const double K0 = left ? UL[0] : UR[0], K1 = left ? UL[1] : UR[1];
    const double K2 = left ? UL[2] : UR[2], K3 = left ? UL[3] : UR[3];
    const double pK = left ? pL : pR, uK = left ? uL : uR, vK = left ? vL : vR, SK = left ? SL : SR;
    const double f = K0 * (SK - uK) / (SK - Ss);
    const double s3 = f * (K3 / K0 + (Ss - uK) * (Ss + pK / (K0 * (SK - uK))));
    F[0] = K1 + SK * (f - K0);
    F[1] = (K1 * uK + pK) + SK * (f * Ss - K1);
    F[2] = K1 * vK + SK * (f * vK - K2);
    F[3] = (K3 + pK) * uK + SK * (s3 - K3);
}

// upwind-biased face values from the stencil s[0 .. order] along the face
// normal (the face lies between s[hw-1] and s[hw])
//                                          fv_up7_ducros_2d.cu.bak:105-153
template <int ORDER>
__device__ __forceinline__ void d2_recon(const double *s, double &vL, double &vR)
{
    if constexpr (ORDER == 3) {
        vL = (-s[0] + 5.0 * s[1] + 2.0 * s[2]) / 6.0;
        vR = (2.0 * s[1] + 5.0 * s[2] - s[3]) / 6.0;
    } else if constexpr (ORDER == 5) {
        vL = (2.0 * s[0] - 13.0 * s[1] + 47.0 * s[2] + 27.0 * s[3] - 3.0 * s[4]) / 60.0;
        vR = (-3.0 * s[1] + 27.0 * s[2] + 47.0 * s[3] - 13.0 * s[4] + 2.0 * s[5]) / 60.0;
    } else if constexpr (ORDER == 9) {
        // the published weights as they stand (the left-biased set sums to
        // 4217/2520)                            fv_up7_ducros_2d.cu.bak:132-142
        vL = (3.0 * s[0] - 25.0 * s[1] + 101.0 * s[2] - 319.0 * s[3] + 2765.0 * s[4] + 2139.0 * s[5] -
              533.0 * s[6] + 97.0 * s[7] - 11.0 * s[8]) /
             2520.0;
        vR = (-11.0 * s[1] + 97.0 * s[2] - 533.0 * s[3] + 2139.0 * s[4] + 2765.0 * s[5] - 319.0 * s[6] +
              101.0 * s[7] - 25.0 * s[8] + 3.0 * s[9]) /
             2520.0;
    } else {
        vL = (-3.0 * s[0] + 25.0 * s[1] - 101.0 * s[2] + 319.0 * s[3] + 214.0 * s[4] - 38.0 * s[5] + 4.0 * s[6]) /
             420.0;
        vR = (4.0 * s[1] - 38.0 * s[2] + 214.0 * s[3] + 319.0 * s[4] - 101.0 * s[5] + 25.0 * s[6] - 3.0 * s[7]) /
             420.0;
    }
}

// ---- the same operations with the quotients and roots of fvb_ieee.cuh ------
// Every function below returns the bits of its operator form above while its
// range tests hold (their result: true); the caller evaluates the operator
// form otherwise.

struct D2State {
    double p, c, u, v, y;  // y: reciprocal of the density
};

// The forms of a face and of a cell: quotients from shared reciprocals, for tiles
// without small momenta (see the kernel); the same with small numerators looked
// after; the operators, for whatever leaves the range.
enum { D2_NEAR, D2_SMALL, D2_PLAIN };

// (a velocity whose quotient underflows is off, which p and |u| + c do not notice)
__device__ __forceinline__ bool d2_prim_near(double gam, const double U[4], D2State &w)
{
    const double y = recip(U[0]);
    w.y = y;
    w.u = quot(U[1], U[0], y);
    w.v = quot(U[2], U[0], y);
    w.p = (gam - 1.0) * (U[3] - 0.5 * (U[1] * w.u + U[2] * w.v));
    const double gp = gam * w.p, cs2 = quot(gp, U[0], y);
    const double x = cs2 > 1e-14 ? cs2 : 1e-14;
    w.c = root(x);
    return pos_ok(U[0]) && fin_ok(U[1], U[2]) && pos_ok(gp) && fin_ok(x);
}

template <int FORM>
__device__ __forceinline__ bool d2_hllc_near(double gam, const double UL[4], const double UR[4], double F[4])
{
    D2State l, r;
    bool ok = d2_prim_near(gam, UL, l);
    ok = d2_prim_near(gam, UR, r) && ok;
    if constexpr (FORM == D2_SMALL) {
        // (p and c of either side take nothing from a small momentum)
        if (is_small(UL[1])) l.u = small_quot(UL[1], UL[0], l.y);
        if (is_small(UL[2])) l.v = small_quot(UL[2], UL[0], l.y);
        if (is_small(UR[1])) r.u = small_quot(UR[1], UR[0], r.y);
        if (is_small(UR[2])) r.v = small_quot(UR[2], UR[0], r.y);
    }
    const double SL = smin<double>(l.u - l.c, r.u - r.c);
    const double SR = smax<double>(l.u + l.c, r.u + r.c);
    if (SL >= 0.0) {
        F[0] = UL[1]; F[1] = UL[1] * l.u + l.p; F[2] = UL[1] * l.v; F[3] = (UL[3] + l.p) * l.u;
        return ok;
    }
    if (SR <= 0.0) {
        F[0] = UR[1]; F[1] = UR[1] * r.u + r.p; F[2] = UR[1] * r.v; F[3] = (UR[3] + r.p) * r.u;
        return ok;
    }
    const double dL = UL[0] * (SL - l.u), dR = UR[0] * (SR - r.u);
    const double sn = r.p - l.p + dL * l.u - dR * r.u, sd = dL - dR, yd = recip(sd);
    double Ss = squot(sn, sd, yd);
    if (FORM == D2_SMALL && is_small(sn)) Ss = small_quot(sn, sd, yd);
    const bool left = Ss >= 0.0;
    const double K0 = left ? UL[0] : UR[0], K1 = left ? UL[1] : UR[1];
    const double K2 = left ? UL[2] : UR[2], K3 = left ? UL[3] : UR[3];
    const double pK = left ? l.p : r.p, uK = left ? l.u : r.u, vK = left ? l.v : r.v, SK = left ? SL : SR;
    const double yK = left ? l.y : r.y;
    const double dK = left ? dL : dR;  // K0 (SK - uK), the same product
    const double sq = SK - Ss;
    const double f = squot(dK, sq, recip(sq));
    const double s3 = f * (quot(K3, K0, yK) + (Ss - uK) * (Ss + squot(pK, dK, recip(dK))));
    F[0] = K1 + SK * (f - K0);
    F[1] = (K1 * uK + pK) + SK * (f * Ss - K1);
    F[2] = K1 * vK + SK * (f * vK - K2);
    F[3] = (K3 + pK) * uK + SK * (s3 - K3);
    return ok && den_ok(sd) && den_ok(sq) && den_ok(dK) && fin_ok(sn) && pos_ok(K3);
}

// (a product with 2 or 4 is exact, so fused with the sum beside it it rounds
// as the separate operations do; SMALL: sums whose quotients underflow are
// looked after)
template <int ORDER, bool SMALL>
__device__ __forceinline__ void d2_recon_near(const double *s, double &vL, double &vR)
{
    constexpr double D = ORDER == 3 ? 6.0 : ORDER == 5 ? 60.0 : ORDER == 9 ? 2520.0 : 420.0;
    double a, b;
    if constexpr (ORDER == 3) {
        a = fma(2.0, s[2], -s[0] + 5.0 * s[1]);
        b = fma(2.0, s[1], 5.0 * s[2]) - s[3];
    } else if constexpr (ORDER == 5) {
        a = fma(2.0, s[0], -(13.0 * s[1])) + 47.0 * s[2] + 27.0 * s[3] - 3.0 * s[4];
        b = fma(2.0, s[5], -3.0 * s[1] + 27.0 * s[2] + 47.0 * s[3] - 13.0 * s[4]);
    } else if constexpr (ORDER == 9) {
        a = 3.0 * s[0] - 25.0 * s[1] + 101.0 * s[2] - 319.0 * s[3] + 2765.0 * s[4] + 2139.0 * s[5] - 533.0 * s[6] +
            97.0 * s[7] - 11.0 * s[8];
        b = -11.0 * s[1] + 97.0 * s[2] - 533.0 * s[3] + 2139.0 * s[4] + 2765.0 * s[5] - 319.0 * s[6] + 101.0 * s[7] -
            25.0 * s[8] + 3.0 * s[9];
    } else {
        a = fma(4.0, s[6], -3.0 * s[0] + 25.0 * s[1] - 101.0 * s[2] + 319.0 * s[3] + 214.0 * s[4] - 38.0 * s[5]);
        b = fma(4.0, s[1], -(38.0 * s[2])) + 214.0 * s[3] + 319.0 * s[4] - 101.0 * s[5] + 25.0 * s[6] - 3.0 * s[7];
    }
    vL = quot(a, D, 1.0 / D);
    vR = quot(b, D, 1.0 / D);
    if (SMALL && is_small(a, b)) {
        if (is_small(a)) vL = small_quot(a, D, 1.0 / D);
        if (is_small(b)) vR = small_quot(b, D, 1.0 / D);
    }
}

template <int ORDER>
struct D2Shape {
    static constexpr int HW = (ORDER + 1) / 2;         // reconstruction half width
    static constexpr int HB = HW > 3 ? HW : 3;         // halo of the box (= the grid's ghost width)
    static constexpr int BW = DTX + 2 * HB, BH = DTY + 2 * HB, PL = BW * BH;
    static constexpr int NFX = (DTX + 1) * DTY, NFY = DTX * (DTY + 1);
    // Q[4][PL] | SU, SV, LX, LY, CS [PL each] | FX[4][NFX] | FY[4][NFY]
    static constexpr size_t SMEM = sizeof(double) * (9 * PL + 4 * NFX + 4 * NFY);
    // resident CTAs an SM is compiled for: four (56 KB each, <= 64
    // registers) with the 3-cell halo, three (64 KB, 72 KB) with UP7's 4
    // and UP9's 5
    static constexpr int MINB = HB == 3 ? 4 : 3;
};

// the flux of one face in its normal frame, b its right / top cell, st the
// stride to the left / bottom one
template <int ORDER, int FORM>
__device__ __forceinline__ bool d2_face(const double *Q, int b, int st, bool xf, double gam, double Fn[4])
{
    using S = D2Shape<ORDER>;
    constexpr int HW = S::HW;
    double L[4], R[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        double s[2 * HW];
#pragma unroll
        for (int d = 0; d < 2 * HW; ++d) s[d] = Q[q * S::PL + b + (d - HW) * st];
        if constexpr (FORM == D2_PLAIN) d2_recon<ORDER>(s, L[q], R[q]);
        else if (q == 1 || q == 2) d2_recon_near<ORDER, FORM == D2_SMALL>(s, L[q], R[q]);
        else d2_recon_near<ORDER, false>(s, L[q], R[q]);
    }
    const double UL[4] = {L[0], xf ? L[1] : L[2], xf ? L[2] : L[1], L[3]};
    const double UR[4] = {R[0], xf ? R[1] : R[2], xf ? R[2] : R[1], R[3]};
    if constexpr (FORM != D2_PLAIN) return d2_hllc_near<FORM>(gam, UL, UR, Fn);
    d2_hllc(gam, UL, UR, Fn);
    return true;
}

// a face that the forms above gave up
template <int ORDER>
__device__ __noinline__ void d2_face_any(const double *Q, int b, int st, bool xf, double gam, double Fn[4])
{
    d2_face<ORDER, D2_PLAIN>(Q, b, st, xf, gam, Fn);
}

// the faces of a tile
template <int ORDER, int FORM>
__device__ __forceinline__ void d2_faces(const double *Q, double *FX, double *FY, double gam, int tid)
{
    using S = D2Shape<ORDER>;
    constexpr int HB = S::HB, BW = S::BW;
    for (int f = tid; f < S::NFX + S::NFY; f += DNT) {
        const bool xf = f < S::NFX;
        int r, c, st;
        if (xf) { r = f / (DTX + 1); c = f - r * (DTX + 1); st = 1; }
        else { const int f2 = f - S::NFX; r = f2 / DTX; c = f2 - r * DTX; st = BW; }
        const int b = (r + HB) * BW + (c + HB);
        double Fn[4];
        if (!d2_face<ORDER, FORM>(Q, b, st, xf, gam, Fn)) {
            double Fa[4];
            d2_face_any<ORDER>(Q, b, st, xf, gam, Fa);
#pragma unroll
            for (int q = 0; q < 4; ++q) Fn[q] = Fa[q];
        }
        const int qn = xf ? 1 : 2, qt = xf ? 2 : 1;
        double *o = xf ? FX + r * (DTX + 1) + c : FY + r * DTX + c;
        const int os = xf ? S::NFX : S::NFY;
        o[0] = Fn[0];
        o[qn * os] = Fn[1];
        o[qt * os] = Fn[2];
        o[3 * os] = Fn[3];
    }
}

// per-cell quantities of the box in the operator form
__device__ __noinline__ void d2_box_any(double gam, double U0, double U1, double U2, double U3, double o[5])
{
    const double U[4] = {U0, U1, U2, U3};
    const double rf = U[0] > 1e-14 ? U[0] : 1e-14;
    double p, cc, u, v;
    d2_prim(gam, U[0], U[1], U[2], U[3], p, cc, u, v);
    o[0] = U[1] / rf;
    o[1] = U[2] / rf;
    o[2] = fabs(u) + cc;
    o[3] = fabs(v) + cc;
    o[4] = cc;
}

__device__ __noinline__ double d2_lam_any(double gam, double U0, double U1, double U2, double U3)
{
    const double U[4] = {U0, U1, U2, U3};
    double p, cc, u, v;
    d2_prim(gam, U[0], U[1], U[2], U[3], p, cc, u, v);
    return fabs(u) + fabs(v) + cc;
}

// what the cell update needs that is the same for every cell
struct D2Cell {
    double h, yh, h60, y60, c2h, cgh, sch, dt;  // y*: reciprocals of h and 60 h
    int stage;
    bool global;  // Cg is not 0
    bool hok;     // h within 2^+-90: h and 60 h are denominators in range, and see d2_cell
};

// residual (flux divergence, Ducros weight, viscosity) and RK combination of
// the cell at b of the box; ua: U0 of the cell; false: out of range.  (Only the
// momenta can be as small as a flux difference whose quotient underflows, and a
// velocity difference of that kind squares to 0.)
//                                          fv_up7_ducros_2d.cu.bak:344-445
template <int ORDER, int FORM>
__device__ __forceinline__ bool d2_cell(const double *Q, const double *FX, const double *FY, int b, int r, int c,
                                        const D2Cell &k, const double ua[4], double v[4])
{
    using S = D2Shape<ORDER>;
    constexpr int BW = S::BW, PL = S::PL;
    const double *SU = Q + 4 * PL, *SV = SU + PL, *LX = SV + PL, *LY = LX + PL, *CS = LY + PL;
    const double wc[6] = {-1., 9., -45., 45., -9., 1.};
    const int wo[6] = {-3, -2, -1, 1, 2, 3};
    double du_dx = 0., dv_dy = 0.;
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        du_dx += wc[m] * SU[b + wo[m]];
        dv_dy += wc[m] * SV[b + wo[m] * BW];
    }
    if constexpr (FORM != D2_PLAIN) {
        du_dx = quot(du_dx, k.h60, k.y60);
        dv_dy = quot(dv_dy, k.h60, k.y60);
    } else {
        du_dx /= k.h60;
        dv_dy /= k.h60;
    }
    double div_u = du_dx + dv_dy;
    if (div_u > 0.) div_u = 0.;
    const double c0 = CS[b];
    const double sos2 = k.sch * c0 * c0;
    const double dd = div_u * div_u, den = dd + sos2 + 1e-40;
    double S_D;
    if constexpr (FORM != D2_PLAIN) {
        const double y = recip(den);
        S_D = quot(dd, den, y);
        if (FORM == D2_SMALL && is_small(dd)) S_D = small_quot(dd, den, y);
    } else {
        S_D = dd / den;
    }
    // face-averaged directional wave speeds   :359-367
    const double lamx_c = LX[b], lamy_c = LY[b];
    const double lhxp = 0.5 * (lamx_c + LX[b + 1]);
    const double lhxm = 0.5 * (lamx_c + LX[b - 1]);
    const double lhyp = 0.5 * (lamy_c + LY[b + BW]);
    const double lhym = 0.5 * (lamy_c + LY[b - BW]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double *Qq = Q + q * PL;
        const double Uc = Qq[b];
        const double dxp = Qq[b + 1] - Uc, dxm = Uc - Qq[b - 1];
        const double dyp = Qq[b + BW] - Uc, dym = Uc - Qq[b - BW];
        double D2 = k.c2h * (lhxp * S_D * dxp - lhxm * S_D * dxm + lhyp * S_D * dyp - lhym * S_D * dym);
        // (with Cg = 0 the term is +0 or -0 for finite states: nothing to add)
        if (FORM == D2_PLAIN || k.global)
            D2 = D2 + k.cgh * (lhxp * (1. - S_D) * dxp - lhxm * (1. - S_D) * dxm + lhyp * (1. - S_D) * dyp -
                               lhym * (1. - S_D) * dym);
        const double *fx = FX + q * S::NFX + r * (DTX + 1) + c;
        const double *fy = FY + q * S::NFY + r * DTX + c;
        double L;
        if constexpr (FORM != D2_PLAIN) {
            const double dx = fx[1] - fx[0], dy = fy[DTX] - fy[0];
            double qx = quot(dx, k.h, k.yh), qy = quot(dy, k.h, k.yh);
            if (FORM == D2_SMALL && (q == 1 || q == 2) && is_small(dx)) qx = small_quot(dx, k.h, k.yh);
            if (FORM == D2_SMALL && (q == 1 || q == 2) && is_small(dy)) qy = small_quot(dy, k.h, k.yh);
            L = -qx - qy + D2;
        } else {
            L = -(fx[1] - fx[0]) / k.h - (fy[DTX] - fy[0]) / k.h + D2;  // :386
        }
        if (k.stage == 1) v[q] = ua[q] + k.dt * L;                                   // :433-435
        else if (k.stage == 2) v[q] = 0.75 * ua[q] + 0.25 * (Uc + k.dt * L);         // :437-440
        else v[q] = (1. / 3.) * ua[q] + (2. / 3.) * (Uc + k.dt * L);                 // :442-445
    }
    return FORM == D2_PLAIN || (k.hok && pos_ok(den) && (FORM == D2_SMALL || !is_small(dd)) && fin_ok(v[0], v[1]) &&
                                fin_ok(v[2], v[3]));
}

template <int ORDER>
__device__ __noinline__ void d2_cell_any(const double *Q, const double *FX, const double *FY, int b, int r, int c,
                                         const D2Cell &k, const double ua[4], double v[4])
{
    d2_cell<ORDER, D2_PLAIN>(Q, FX, FY, b, r, c, k, ua, v);
}

// A tile whose momenta are 0 or at least 2^-300 and whose densities lie within
// 2^+-30, box and all, has no face and no flux difference with a small numerator
// (fvb_ieee.cuh): a sum that is not 0 is at least an ulp of its smaller term, so
// reconstructions are 0 or from 2^-364 on, velocities 2^-396, products of the
// two 2^-760, fluxes 2^-812 and their differences 2^-864.  The others, in the
// tails ahead of a front, take the form that looks after them.
constexpr unsigned kMomMin = 0x2d300000u, kRhoMin = 0x3e100000u, kRhoMax = 0x41d00000u;

// one SSP-RK3 stage                        fv_up7_ducros_2d.cu.bak:287-446
template <int ORDER>
__global__ void __launch_bounds__(DNT, D2Shape<ORDER>::MINB)
    d2av_stage_kernel(const __grid_constant__ GridDev gd, int stage, int ntiles, D2Params av)
{
    using S = D2Shape<ORDER>;
    constexpr int HB = S::HB, BW = S::BW, PL = S::PL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *Q = reinterpret_cast<double *>(smem_raw);  // [4][BH][BW] stage input
    double *SU = Q + 4 * PL;                           // rho u / max(rho, 1e-14)
    double *SV = SU + PL;                              // rho v / max(rho, 1e-14)
    double *LX = SV + PL;                              // |u| + c
    double *LY = LX + PL;                              // |v| + c
    double *CS = LY + PL;                              // c
    double *FX = CS + PL;                              // [4][DTY][DTX+1]
    double *FY = FX + 4 * S::NFX;                      // [4][DTY+1][DTX]
    __shared__ double s_red[DNT / 32];
    __shared__ int s_next;
    const int tid = threadIdx.x, n = gd.n, np = n + 2 * HB;
    const double gam = gd.gam, h = gd.h;
    const double *in = (const double *)(stage == 2 ? gd.k1 : stage == 3 ? gd.k2 : gd.st[0]);
    const double *u0 = (const double *)gd.st[0];
    double *out = (double *)(stage == 1 ? gd.k1 : stage == 2 ? gd.k2 : gd.st[0]);
    double lacc = 0.0;
    // (in shared memory: 18 registers a thread would hold across the faces)
    __shared__ D2Cell ck;
    grid_dependency();
    // the step control, the same for every tile
    const TileCtl ctl = tile_control<P64>(gd.ctrl, stage, tid == 0 && blockIdx.x == 0);
    if (tid == 0)
        ck = D2Cell{h, recip(h), 60. * h, recip(60. * h), av.c2 / h, av.cg / h, av.sc / (h * h), ctl.dt, stage,
                    av.cg != 0.0, h > 0x1p-90 && h < 0x1p90};

    // From two whole waves up a CTA takes its next tile as it comes free: us a
    // stage, fixed share / taken, order 5: 600^2 34.4 / 32.7, 800^2 55.7 / 54.8, 1024^2
    // 91.0 / 86.6, 2048^2 346 / 320 (below, taken: 400^2 20.4 / 22.2).
    const bool queued = ntiles > 2 * (int)gridDim.x;
    if (tid == 0 && blockIdx.x == 0) clear_tile_queue(gd.ctrl, stage);
    for (int t = blockIdx.x, next; t < ntiles && ctl.run; t = next) {
        const int tx0 = (t % gd.tiles_x) * DTX, ty0 = (t / gd.tiles_x) * DTY;
        // ---- halo box of the stage input and its per-cell quantities: the
        //      sensor's velocities in the rows / columns it reaches, the wave
        //      speeds on the cells and their direct neighbours --------------
        unsigned least = 0x7fffffffu;  // least momentum of this thread's cells; 0: a density out of range
        for (int k = tid; k < PL; k += DNT) {
            const int r = k / BW, c = k - r * BW, jp = ty0 + r, ip = tx0 + c;
            double U[4] = {1.0, 0.0, 0.0, 2.5};  // admissible filler beyond the padded grid
            if (jp < np && ip < np) {
                const long long e = (long long)jp * gd.pitch + ip + gd.xoff;
#pragma unroll
                for (int q = 0; q < 4; ++q) U[q] = in[e + q * gd.plane];
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) Q[q * PL + k] = U[q];
            least = min(least, min(hi_below(U[1]), hi_below(U[2])));
            if ((unsigned)__double2hiint(U[0]) - kRhoMin >= kRhoMax - kRhoMin) least = 0u;
            const bool inr = (unsigned)(r - HB) < (unsigned)DTY, inc = (unsigned)(c - HB) < (unsigned)DTX;
            if (!inr && !inc) continue;
            D2State w;
            // (the sensor's velocities divide by the density floored at 1e-14; one that is
            // off is below 2^-850 and changes no divergence whose square is not 0)
            if (d2_prim_near(gam, U, w) && U[0] > 1e-14) {
                SU[k] = w.u;
                SV[k] = w.v;
                LX[k] = fabs(w.u) + w.c;
                LY[k] = fabs(w.v) + w.c;
                CS[k] = w.c;
            } else {
                double o[5];
                d2_box_any(gam, U[0], U[1], U[2], U[3], o);
#pragma unroll
                for (int m = 0; m < 5; ++m) SU[m * PL + k] = o[m];
            }
        }
        const bool small = __syncthreads_or(least < kMomMin);
        int taken = ntiles;  // the next tile, taken while the faces are computed
        if (queued && tid == 0) taken = (int)gridDim.x + atomicAdd(tile_queue(gd.ctrl, stage), 1);
        // ---- faces: x-face (r, c) between tile cells c-1 and c, y-face
        //      (r, c) between rows r-1 and r; b = the right / top cell -----
        if (small) d2_faces<ORDER, D2_SMALL>(Q, FX, FY, gam, tid);
        else d2_faces<ORDER, D2_NEAR>(Q, FX, FY, gam, tid);
        if (queued && tid == 0) s_next = taken;
        __syncthreads();
        next = queued ? s_next : t + (int)gridDim.x;
        if (next >= ntiles) grid_release();
        // ---- cells: residual, sensor, viscosity, RK combination, stores ---
        for (int k = tid; k < DTX * DTY; k += DNT) {
            const int r = k / DTX, c = k - r * DTX, i = tx0 + c, j = ty0 + r;
            if (i >= n || j >= n) continue;
            const int b = (r + HB) * BW + (c + HB);
            const long long e = (long long)(j + HB) * gd.pitch + (i + HB) + gd.xoff;
            double ua[4], v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) ua[q] = stage == 1 ? Q[q * PL + b] : u0[e + q * gd.plane];
            const bool ok = small ? d2_cell<ORDER, D2_SMALL>(Q, FX, FY, b, r, c, ck, ua, v)
                                  : d2_cell<ORDER, D2_NEAR>(Q, FX, FY, b, r, c, ck, ua, v);
            if (!ok) {
                double ub[4], va[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) ub[q] = ua[q];
                d2_cell_any<ORDER>(Q, FX, FY, b, r, c, ck, ub, va);
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = va[q];
            }
            put_cell<double>(gd, out, j, i, v);
            if (stage == 3) {
                D2State w;
                lacc = smax<double>(d2_prim_near(gam, v, w) ? fabs(w.u) + fabs(w.v) + w.c : d2_lam_any(gam, v[0], v[1], v[2], v[3]),
                                    lacc);  // lam_c, :362
            }
        }
        if (stage == 3 && tid == 0 && t == 0) leader_finish<P64>(gd.ctrl);
        __syncthreads();
    }
    if (stage == 3) {
        for (int o = 16; o > 0; o >>= 1) lacc = fmax(lacc, __shfl_xor_sync(0xffffffffu, lacc, o));
        if ((tid & 31) == 0) s_red[tid >> 5] = lacc;
        __syncthreads();
        if (tid == 0) {
            double m = 0.0;
            for (int w = 0; w < DNT / 32; ++w) m = fmax(m, s_red[w]);
            if (m > 0.0) atomicMax(&gd.ctrl->lam_acc, (unsigned long long)__double_as_longlong(m));
        }
    }
}

__device__ __forceinline__ long long d2_at(const GridDev &gd, int j, int i)
{
    return (long long)(j + gd.g) * gd.pitch + (i + gd.g) + gd.xoff;
}

// |u| + |v| + c of a state, max into ctrl->lam_acc      :77-83, :593-612
__global__ void d2av_lam_kernel(const GridDev gd, const double *buf)
{
    __shared__ double sh[32];
    const long long n2 = (long long)gd.n * gd.n;
    double m = 0.0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n2;
         k += (long long)blockDim.x * gridDim.x) {
        const long long e = d2_at(gd, (int)(k / gd.n), (int)(k % gd.n));
        double p, c, u, v;
        d2_prim(gd.gam, buf[e], buf[e + gd.plane], buf[e + 2 * gd.plane], buf[e + 3 * gd.plane], p, c, u, v);
        m = fmax(m, fabs(u) + fabs(v) + c);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) b = fmax(b, sh[w]);
        if (b > 0.0) atomicMax(&gd.ctrl->lam_acc, (unsigned long long)__double_as_longlong(b));
    }
}

// Ducros weight of every cell, FP32, for the frame's sensor panel
//                                          fv_up7_ducros_2d.cu.bak:393-428
__global__ void d2av_sensor_kernel(const GridDev gd, const double *buf, double sc, float *out)
{
    const int n = gd.n;
    const double h = gd.h;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < (long long)n * n;
         k += (long long)blockDim.x * gridDim.x) {
        const int j = (int)(k / n), i = (int)(k % n);
        const long long e = d2_at(gd, j, i);
        double p, c0, u, v;
        d2_prim(gd.gam, buf[e], buf[e + gd.plane], buf[e + 2 * gd.plane], buf[e + 3 * gd.plane], p, c0, u, v);
        const double wc[6] = {-1., 9., -45., 45., -9., 1.};
        const int wo[6] = {-3, -2, -1, 1, 2, 3};
        double du_dx = 0., dv_dy = 0.;
        for (int m = 0; m < 6; ++m) {
            const long long ex = e + wo[m], ey = e + (long long)wo[m] * gd.pitch;
            double rx = buf[ex], ry = buf[ey];
            rx = rx > 1e-14 ? rx : 1e-14;
            ry = ry > 1e-14 ? ry : 1e-14;
            du_dx += wc[m] * (buf[ex + gd.plane] / rx);
            dv_dy += wc[m] * (buf[ey + 2 * gd.plane] / ry);
        }
        du_dx /= 60. * h;
        dv_dy /= 60. * h;
        double div_u = du_dx + dv_dy;
        if (div_u > 0.) div_u = 0.;
        const double sos2 = (sc / (h * h)) * c0 * c0;
        out[k] = (float)((div_u * div_u) / (div_u * div_u + sos2 + 1e-40));
    }
}

int sm_count()
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

template <int ORDER>
cudaError_t launch_order(const GridDev &gd, int stage, int tiles, const D2Params &av, cudaStream_t s)
{
    constexpr size_t smem = D2Shape<ORDER>::SMEM;
    LaunchFacts f{};
    cudaError_t e = launch_facts((const void *)d2av_stage_kernel<ORDER>, DNT, smem, f);
    if (e != cudaSuccess) return e;
    const int cap = f.ctas_per_sm * f.sms;
    void *args[] = {(void *)&gd, (void *)&stage, (void *)&tiles, (void *)&av};
    return launch_chained((const void *)d2av_stage_kernel<ORDER>, tiles < cap ? tiles : cap, DNT, smem, s, args);
}

}  // namespace

int d2av_ghost(int order) { return std::max((order + 1) / 2, 3); }

void d2av_tiles(int n, int &tiles_x, int &tiles)
{
    tiles_x = (n + DTX - 1) / DTX;
    tiles = tiles_x * ((n + DTY - 1) / DTY);
}

cudaError_t d2av_launch_stage(const GridDev &gd, int order, int stage, int tiles, const D2Params &av,
                              cudaStream_t s)
{
    if (order == 3) return launch_order<3>(gd, stage, tiles, av, s);
    if (order == 5) return launch_order<5>(gd, stage, tiles, av, s);
    if (order == 7) return launch_order<7>(gd, stage, tiles, av, s);
    if (order == 9) return launch_order<9>(gd, stage, tiles, av, s);
    return cudaErrorInvalidValue;
}

cudaError_t d2av_lam_into(const GridDev &gd, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(&gd.ctrl->lam_acc, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    const long long n2 = (long long)gd.n * gd.n;
    const int blocks = (int)std::min<long long>((n2 + 255) / 256, 4LL * sm_count());
    d2av_lam_kernel<<<blocks, 256, 0, s>>>(gd, (const double *)gd.st[0]);
    return cudaGetLastError();
}

cudaError_t d2av_sensor_into(const GridDev &gd, double sc, float *out, cudaStream_t s)
{
    const long long n2 = (long long)gd.n * gd.n;
    const int blocks = (int)std::min<long long>((n2 + 255) / 256, 4LL * sm_count());
    d2av_sensor_kernel<<<blocks, 256, 0, s>>>(gd, (const double *)gd.st[0], sc, out);
    return cudaGetLastError();
}

}  // namespace fvb
