// fvb_rec3.cu -- the rec3 + HLLC + 2x2-block Zhang-Shu scheme of
// fv_rec3_2d.cu on the device (FP64, conserved cell averages, g = 2,
// periodic, N even).
//
// Per face: unlimited 3rd-order parabolic reconstruction of the conserved
// variables on both sides, each face state scaled toward its own cell's
// average until rho and p clear their floors (the pointwise Zhang-Shu
// scaling), conversion to floored primitives, HLLC.  Per cell: the residual,
// the SSP-RK3 combination, then the a-posteriori Zhang-Shu limiter on the
// non-overlapping 2x2 blocks of the new state (block corners by bilinear
// extrapolation, one common theta per block, block total conserved).
//
// One launch per stage does all of it for a tile of 32 x 14 cells: tiles
// start on even cells, so every 2x2 block lies in one tile.  Two halo boxes
// alternate (TMA, the next one in flight from the end of a tile's faces) and U0
// arrives during the faces; after the face fluxes a warp takes 2 rows of 16 cells, a
// block being four of its lanes, so that residual, RK combination, limiter and
// stores (interior + periodic ghost images) need no barrier between; stage 3
// max-reduces the wave speed of the limited state.
//
// The reference scatters each face flux into its two cells with atomicAdd;
// here every cell gathers its four face terms in the order a serial run of
// that scatter adds them (by source cell index), and this file is compiled
// without FMA contraction (-fmad=false), so each stage reproduces the
// reference's arithmetic operation for operation.
//
// What bounds it: instruction issue, and on shocks the bisections' dependent
// chains; not memory (1024^2: 14 us of a stage at the copy bandwidth).
// Quotients and roots come from shared reciprocals (fvb_ieee.cuh: 2500 -> 1090
// instructions a cell).  A face or block that clears its floors, nearly all,
// needs no scaling and takes none of its code; the faces that do not are
// listed and then handled one a thread: in place, each warp along the shock
// went through 25 dependent steps for one or two of its lanes, face after
// face, and the tiles of the ring held the launch up (84 us of it).  The
// limiter's bisection likewise takes a block's four corners side by side.
// us a stage at 1024^2, mean over ten steps of the Sod (a smooth state): 225
// (242) as it was, 116 (97) with shared reciprocals, the list and plain loads
// into 32 x 32 tiles, 105 (77) with the pipeline above, 94 with tiles taken as
// CTAs come free.
#include <algorithm>

#include "fvb_aux.h"
#include "fvb_device.cuh"
#include "fvb_ieee.cuh"
#include "fvb_tma.cuh"

namespace fvb {
namespace {

constexpr double R3_GAM = 1.4, R3_PFLOOR = 1e-9, R3_RHOFLOOR = 1e-12;
constexpr int RTX = 32, RTY = 14, RNT = 256, RG = 2;
using RPipe = BoxPipe<RG, RTX, RTY, RNT>;
constexpr int RSW = RPipe::SW, RPL = RPipe::PL;
static_assert(RPipe::XO == 0, "the box starts at the tile's first padded column");
// shared memory, in doubles: two boxes, U0, x-fluxes, y-fluxes
constexpr int ROU0 = 2 * RPipe::BOX, ROFX = ROU0 + RPipe::U0, ROFY = ROFX + 4 * RTY * (RTX + 1);
constexpr int RNF = RTY * (RTX + 1) + (RTY + 1) * RTX;  // faces of a tile

// c = sqrt(gamma p / rho)                       fv_rec3_2d.cu:68-69
__device__ __forceinline__ double r3_snd(double rho, double p) { return sqrt(R3_GAM * p / rho); }

// conserved point value -> floored primitives  fv_rec3_2d.cu:71-79
__device__ __forceinline__ void r3_w(const double U[4], double W[4])
{
    const double r = smax<double>(U[0], R3_RHOFLOOR);
    const double u = U[1] / r, v = U[2] / r;
    const double p = (R3_GAM - 1.0) * (U[3] - 0.5 * r * (u * u + v * v));
    W[0] = r; W[1] = u; W[2] = v; W[3] = smax<double>(p, R3_PFLOOR);
}

// pressure of a conserved state                fv_rec3_2d.cu:81-87
__device__ __forceinline__ double r3_p(const double U[4])
{
    const double r = smax<double>(U[0], R3_RHOFLOOR);
    const double u = U[1] / r, v = U[2] / r;
    return (R3_GAM - 1.0) * (U[3] - 0.5 * r * (u * u + v * v));
}

// HLLC with Davis bounds and each side's star state, in the face-normal
// frame (rho, un, ut, p); a y-face swaps (u, v) in and the momentum
// fluxes back, which for the normal (0, 1) equals the reference's rotation
// bit for bit                                  fv_rec3_2d.cu:90-123
__device__ void r3_hllc(const double L[4], const double R[4], double F[4])
{
    const double rL = L[0], uL = L[1], tL = L[2], pL = L[3];
    const double rR = R[0], uR = R[1], tR = R[2], pR = R[3];
    const double cL = r3_snd(rL, pL), cR = r3_snd(rR, pR);
    const double EL = pL / (R3_GAM - 1.) + 0.5 * rL * (uL * uL + tL * tL);
    const double ER = pR / (R3_GAM - 1.) + 0.5 * rR * (uR * uR + tR * tR);
    const double SL = smin<double>(uL - cL, uR - cR), SR = smax<double>(uL + cL, uR + cR);
    const double FL[4] = {rL * uL, rL * uL * uL + pL, rL * uL * tL, (EL + pL) * uL};
    const double FR[4] = {rR * uR, rR * uR * uR + pR, rR * uR * tR, (ER + pR) * uR};
    if (SL >= 0.) { for (int q = 0; q < 4; q++) F[q] = FL[q]; return; }
    if (SR <= 0.) { for (int q = 0; q < 4; q++) F[q] = FR[q]; return; }
    const double dL = rL * (SL - uL), dR = rR * (SR - uR);
    const double Ss = (pR - pL + dL * uL - dR * uR) / (dL - dR);
    const bool left = Ss >= 0.;
    const double rK = left ? rL : rR, uK = left ? uL : uR, tK = left ? tL : tR, pK = left ? pL : pR;
    const double EK = left ? EL : ER, SK = left ? SL : SR;
    const double f = rK * (SK - uK) / (SK - Ss);
    const double Us[4] = {f, f * Ss, f * tK, f * (EK / rK + (Ss - uK) * (Ss + pK / (rK * (SK - uK))))};
    const double U[4] = {rK, rK * uK, rK * tK, EK};
    for (int q = 0; q < 4; q++) F[q] = (left ? FL[q] : FR[q]) + SK * (Us[q] - U[q]);
}

// Zhang-Shu scaling of a face state toward its cell average (linear for
// rho, 25-step bisection for p), then its floored primitives: the density,
// velocity and pressure that the pressure test forms are the primitives'
// own unless the bisection moved the state, so they are reused (the same
// operations on the same values as scaling, then converting)
//                                               fv_rec3_2d.cu:125-145, :71-79
__device__ __forceinline__ void r3_scale_w(const double Ub[4], double U[4], double W[4])
{
    if (U[0] < R3_RHOFLOOR) {
        const double d = Ub[0] - U[0];
        const double th = (d > 0.) ? (Ub[0] - R3_RHOFLOOR) / d : 0.;
        for (int q = 0; q < 4; q++) U[q] = Ub[q] + th * (U[q] - Ub[q]);
    }
    double r = smax<double>(U[0], R3_RHOFLOOR);
    double u = U[1] / r, v = U[2] / r;
    double p = (R3_GAM - 1.0) * (U[3] - 0.5 * r * (u * u + v * v));
    if (p < R3_PFLOOR) {
        double lo = 0., hi = 1.;
        for (int it = 0; it < 25; it++) {
            const double mid = 0.5 * (lo + hi);
            double V[4];
            for (int q = 0; q < 4; q++) V[q] = Ub[q] + mid * (U[q] - Ub[q]);
            if (V[0] >= R3_RHOFLOOR && r3_p(V) >= R3_PFLOOR) lo = mid;
            else hi = mid;
        }
        for (int q = 0; q < 4; q++) U[q] = Ub[q] + lo * (U[q] - Ub[q]);
        r = smax<double>(U[0], R3_RHOFLOOR);
        u = U[1] / r;
        v = U[2] / r;
        p = (R3_GAM - 1.0) * (U[3] - 0.5 * r * (u * u + v * v));
    }
    W[0] = r; W[1] = u; W[2] = v; W[3] = smax<double>(p, R3_PFLOOR);
}

// ---- the same operations with the quotients and roots of fvb_ieee.cuh ------
// Each returns the bits of its operator form above while its range tests hold
// (`ok` stays true); the caller evaluates the operator form otherwise.
constexpr double R3_GM1 = R3_GAM - 1.0, R3_YGM1 = 1.0 / R3_GM1;

// Velocity and pressure of a conserved state; r: the floored density.  (The
// pressure takes nothing from a small momentum: its square is 0.  The velocities
// do, so who uses them tests that.)
__device__ __forceinline__ double r3_p_of(const double U[4], double &r, double &u, double &v)
{
    r = smax<double>(U[0], R3_RHOFLOOR);
    const double y = recip(r);
    u = quot(U[1], r, y);
    v = quot(U[2], r, y);
    return R3_GM1 * (U[3] - 0.5 * r * (u * u + v * v));
}
__device__ __forceinline__ double r3_p_near(const double U[4], double &r, double &u, double &v, bool &ok)
{
    const double p = r3_p_of(U, r, u, v);
    ok = ok && pos_ok(r) && fin_ok(U[1], U[2]) && fin_ok(U[3]);
    return p;
}

__device__ __noinline__ void r3_scale_any(const double Ub[4], double U[4], double W[4])
{
    r3_scale_w(Ub, U, W);
}

// r3_scale_w of a face state that clears its floors (nearly all): converted
// at once; false: it needs the scaling, or is out of range.  (Momenta out of
// range above give no pressure that clears the floor.)
__device__ __forceinline__ bool r3_clear_near(const double U[4], double W[4])
{
    W[3] = r3_p_of(U, W[0], W[1], W[2]);
    return U[0] >= R3_RHOFLOOR && pos_ok(U[0]) && fin_ok(U[3]) && !is_small(U[1], U[2]) && W[3] >= R3_PFLOOR;
}

// r3_scale_w with the bisection's pressures in the shared-reciprocal form
__device__ __forceinline__ void r3_scale_near(const double Ub[4], double U[4], double W[4])
{
    bool ok = true;
    double S[4] = {U[0], U[1], U[2], U[3]};
    if (S[0] < R3_RHOFLOOR) {
        const double d = Ub[0] - S[0];
        const double th = (d > 0.) ? (Ub[0] - R3_RHOFLOOR) / d : 0.;
#pragma unroll
        for (int q = 0; q < 4; q++) S[q] = Ub[q] + th * (S[q] - Ub[q]);
    }
    double p = r3_p_near(S, W[0], W[1], W[2], ok);
    if (p < R3_PFLOOR) {
        double lo = 0., hi = 1.;
#pragma unroll 1
        for (int it = 0; it < 25; it++) {
            const double mid = 0.5 * (lo + hi);
            double V[4], r, u, v;
#pragma unroll
            for (int q = 0; q < 4; q++) V[q] = Ub[q] + mid * (S[q] - Ub[q]);
            const double pv = r3_p_near(V, r, u, v, ok);
            const bool in = V[0] >= R3_RHOFLOOR && pv >= R3_PFLOOR;
            lo = in ? mid : lo;
            hi = in ? hi : mid;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) S[q] = Ub[q] + lo * (S[q] - Ub[q]);
        p = r3_p_near(S, W[0], W[1], W[2], ok);
    }
    W[3] = smax<double>(p, R3_PFLOOR);
    if (!(ok && num_ok(S[1], S[2]))) {
        // (by copies, so that the arrays of the usual path stay in registers)
        double B[4], X[4];
#pragma unroll
        for (int q = 0; q < 4; q++) { B[q] = Ub[q]; S[q] = U[q]; }
        double T[4] = {S[0], S[1], S[2], S[3]};
        r3_scale_any(B, T, X);
#pragma unroll
        for (int q = 0; q < 4; q++) W[q] = X[q];
    }
}

// HLLC of floored face states (rho, un, ut, p)
__device__ __forceinline__ bool r3_hllc_near(const double L[4], const double R[4], double F[4])
{
    const double rL = L[0], uL = L[1], tL = L[2], pL = L[3];
    const double rR = R[0], uR = R[1], tR = R[2], pR = R[3];
    const double yL = recip(rL), yR = recip(rR);
    const double xL = quot(R3_GAM * pL, rL, yL), xR = quot(R3_GAM * pR, rR, yR);
    const double cL = root(xL), cR = root(xR);
    bool ok = pos_ok(rL) && pos_ok(rR) && pos_ok(xL) && pos_ok(xR) && fin_ok(pL, pR);  // (p >= 1e-9)
    const double SL = smin<double>(uL - cL, uR - cR), SR = smax<double>(uL + cL, uR + cR);
    const bool supL = SL >= 0., sup = supL || SR <= 0.;
    const double dL = rL * (SL - uL), dR = rR * (SR - uR);
    const double sn = pR - pL + dL * uL - dR * uR, sd = dL - dR;
    const double Ss = squot(sn, sd, recip(sd));
    // the side whose state the flux needs: the upwind one, or the contact's
    const bool left = sup ? supL : Ss >= 0.;
    const double rK = left ? rL : rR, uK = left ? uL : uR, tK = left ? tL : tR, pK = left ? pL : pR;
    const double SK = left ? SL : SR, yK = left ? yL : yR, dK = left ? dL : dR;  // dK = rK (SK - uK)
    const double EK = quot(pK, R3_GM1, R3_YGM1) + 0.5 * rK * (uK * uK + tK * tK);
    const double mK = rK * uK;
    const double F0 = mK, F1 = mK * uK + pK, F2 = mK * tK, F3 = (EK + pK) * uK;
    if (sup) {
        F[0] = F0; F[1] = F1; F[2] = F2; F[3] = F3;
        return ok;
    }
    const double sq = SK - Ss;
    const double f = squot(dK, sq, recip(sq));
    const double Us3 = f * (quot(EK, rK, yK) + (Ss - uK) * (Ss + squot(pK, dK, recip(dK))));
    F[0] = F0 + SK * (f - rK);
    F[1] = F1 + SK * (f * Ss - mK);
    F[2] = F2 + SK * (f * tK - rK * tK);
    F[3] = F3 + SK * (Us3 - EK);
    return ok && den_ok(sd) && den_ok(sq) && den_ok(dK) && num_ok(sn) && fin_ok(EK);
}

__device__ __noinline__ void r3_hllc_any(const double L[4], const double R[4], double F[4]) { r3_hllc(L, R, F); }

// 2x2-block limiter on U[c][q] (cells c = 0..3: (i0,j0), (i0+1,j0),
// (i0,j0+1), (i0+1,j0+1)); true if the block changed; *brutal counts a
// block whose mean itself needed the floor fix  fv_rec3_2d.cu:252-337
__device__ bool r3_limit_block(double U[4][4], int *brutal)
{
    double Ub[4] = {0., 0., 0., 0.};
    for (int c = 0; c < 4; c++)
        for (int q = 0; q < 4; q++) Ub[q] += 0.25 * U[c][q];
    const double pb = r3_p(Ub);
    if (Ub[0] < R3_RHOFLOOR || pb < R3_PFLOOR) {
        ++*brutal;
        const double rb = smax<double>(Ub[0], 10. * R3_RHOFLOOR);
        const double Efix = (10. * R3_PFLOOR) / (R3_GAM - 1.) + 0.5 * (Ub[1] * Ub[1] + Ub[2] * Ub[2]) / rb;
        Ub[0] = rb;
        Ub[3] = smax<double>(Ub[3], Efix);
    }
    double C[4][4];
    for (int q = 0; q < 4; q++) {
        C[0][q] = (9. * U[0][q] - 3. * U[1][q] - 3. * U[2][q] + U[3][q]) * 0.25;
        C[1][q] = (9. * U[1][q] - 3. * U[0][q] - 3. * U[3][q] + U[2][q]) * 0.25;
        C[2][q] = (9. * U[2][q] - 3. * U[3][q] - 3. * U[0][q] + U[1][q]) * 0.25;
        C[3][q] = (9. * U[3][q] - 3. * U[2][q] - 3. * U[1][q] + U[0][q]) * 0.25;
    }
    double th = 1.;
    for (int c = 0; c < 4; c++)
        if (C[c][0] < R3_RHOFLOOR) {
            const double d = Ub[0] - C[c][0];
            if (d > 0.) th = smin<double>((Ub[0] - R3_RHOFLOOR) / d, th);
        }
    if (th < 1.)
        for (int c = 0; c < 4; c++)
            for (int q = 0; q < 4; q++) {
                U[c][q] = Ub[q] + th * (U[c][q] - Ub[q]);
                C[c][q] = Ub[q] + th * (C[c][q] - Ub[q]);
            }
    bool bad = false;
    for (int c = 0; c < 4; c++)
        if (C[c][0] < R3_RHOFLOOR || r3_p(C[c]) < R3_PFLOOR) bad = true;
    if (bad) {
        double lo = 0., hi = 1.;
        for (int it = 0; it < 30; it++) {
            const double mid = 0.5 * (lo + hi);
            bool ok = true;
            for (int c = 0; c < 4 && ok; c++) {
                double V[4];
                for (int q = 0; q < 4; q++) V[q] = Ub[q] + mid * (C[c][q] - Ub[q]);
                if (V[0] < R3_RHOFLOOR || r3_p(V) < R3_PFLOOR) ok = false;
            }
            if (ok) lo = mid;
            else hi = mid;
        }
        for (int c = 0; c < 4; c++)
            for (int q = 0; q < 4; q++) U[c][q] = Ub[q] + lo * (U[c][q] - Ub[q]);
    }
    return th < 1. || bad;
}

__device__ __noinline__ double r3_lam_any(double U0, double U1, double U2, double U3)
{
    const double U[4] = {U0, U1, U2, U3};
    double W[4];
    r3_w(U, W);
    return fabs(W[1]) + fabs(W[2]) + r3_snd(W[0], W[3]);
}

// Is this lane's corner of its 2x2 block (lanes l, l ^ 1, l ^ 16, l ^ 17) well
// clear of the floors?  If all four are, the block needs no limiter: its mean,
// the corners' average, then clears them too (the pressure is concave; with
// rho, p >= 1e-6 and E <= 1e6 the rounding of any of these is below 1e-7).
__device__ __forceinline__ bool r3_clear_corner(const double U[4])
{
    double C[4], r, u, v;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double a = __shfl_xor_sync(0xffffffffu, U[q], 1), b = __shfl_xor_sync(0xffffffffu, U[q], 16);
        const double o = __shfl_xor_sync(0xffffffffu, U[q], 17);
        C[q] = (9. * U[q] - 3. * a - 3. * b + o) * 0.25;
    }
    bool ok = true;
    const double p = r3_p_near(C, r, u, v, ok);
    return ok && C[0] >= 1e-6 && p >= 1e-6 && C[3] <= 1e6;
}

// The limiter (r3_limit_block) of a warp's eight 2x2 blocks, each lane on its
// own cell and corner, so that a bisection step is one pressure for all four
// corners and not four in a row (and in place of one lane a block: 9 us a warp
// on the shock).  A block that turns out to need none is left as it is; one
// whose mean is not admissible or whose values leave the quotients' range goes
// to r3_limit_block, one lane.
__device__ __noinline__ void r3_limit_warp_any(double U[4], bool take, int lane, int *brutal)
{
    const int base = lane & 14, mine = (lane >> 4) * 2 + (lane & 1);
    double T[4][4];
    for (int c = 0; c < 4; c++)
        for (int q = 0; q < 4; q++) T[c][q] = __shfl_sync(0xffffffffu, U[q], base + (c & 1) + 16 * (c >> 1));
    if (take && mine == 0) r3_limit_block(T, brutal);
    for (int c = 0; c < 4; c++)
        for (int q = 0; q < 4; q++) {
            const double v = __shfl_sync(0xffffffffu, T[c][q], base);
            if (take && c == mine) U[q] = v;
        }
}

__device__ __noinline__ void r3_limit_warp_(double U[4], bool in, int lane, int *brutal)
{
    const int base = lane & 14;
    const unsigned block = 0x30003u << base;
    double Ub[4], C[4], r, u, v;
    bool ok = true;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        Ub[q] = 0.;
#pragma unroll
        for (int c = 0; c < 4; c++)
            Ub[q] += 0.25 * __shfl_sync(0xffffffffu, U[q], base + (c & 1) + 16 * (c >> 1));
        const double a = __shfl_xor_sync(0xffffffffu, U[q], 1), b = __shfl_xor_sync(0xffffffffu, U[q], 16);
        const double o = __shfl_xor_sync(0xffffffffu, U[q], 17);
        C[q] = (9. * U[q] - 3. * a - 3. * b + o) * 0.25;
    }
    const double pb = r3_p_near(Ub, r, u, v, ok);
    ok = ok && Ub[0] >= R3_RHOFLOOR && pb >= R3_PFLOOR;
    double th = 1.;
    if (C[0] < R3_RHOFLOOR) {
        const double d = Ub[0] - C[0];
        if (d > 0.) th = smin<double>((Ub[0] - R3_RHOFLOOR) / d, th);
    }
    th = smin<double>(__shfl_xor_sync(0xffffffffu, th, 1), th);
    th = smin<double>(__shfl_xor_sync(0xffffffffu, th, 16), th);
    if (th < 1.)
#pragma unroll
        for (int q = 0; q < 4; q++) C[q] = Ub[q] + th * (C[q] - Ub[q]);
    const double pc = r3_p_near(C, r, u, v, ok);
    const bool bad = (__ballot_sync(0xffffffffu, in && (C[0] < R3_RHOFLOOR || pc < R3_PFLOOR)) & block) != 0;
    double lo = 0., hi = 1.;
    if (__any_sync(0xffffffffu, bad)) {
#pragma unroll 1
        for (int it = 0; it < 30; it++) {
            const double mid = 0.5 * (lo + hi);
            double V[4];
#pragma unroll
            for (int q = 0; q < 4; q++) V[q] = Ub[q] + mid * (C[q] - Ub[q]);
            const double p = r3_p_near(V, r, u, v, ok);
            const bool out = (__ballot_sync(0xffffffffu, V[0] < R3_RHOFLOOR || p < R3_PFLOOR) & block) != 0;
            hi = out ? mid : hi;
            lo = out ? lo : mid;
        }
    }
    const unsigned odd = __ballot_sync(0xffffffffu, in && !ok);
    if (odd) r3_limit_warp_any(U, in && (odd & block) != 0, lane, brutal);
    if ((odd & block) == 0)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (th < 1.) U[q] = Ub[q] + th * (U[q] - Ub[q]);
            if (bad) U[q] = Ub[q] + lo * (U[q] - Ub[q]);
        }
}
// (with copies, so that the usual path's state stays in registers)
__device__ __forceinline__ void r3_limit_warp(double U[4], bool in, int lane, int &brutal)
{
    double X[4] = {U[0], U[1], U[2], U[3]};
    int nb = 0;
    r3_limit_warp_(X, in, lane, &nb);
    brutal += nb;
#pragma unroll
    for (int q = 0; q < 4; q++) U[q] = X[q];
}

__device__ __forceinline__ long long r3_at(const GridDev &gd, int j, int i)
{
    return (long long)(j + RG) * gd.pitch + (i + RG) + gd.xoff;
}

// the flux of face f of a tile's x- or y-faces into its plane set; SCALE: with
// the scaling of its states, else only if both clear the floors (false: not
// stored)
template <bool XF, bool SCALE>
__device__ __forceinline__ bool r3_face(const double *Q, int f, double *FP)
{
    constexpr int W = XF ? RTX + 1 : RTX, st = XF ? 1 : RSW, os = XF ? RTY * (RTX + 1) : (RTY + 1) * RTX;
    constexpr int QN = XF ? 1 : 2, QT = XF ? 2 : 1;
    const int r = f / W, c = f - r * W;
    const int b = (r + RG) * RSW + (c + RG), a = b - st;
    double UL[4], UR[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double *v = Q + q * RPL;
        const double um = v[a - st], uc = v[a], up = v[b], u2 = v[b + st];
        UL[q] = fma(2., up, -um + 5. * uc) * (1. / 6.);  // (2 up is exact: the reference's own rounding)
        UR[q] = (fma(2., uc, 5. * up) - u2) * (1. / 6.);
    }
    double WL[4], WR[4], Fn[4];
    if constexpr (SCALE) {
        const double UbL[4] = {Q[a], Q[RPL + a], Q[2 * RPL + a], Q[3 * RPL + a]};
        const double UbR[4] = {Q[b], Q[RPL + b], Q[2 * RPL + b], Q[3 * RPL + b]};
        r3_scale_near(UbL, UL, WL);
        r3_scale_near(UbR, UR, WR);
    } else {
        const bool l = r3_clear_near(UL, WL), r2 = r3_clear_near(UR, WR);
        if (!(l && r2)) return false;
    }
    const double L[4] = {WL[0], WL[QN], WL[QT], WL[3]}, Rr[4] = {WR[0], WR[QN], WR[QT], WR[3]};
    if (!r3_hllc_near(L, Rr, Fn)) {
        if (!SCALE) return false;
        double A[4], B[4], G[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) { A[q] = L[q]; B[q] = Rr[q]; }
        r3_hllc_any(A, B, G);
#pragma unroll
        for (int q = 0; q < 4; ++q) Fn[q] = G[q];
    }
    double *o = FP + f;
    o[0] = Fn[0]; o[QN * os] = Fn[1]; o[QT * os] = Fn[2]; o[3 * os] = Fn[3];
    return true;
}

// One SSP-RK3 stage                             fv_rec3_2d.cu:166-353
// The shock's tiles, with bisected faces and limited blocks, cost several
// times the others: with a fixed share of the tiles a CTA the SMs were busy
// 79 % of a stage (1024^2 circular Sod: a stage 105 us, now 94), so a CTA takes
// its next tile when it comes to it (tile_queue, fvb_device.cuh).
__global__ void __launch_bounds__(RNT, 2) rec3_stage_kernel(const __grid_constant__ GridDev gd, int stage, int ntiles)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    double *sm = reinterpret_cast<double *>(smem_raw);
    double *U0 = sm + ROU0;  // [4][RTY][RTX]
    double *FX = sm + ROFX;  // [4][RTY][RTX+1]
    double *FY = sm + ROFY;  // [4][RTY+1][RTX]
    __shared__ double s_red[RNT / 32];
    __shared__ __align__(8) uint64_t s_bar[3];
    __shared__ int s_err, s_nlist, s_next;
    __shared__ unsigned short s_list[RNF];  // faces that need the scaling
    const int tid = threadIdx.x, lane = tid & 31, n = gd.n;
    const double *u0 = (const double *)gd.st[0];
    double *out = (double *)(stage == 1 ? gd.k1 : stage == 2 ? gd.k2 : gd.st[0]);
    const double inv_h = 1. / gd.h;
    const double ca = stage == 1 ? 0. : stage == 2 ? 0.75 : 1. / 3.;
    const double cb = stage == 1 ? 1. : stage == 2 ? 0.25 : 2. / 3.;
    int brutal = 0;
    double lacc = 0.0;

    RPipe pipe(s_bar, &s_err, tid);
    grid_dependency();
    int t = blockIdx.x, buf = 0;
    // failure injection (fvb_debug_drop): CTA 0 issues no first box load, or no U0 load for its first tile
    const int armed = blockIdx.x == 0 && gd.tmap ? *(volatile int *)&gd.ctrl->drop_load : 0;
    const bool drop = armed == FVB_DROP_BOX, drop_u0 = armed == FVB_DROP_U0 && stage >= 2;
    if (t < ntiles && !drop) pipe.start_box(gd, stage, t, sm, 0, tid);
    const TileCtl ctl = tile_control<P64>(gd.ctrl, stage, tid == 0 && t == 0);
    int *queue = tile_queue(gd.ctrl, stage);
    if (tid == 0 && t == 0) clear_tile_queue(gd.ctrl, stage);
    pipe.finish_box(gd, 0, t < ntiles);
    if ((drop || drop_u0) && tid == 0) gd.ctrl->drop_load = 0;
    if (t < ntiles && s_err) {
        // the box never arrived: record it, stop
        if (tid == 0) gd.ctrl->status = FVB_ERR_TIMEOUT;
        t = ntiles;
    }
    if (!ctl.run) t = ntiles;
    while (t < ntiles) {
        const int tx0 = (t % gd.tiles_x) * RTX, ty0 = (t / gd.tiles_x) * RTY;
        const bool u0_tma = stage >= 2 && gd.tmap;
        if (u0_tma && !drop_u0) pipe.start_u0(gd, tx0, ty0, U0, tid);
        const double *Q = sm + buf * RPipe::BOX;  // [4][RSH][RSW] stage input
        if (tid == 0) s_nlist = 0;
        __syncthreads();
        // ---- faces: x-face (r, c) lies between cells c-1 and c; a face with
        //      a state below the floors goes on the list ------------------------
        //      (faces of cells outside the grid are left out)
        for (int f = tid; f < RTY * (RTX + 1); f += RNT) {
            const int r = f / (RTX + 1), c = f - r * (RTX + 1);
            if (ty0 + r < n && tx0 + c <= n && !r3_face<true, false>(Q, f, FX))
                s_list[atomicAdd(&s_nlist, 1)] = (unsigned short)f;
        }
        // the next tile, taken while the y-faces are computed
        const int q = tid == 0 && ntiles > (int)gridDim.x ? (int)gridDim.x + atomicAdd(queue, 1) : ntiles;
        for (int f = tid; f < (RTY + 1) * RTX; f += RNT) {
            const int r = f / RTX, c = f - r * RTX;
            if (ty0 + r <= n && tx0 + c < n && !r3_face<false, false>(Q, f, FY))
                s_list[atomicAdd(&s_nlist, 1)] = (unsigned short)(f + RTY * (RTX + 1));
        }
        if (tid == 0) s_next = q;
        __syncthreads();
        const int next = s_next;
        const bool has_next = next < ntiles;
        if (has_next) pipe.start_box(gd, stage, next, sm + (buf ^ 1) * RPipe::BOX, buf ^ 1, tid);
        // ---- the listed faces, one a thread, so that their bisections (25
        //      dependent steps a side) run side by side ---------------------------
        const int nl = s_nlist;
        if (nl > 0) {
            for (int m = tid; m < nl; m += RNT) {
                const int f = s_list[m];
                if (f < RTY * (RTX + 1)) r3_face<true, true>(Q, f, FX);
                else r3_face<false, true>(Q, f - RTY * (RTX + 1), FY);
            }
            __syncthreads();
        }
        // ---- cells, a warp on 2 rows of 16, so that a 2x2 block is four lanes:
        //      residual in the serial scatter's order, RK combination, the
        //      block limiter, stores with the periodic ghost images, stage-3
        //      wave speed ------------------------------------------------------
        if (!has_next) grid_release();
        const bool u0_ok = !u0_tma || pipe.wait(2);
        for (int w = tid >> 5; w < (RTY / 2) * (RTX / 16); w += RNT / 32) {
            const int r = 2 * (w / (RTX / 16)) + (lane >> 4), c = 16 * (w % (RTX / 16)) + (lane & 15);
            const int i = tx0 + c, j = ty0 + r;
            const bool in = i < n && j < n && u0_ok;  // (n even: a block is inside as a whole)
            double U[4] = {1., 0., 0., 2.5};
            if (in) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const double *fx = FX + q * RTY * (RTX + 1) + r * (RTX + 1) + c;
                    const double *fy = FY + q * (RTY + 1) * RTX + r * RTX + c;
                    const double tl = fx[0] * inv_h, tr = -fx[1] * inv_h;      // left face in, right face out
                    const double tb = fy[0] * inv_h, tt = -fy[RTX] * inv_h;    // bottom in, top out
                    double L;
                    if (i > 0 && j > 0) L = ((tb + tl) + tr) + tt;
                    else if (i == 0 && j > 0) L = ((tb + tr) + tt) + tl;
                    else if (i > 0) L = ((tl + tr) + tt) + tb;
                    else L = ((tr + tt) + tl) + tb;
                    const double qb = Q[q * RPL + (r + RG) * RSW + (c + RG)];
                    const double qa = stage == 1 ? qb
                                      : u0_tma   ? U0[(q * RTY + r) * RTX + c]
                                                 : u0[r3_at(gd, j, i) + q * gd.plane];
                    U[q] = ca * qa + cb * (qb + ctl.dt * L);
                }
            }
            const bool clear = r3_clear_corner(U);  // (every lane: it shuffles)
            if (__any_sync(0xffffffffu, in && !clear)) r3_limit_warp(U, in, lane, brutal);
            if (in) {
                put_cell<double>(gd, out, j, i, U);
                if (stage == 3) {
                    double rr, u, v;
                    bool ok = true;
                    const double p = smax<double>(r3_p_near(U, rr, u, v, ok), R3_PFLOOR);
                    const double x = quot(R3_GAM * p, rr, recip(rr));
                    const double lam = fabs(u) + fabs(v) + root(x);
                    lacc = smax<double>(ok && pos_ok(x) ? lam : r3_lam_any(U[0], U[1], U[2], U[3]), lacc);
                }
            }
        }
        if (stage == 3 && tid == 0 && t == 0) leader_finish<P64>(gd.ctrl);
        pipe.finish_box(gd, buf ^ 1, has_next);
        if (s_err) {
            if (tid == 0) gd.ctrl->status = FVB_ERR_TIMEOUT;
            break;
        }
        t = next;
        buf ^= 1;
    }
    if (!drop && !drop_u0) pipe.drain();
    if (brutal) atomicAdd(&gd.ctrl->aux, (unsigned long long)brutal);
    if (stage == 3) {
        for (int o = 16; o > 0; o >>= 1) lacc = fmax(lacc, __shfl_xor_sync(0xffffffffu, lacc, o));
        if ((tid & 31) == 0) s_red[tid >> 5] = lacc;
        __syncthreads();
        if (tid == 0) {
            double m = 0.0;
            for (int w = 0; w < RNT / 32; ++w) m = fmax(m, s_red[w]);
            if (m > 0.0) atomicMax(&gd.ctrl->lam_acc, (unsigned long long)__double_as_longlong(m));
        }
    }
}

// limiter pass over a whole state (after an initial state is set), one
// thread per 2x2 block                          fv_rec3_2d.cu:542
__global__ void rec3_limit_kernel(const GridDev gd, double *buf)
{
    const int nb = gd.n / 2;
    int brutal = 0;
    for (long long kb = blockIdx.x * (long long)blockDim.x + threadIdx.x; kb < (long long)nb * nb;
         kb += (long long)blockDim.x * gridDim.x) {
        const int jb = (int)(kb / nb), ib = (int)(kb - (long long)jb * nb);
        double U[4][4];
        for (int cc = 0; cc < 4; cc++) {
            const long long e = r3_at(gd, 2 * jb + (cc >> 1), 2 * ib + (cc & 1));
            for (int q = 0; q < 4; q++) U[cc][q] = buf[e + q * gd.plane];
        }
        if (r3_limit_block(U, &brutal))
            for (int cc = 0; cc < 4; cc++) {
                const long long e = r3_at(gd, 2 * jb + (cc >> 1), 2 * ib + (cc & 1));
                for (int q = 0; q < 4; q++) buf[e + q * gd.plane] = U[cc][q];
            }
    }
    if (brutal) atomicAdd(&gd.ctrl->aux, (unsigned long long)brutal);
}

// |u| + |v| + c of the floored primitives, max into ctrl->lam_acc
__global__ void rec3_lam_kernel(const GridDev gd, const double *buf)
{
    __shared__ double sh[32];
    const long long n2 = (long long)gd.n * gd.n;
    double m = 0.0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n2;
         k += (long long)blockDim.x * gridDim.x) {
        const long long e = r3_at(gd, (int)(k / gd.n), (int)(k % gd.n));
        double U[4], W[4];
        for (int q = 0; q < 4; q++) U[q] = buf[e + q * gd.plane];
        r3_w(U, W);
        m = fmax(m, fabs(W[1]) + fabs(W[2]) + r3_snd(W[0], W[3]));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) b = fmax(b, sh[w]);
        atomicMax(&gd.ctrl->lam_acc, (unsigned long long)__double_as_longlong(b));
    }
}

// initial cell averages of fv_rec3's cases: 0 circular Sod (sharp,
// midpoint), 1 the paper's isentropic vortex on [0,10]^2, 2 the Gresho
// low-Mach vortex; 4x4 Gauss averages for the smooth ones
//                                               fv_rec3_2d.cu:356-416
__device__ void r3_pv(double x, double y, double *ro, double *uo, double *vo, double *po)
{
    const double gg = R3_GAM, eps = 5., pi = 3.14159265358979323846;
    const double dx = x - 5., dy = y - 5., r2 = dx * dx + dy * dy;
    const double f = eps / (2. * pi) * exp(0.5 * (1. - r2));
    const double dT = -(gg - 1.) * eps * eps / (8. * gg * pi * pi) * exp(1. - r2);
    double T = 1. + dT;
    if (T < 1e-6) T = 1e-6;
    *ro = pow(T, 1. / (gg - 1.));
    *po = pow(T, gg / (gg - 1.));
    *uo = -f * dy;
    *vo = f * dx;
}
__device__ void r3_lmv(double x, double y, double p0, double *ro, double *uo, double *vo, double *po)
{
    const double dx = x - 0.5, dy = y - 0.5, r = sqrt(dx * dx + dy * dy);
    const double vp = r < 0.2 ? 5. * r : r < 0.4 ? 2. - 5. * r : 0.;
    const double ir = (r > 1e-30) ? 1. / r : 0.;
    *ro = 1.; *uo = -vp * dy * ir; *vo = vp * dx * ir;
    *po = r < 0.2 ? p0 + 12.5 * r * r : r < 0.4 ? p0 + 4. * log(5. * r) + 4. - 20. * r + 12.5 * r * r
                                                : p0 + 4. * log(2.) - 2.;
}

__global__ void rec3_ic_kernel(const GridDev gd, double *buf, int icase, double p0)
{
    const double gx[4] = {-0.861136311594053, -0.339981043584856, 0.339981043584856, 0.861136311594053};
    const double gw[4] = {0.347854845137454, 0.652145154862546, 0.652145154862546, 0.347854845137454};
    const int n = gd.n;
    const double h = gd.h;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < (long long)n * n;
         k += (long long)blockDim.x * gridDim.x) {
        const int j = (int)(k / n), i = (int)(k % n);
        const double xc = (i + 0.5) * h, yc = (j + 0.5) * h;
        double Qc[4] = {0., 0., 0., 0.};
        if (icase == 0) {
            const double r = sqrt((xc - 0.5) * (xc - 0.5) + (yc - 0.5) * (yc - 0.5));
            Qc[0] = r < 0.25 ? 10.0 : 0.125;
            Qc[3] = (r < 0.25 ? 10.0 : 0.1) / (R3_GAM - 1.);
        } else {
            for (int a = 0; a < 4; a++)
                for (int b = 0; b < 4; b++) {
                    const double x = xc + 0.5 * h * gx[a], y = yc + 0.5 * h * gx[b];
                    double r, u, v, p;
                    if (icase == 1) r3_pv(x, y, &r, &u, &v, &p);
                    else r3_lmv(x, y, p0, &r, &u, &v, &p);
                    const double w = 0.25 * gw[a] * gw[b];
                    Qc[0] += w * r; Qc[1] += w * r * u; Qc[2] += w * r * v;
                    Qc[3] += w * (p / (R3_GAM - 1.) + 0.5 * r * (u * u + v * v));
                }
        }
        const long long e = r3_at(gd, j, i);
        for (int q = 0; q < 4; q++) buf[e + q * gd.plane] = Qc[q];
    }
}

size_t rec3_smem() { return sizeof(double) * (ROFY + 4 * (RTY + 1) * RTX); }

int sm_count()
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace

void rec3_tiles(int n, int &tiles_x, int &tiles)
{
    tiles_x = (n + RTX - 1) / RTX;
    tiles = tiles_x * ((n + RTY - 1) / RTY);
}

void rec3_tile(int &tx, int &ty)
{
    tx = RTX;
    ty = RTY;
}

cudaError_t rec3_launch_stage(const GridDev &gd, int stage, int tiles, cudaStream_t s)
{
    LaunchFacts f{};
    cudaError_t e = launch_facts((const void *)rec3_stage_kernel, RNT, rec3_smem(), f);
    if (e != cudaSuccess) return e;
    const int cap = f.ctas_per_sm * f.sms;
    void *args[] = {(void *)&gd, (void *)&stage, (void *)&tiles};
    return launch_chained((const void *)rec3_stage_kernel, tiles < cap ? tiles : cap, RNT, rec3_smem(), s, args);
}

cudaError_t rec3_limit_into(const GridDev &gd, void *buf, cudaStream_t s)
{
    const long long nb = (long long)(gd.n / 2) * (gd.n / 2);
    const int blocks = (int)std::min<long long>((nb + 255) / 256, 4LL * sm_count());
    rec3_limit_kernel<<<blocks > 0 ? blocks : 1, 256, 0, s>>>(gd, (double *)buf);
    return cudaGetLastError();
}

cudaError_t rec3_lam_into(const GridDev &gd, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(&gd.ctrl->lam_acc, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    const long long n2 = (long long)gd.n * gd.n;
    const int blocks = (int)std::min<long long>((n2 + 255) / 256, 4LL * sm_count());
    rec3_lam_kernel<<<blocks, 256, 0, s>>>(gd, (const double *)gd.st[0]);
    return cudaGetLastError();
}

cudaError_t rec3_init_case(const GridDev &gd, int icase, double p0, cudaStream_t s)
{
    const long long n2 = (long long)gd.n * gd.n;
    const int blocks = (int)std::min<long long>((n2 + 255) / 256, 4LL * sm_count());
    rec3_ic_kernel<<<blocks, 256, 0, s>>>(gd, (double *)gd.st[0], icase, p0);
    return cudaGetLastError();
}

}  // namespace fvb
