// fvb_keep.cu -- the KEEP flux family of keep_fv_euler_2d.cu on the device.
//
// Collocated FV on conserved cell averages (g = 2), FP64.  Per face:
//   F = F_EC + (1 - phi) F_JST + phi F_RH
// with F_EC the entropy-conserving / kinetic-energy-preserving central flux,
// F_JST a 4th-order background dissipation, F_RH the MOVERS-RH scalar
// dissipation, and phi in {0, 1} the entropy-distance shock sensor scaled by
// the stage input's global maximum (keep_fv_euler_2d.cu:145-369).
//
// That maximum must be known before any flux, so a stage is two launches:
// keep_ed_kernel (per-cell entropy distance, block max, atomicMax into the
// step control) and keep_stage_kernel (tile in shared memory, every face
// once, divergence, RK combination with floors, stores with ghost images,
// and in stage 3 the wave-speed max for the next dt).  Both convert each
// cell of a tile once -- floored primitives, entropy and entropy variables
// -- and form every face's terms from those, so no face repeats the
// divisions and logarithms of its two cells.  The step control is the same
// device-side Ctrl as the UP path.
//
// What bounds it: instruction issue and latency, not memory (1024^2: 16 us of
// a stage at the copy bandwidth).  log and pow of every cell, once for each
// of the two kernels and for every halo, IEEE divisions and exp per face were
// 3340 instructions a cell; now a cell's entropy is formed once (the sensor
// pass leaves it in a plane for the stage kernel), quotients share
// reciprocals (fvb_ieee.cuh), a face evaluates the one dissipation its sensor
// selects, and exp is evaluated only next to the sensor's threshold: 1890
// instructions a cell, 202 -> 131 us a stage, bit-identical.  With registers
// in place of local arrays, step control once a CTA and chained launches: 108.
#include "fvb_aux.h"
#include "fvb_physics.cuh"
#include "fvb_device.cuh"
#include "fvb_ieee.cuh"

namespace fvb {
namespace {

constexpr double KG_MIN = 1e-14;

__device__ __forceinline__ double k_snd(double rho, double p, double gam) { return sqrt(gam * p / rho); }

// floored primitives and entropy s = ln(p / rho^gamma) of a conserved cell
//                                              keep_fv_euler_2d.cu:99-132
__device__ __forceinline__ void k_cell(const double U[4], double gam, double W[4], double Uf[4], double &s)
{
    double rho = smax<double>(U[0], KG_MIN), mx = U[1], my = U[2], E = U[3];
    double u = mx / rho, v = my / rho;
    W[0] = rho;
    W[1] = mx / rho;
    W[2] = my / rho;
    W[3] = smax<double>((gam - 1.) * (E - 0.5 * rho * (u * u + v * v)), KG_MIN);
    Uf[0] = rho; Uf[1] = mx; Uf[2] = my; Uf[3] = E;
    s = log(W[3] / pow(W[0], gam));
}

// entropy variables from primitives and their entropy   keep_fv:123-132
__device__ __forceinline__ void k_evars(const double W[4], double s, double gam, double V[4])
{
    double rho = W[0], u = W[1], v = W[2], p = W[3];
    V[0] = (gam - s) / (gam - 1.) - rho * (u * u + v * v) / (2. * p);
    V[1] = rho * u / p;
    V[2] = rho * v / p;
    V[3] = -rho / p;
}

// The same conversions with the quotients of fvb_ieee.cuh (one reciprocal of
// rho, one of p); true while their range tests hold.  ygm1: recip(gam - 1).
__device__ __forceinline__ bool k_prim_near(const double U[4], double gam, double W[4], double Uf[4])
{
    double rho = smax<double>(U[0], KG_MIN), mx = U[1], my = U[2], E = U[3];
    const double y = recip(rho);
    double u = quot(mx, rho, y), v = quot(my, rho, y);
    W[0] = rho;
    W[1] = u;
    W[2] = v;
    W[3] = smax<double>((gam - 1.) * (E - 0.5 * rho * (u * u + v * v)), KG_MIN);
    Uf[0] = rho; Uf[1] = mx; Uf[2] = my; Uf[3] = E;
    return pos_ok(rho) && num_ok(mx, my) && fin_ok(W[3]);
}

__device__ __forceinline__ bool k_evars_near(const double W[4], double s, double gam, double ygm1, double V[4])
{
    double rho = W[0], u = W[1], v = W[2], p = W[3];
    const double y = recip(p);
    const double ke = rho * (u * u + v * v), ru = rho * u, rv = rho * v;
    // (the reciprocal of 2 p is half that of p, exactly)
    V[0] = __dsub_rn(quot(gam - s, gam - 1., ygm1), quot(ke, 2. * p, 0.5 * y));
    V[1] = quot(ru, p, y);
    V[2] = quot(rv, p, y);
    V[3] = -quot(rho, p, y);
    // (ru and rv are the momenta but for a rounding or two, which k_prim_near
    // tests; beside the quotient of a gamma - s that is not 0 the last bits of a
    // small ke's are nothing)
    return pos_ok(p) && fin_ok(ke, s) && den_ok(gam - s);
}

// both in the operator form
__device__ __noinline__ void k_prim_any_(const double U[4], double gam, double W[4])
{
    double Uf[4], s;
    k_cell(U, gam, W, Uf, s);
}
__device__ __noinline__ double k_snd_any(double rho, double p, double gam) { return k_snd(rho, p, gam); }
__device__ __noinline__ void k_evars_any_(const double W[4], double s, double gam, double V[4])
{
    k_evars(W, s, gam, V);
}
// (called with copies, so that the arrays of the usual path stay in registers)
__device__ __forceinline__ void k_prim_any(const double U[4], double gam, double W[4])
{
    const double A[4] = {U[0], U[1], U[2], U[3]};
    double B[4];
    k_prim_any_(A, gam, B);
#pragma unroll
    for (int q = 0; q < 4; ++q) W[q] = B[q];
}
__device__ __forceinline__ void k_evars_any(const double W[4], double s, double gam, double V[4])
{
    const double A[4] = {W[0], W[1], W[2], W[3]};
    double B[4];
    k_evars_any_(A, s, gam, B);
#pragma unroll
    for (int q = 0; q < 4; ++q) V[q] = B[q];
}

// s = ln(p / rho^gamma)
__device__ __forceinline__ double k_entropy(const double W[4], double gam) { return log(W[3] / pow(W[0], gam)); }

// ECKEP central flux (Cartesian) and MOVERS-RH coefficient  keep_fv:145-219
// VL, VR: the two cells' entropy variables in the face frame (the Cartesian
// ones of k_evars with (u, v) -> (un, ut): for the normals (1, 0) and (0, 1)
// a relabelling and one exact negation, so the values are the reference's)
//
// The steps and their association order are the published flux's as the
// reference evaluates them (the ECKEP averages, the MOVERS-RH coefficient
// with its division by dV3^2 + 1e-16 and the sonic fix), not a rewrite:
// where dV3 is small that division amplifies a last-bit difference in its
// operands by many orders of magnitude, so any reassociation here moves the
// low-Mach vortex run outside the spread between the reference's own GPU
// and host builds, which is the tolerance this family is held to.
__device__ __forceinline__ void k_flux(const double WL[4], const double WR[4], const double VL[4],
                                       const double VR[4], double nx, double ny, double gam, double Fec[4],
                                       double *alphaS)
{
    const double rL = WL[0], uL = WL[1], vL = WL[2], pL = WL[3];
    const double rR = WR[0], uR = WR[1], vR = WR[2], pR = WR[3];
    const double unL = uL * nx + vL * ny, utL = -uL * ny + vL * nx;
    const double unR = uR * nx + vR * ny, utR = -uR * ny + vR * nx;
    const double EL = pL / (gam - 1.) + 0.5 * rL * (unL * unL + utL * utL);
    const double ER = pR / (gam - 1.) + 0.5 * rR * (unR * unR + utR * utR);
    const double UL[4] = {rL, rL * unL, rL * utL, EL};
    const double UR[4] = {rR, rR * unR, rR * utR, ER};
    const double FL[4] = {rL * unL, rL * unL * unL + pL, rL * unL * utL, (EL + pL) * unL};
    const double FR[4] = {rR * unR, rR * unR * unR + pR, rR * unR * utR, (ER + pR) * unR};
    const double dV0 = VR[0] - VL[0], dV1 = VR[1] - VL[1], dV2 = VR[2] - VL[2], dV3 = VR[3] - VL[3];
    const double dpsi = rR * unR - rL * unL;
    const double Fc0 = 0.5 * (FL[0] + FR[0]);
    const double unb = 0.5 * (unL + unR), utb = 0.5 * (utL + utR), pb = 0.5 * (pL + pR);
    const double Fc1 = Fc0 * unb + pb;
    const double Fc2 = Fc0 * utb;
    const double Feb = 0.5 * (FL[3] + FR[3]);
    const double num = dV0 * Fc0 + dV1 * Fc1 + dV2 * Fc2 + dV3 * Feb - dpsi;
    const double Fc3 = Feb - (num / (dV3 * dV3 + 1e-16)) * dV3;
    Fec[0] = Fc0;
    Fec[1] = Fc1 * nx - Fc2 * ny;
    Fec[2] = Fc1 * ny + Fc2 * nx;
    Fec[3] = Fc3;
    const double rav = 0.5 * (rL + rR);
    const double aav = k_snd(smax<double>(rav, KG_MIN), smax<double>(pb, KG_MIN), gam);
    const double l1 = fabs(unb - aav), l2 = fabs(unb), l3 = fabs(unb + aav);
    const double lmin = smin<double>(l1, smin<double>(l2, l3)), lmax = smax<double>(l1, smax<double>(l2, l3));
    double aS = lmax;
    for (int q = 0; q < 4; ++q) {
        const double dU = UR[q] - UL[q];
        double sk;
        if (fabs(dU) < 1e-12) {
            sk = lmin;
        } else {
            sk = fabs((FR[q] - FL[q]) / dU);
            if (sk >= lmax) sk = lmax;
            else if (sk <= lmin) sk = lmin;
        }
        if (sk < aS) aS = sk;
    }
    if (aS < 0.1) aS = (aS * aS + 0.1 * 0.1) / (2. * 0.1);
    *alphaS = aS;
}

__device__ __forceinline__ void load_cell(const double *buf, const GridDev &gd, int j, int i, double U[4])
{
    long long e = (long long)(j + gd.g) * gd.pitch + (i + gd.g) + gd.xoff;
    for (int q = 0; q < 4; ++q) U[q] = buf[e + q * gd.plane];
}

constexpr int KTX = 32, KTY = 15, KNT = 256, KG = 2;
constexpr int KSW = KTX + 2 * KG, KSH = KTY + 2 * KG, KPL = KSW * KSH;
constexpr int EW = KTX + 1, EH = KTY + 1, EPL = EW * EH;  // a tile and its right / top neighbours

// sqrt(gam p / rho) of positive rho, p; x: the root's argument for its test
__device__ __forceinline__ double k_snd_near(double rho, double p, double gam, double &x)
{
    x = quot(gam * p, rho, recip(rho));
    return root(x);
}

// what a launch's faces share
struct KFace {
    double gam, ygm1;    // gamma, recip(gamma - 1)
    double edmax, kphi;  // sensor scale, 12 / (edmax + 1e-30)
};

// -ln(0.95): the shock sensor's 1 - exp(-12 sed) > 0.05 is 12 sed above it
constexpr double KG_PHI = 0.051293294387550533427;

// One face's flux F_EC + (1 - phi) F_JST + phi F_RH in Cartesian components,
// the same operations as k_flux and the sum below it (k_face_any): phi is 0 or
// 1, so only the dissipation that it selects is evaluated (the other enters
// the reference's sum as a zero), and exp() only within 1e-10 of the sensor's
// threshold.  XF: an x-face, between cells a and b.  False: a range test
// failed, take k_face_any.
template <bool XF>
__device__ __forceinline__ bool k_face_near(const double *U, const double *W, const double *V, int a, int b,
                                            const KFace &k, double F[4])
{
    constexpr int st = XF ? 1 : KSW;
    constexpr int QN = XF ? 1 : 2, QT = XF ? 2 : 1;
    const double gam = k.gam;
    const double rL = U[a], pL = W[2 * KPL + a], rR = U[b], pR = W[2 * KPL + b];
    // face frame: (un, ut) = (u, v) on x-faces, (v, -u) on y-faces
    const double unL = W[(QN - 1) * KPL + a], unR = W[(QN - 1) * KPL + b];
    const double utL = XF ? W[KPL + a] : -W[a], utR = XF ? W[KPL + b] : -W[b];
    const double VL0 = V[a], VR0 = V[b], VL1 = V[QN * KPL + a], VR1 = V[QN * KPL + b];
    const double VL2 = XF ? V[QT * KPL + a] : -V[QT * KPL + a], VR2 = XF ? V[QT * KPL + b] : -V[QT * KPL + b];
    const double VL3 = V[3 * KPL + a], VR3 = V[3 * KPL + b];
    const double EL = quot(pL, gam - 1., k.ygm1) + 0.5 * rL * (unL * unL + utL * utL);
    const double ER = quot(pR, gam - 1., k.ygm1) + 0.5 * rR * (unR * unR + utR * utR);
    // Which products are rounded before a sum and which enter it fused is
    // fixed here by the _rn forms, so that the values do not depend on what
    // else a compiler finds to share (num / den below turns a last bit into
    // 1e-9 of the energy where dV3 is small).
    const double mL = __dmul_rn(rL, unL), mR = __dmul_rn(rR, unR);
    const double FL3 = __dmul_rn(EL + pL, unL), FR3 = __dmul_rn(ER + pR, unR);
    const double dV0 = VR0 - VL0, dV1 = VR1 - VL1, dV2 = VR2 - VL2, dV3 = VR3 - VL3;
    const double dpsi = __dsub_rn(mR, mL);
    const double Fc0 = 0.5 * __dadd_rn(mL, mR);
    const double unb = 0.5 * (unL + unR), utb = 0.5 * (utL + utR), pb = 0.5 * (pL + pR);
    const double Fc1 = Fc0 * unb + pb;
    const double Fc2 = __dmul_rn(Fc0, utb);
    const double Feb = 0.5 * __dadd_rn(FL3, FR3);
    const double num = dV0 * Fc0 + dV1 * Fc1 + dV2 * Fc2 + dV3 * Feb - dpsi;
    const double den = dV3 * dV3 + 1e-16;
    const double Fc3 = Feb - quot(num, den, recip(den)) * dV3;
    const double rav = 0.5 * (rL + rR);
    double sx;
    const double aav = k_snd_near(rav, pb, gam, sx);
    // (a small num's quotient changes the energy by nothing)
    bool ok = fin_ok(num) && pos_ok(den) && pos_ok(sx) && fin_ok(EL, ER);
    // shock sensor                                 keep_fv:249-258, :347-349
    const double dU0 = rR - rL, dU1 = U[KPL + b] - U[KPL + a], dU2 = U[2 * KPL + b] - U[2 * KPL + a];
    const double dU3 = U[3 * KPL + b] - U[3 * KPL + a];
    double ed = 0.;
    ed += dU0 * (VR0 - VL0);
    ed += dU1 * (V[KPL + b] - V[KPL + a]);
    ed += dU2 * (V[2 * KPL + b] - V[2 * KPL + a]);
    ed += dU3 * (VR3 - VL3);
    const double xs = fabs(ed) * k.kphi;
    bool shock = xs > KG_PHI;
    if (fabs(xs - KG_PHI) < 1e-10 * KG_PHI) {
        const double sed = fabs(ed) / (k.edmax + 1e-30);
        shock = (1. - exp(-12.0 * sed)) > 0.05;
    }
    const double fec[4] = {Fc0, XF ? Fc1 : -Fc2, XF ? Fc2 : Fc1, Fc3};
    if (!shock) {
        const double lamt = smax<double>(fabs(unL), fabs(unR)) + aav;
        const double aJST = (1.0 / 32.0) * lamt;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double *u = U + q * KPL;
            const double jst = __dmul_rn(aJST, u[b + st] - 3. * u[b] + 3. * u[a] - u[a - st]);
            F[q] = __dadd_rn(fec[q], jst);
        }
        return ok;
    }
    const double l1 = fabs(unb - aav), l2 = fabs(unb), l3 = fabs(unb + aav);
    const double lmin = smin<double>(l1, smin<double>(l2, l3)), lmax = smax<double>(l1, smax<double>(l2, l3));
    double aS = lmax;
    const double dUq[4] = {dU0, dpsi, __dsub_rn(__dmul_rn(rR, utR), __dmul_rn(rL, utL)), ER - EL};
    const double dFq[4] = {dpsi, __dsub_rn(__fma_rn(mR, unR, pR), __fma_rn(mL, unL, pL)),
                           __dsub_rn(__dmul_rn(mR, utR), __dmul_rn(mL, utL)), __dsub_rn(FR3, FL3)};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double dU = dUq[q], dF = dFq[q];
        const bool small = fabs(dU) < 1e-12;
        double sk = small ? lmin : fabs(squot(dF, dU, recip(small ? 1.0 : dU)));
        if (sk >= lmax) sk = lmax;
        else if (sk <= lmin) sk = lmin;
        if (sk < aS) aS = sk;
        ok = ok && fin_ok(dF) && hi_mag(dU) < kDenMax;  // (a smaller |dF| gives a speed that the fix replaces)
    }
    if (aS < 0.1) aS = (aS * aS + 0.1 * 0.1) / (2. * 0.1);
    const double dUc[4] = {dU0, dU1, dU2, dU3};
#pragma unroll
    for (int q = 0; q < 4; ++q) F[q] = __dadd_rn(fec[q], __dmul_rn(-0.5 * aS, dUc[q]));
    return ok;
}

// the same face in the operator form, as the reference writes it
__device__ __noinline__ void k_face_any(const double *U, const double *Wuvp, const double *V, int a, int b, bool xf,
                                        double gam, double edmax, double F[4])
{
    const int st = b - a;
    const double nx = xf ? 1. : 0., ny = xf ? 0. : 1.;
    double WL[4], WR[4], UL[4], UR[4], VL[4], VR[4], fec[4], aS;
    for (int q = 0; q < 4; ++q) {
        WL[q] = q ? Wuvp[(q - 1) * KPL + a] : U[a]; WR[q] = q ? Wuvp[(q - 1) * KPL + b] : U[b];
        UL[q] = U[q * KPL + a]; UR[q] = U[q * KPL + b];
        VL[q] = V[q * KPL + a]; VR[q] = V[q * KPL + b];
    }
    const double VLn[4] = {VL[0], xf ? VL[1] : VL[2], xf ? VL[2] : -VL[1], VL[3]};
    const double VRn[4] = {VR[0], xf ? VR[1] : VR[2], xf ? VR[2] : -VR[1], VR[3]};
    k_flux(WL, WR, VLn, VRn, nx, ny, gam, fec, &aS);
    const double unL = WL[1] * nx + WL[2] * ny, unR = WR[1] * nx + WR[2] * ny;
    const double aR = k_snd(0.5 * (WL[0] + WR[0]), 0.5 * (WL[3] + WR[3]), gam);
    const double lamt = smax<double>(fabs(unL), fabs(unR)) + aR;
    const double aJST = (1.0 / 32.0) * lamt;
    // entropy distance of the face                  keep_fv:249-258
    double ed = 0.;
    for (int q = 0; q < 4; ++q) ed += (UR[q] - UL[q]) * (VR[q] - VL[q]);
    const double sed = fabs(ed) / (edmax + 1e-30);
    const double phi = (1. - exp(-12.0 * sed)) > 0.05 ? 1. : 0.;
    for (int q = 0; q < 4; ++q) {
        const double jst = aJST * (U[q * KPL + b + st] - 3. * UR[q] + 3. * UL[q] - U[q * KPL + a - st]);
        const double rh = -0.5 * aS * (UR[q] - UL[q]);
        F[q] = fec[q] + (1. - phi) * jst + phi * rh;
    }
}

// where the sensor pass of a stage leaves its max; the pass of the stage before
// clears it, so no launch does that alone
__device__ __forceinline__ unsigned long long *sensor_word(Ctrl *c, int stage)
{
    return stage == 1 ? &c->aux : &c->aux23[stage - 2];
}

// store a per-cell scalar and its ghost images (no sign: it is even in the
// velocities)
__device__ __forceinline__ void put_scalar(const GridDev &gd, double *buf, int j, int i, double v)
{
    buf[gidx(gd, 0, j, i)] = v;
    const int g = gd.g, n = gd.n;
    if (i >= g && i < n - g && j >= g && j < n - g) return;
    const int nx = n_images(i, n, g, gd.bcx), ny = n_images(j, n, g, gd.bcy);
    bool f;
    for (int ka = 0; ka < ny; ++ka)
        for (int kb = (ka == 0 ? 1 : 0); kb < nx; ++kb)
            buf[gidx(gd, 0, image_of(ka, j, n, g, gd.bcy, f), image_of(kb, i, n, g, gd.bcx, f))] = v;
}

// per-cell max of the entropy distance |(U_n - U_c) . (V_n - V_c)| across
// its right and top faces, max-reduced into ctrl->aux; a tile's cells and
// their right / top neighbours are converted once each (floored conserved
// state and entropy variables in shared memory)   keep_fv_euler_2d.cu:249-277
// Each cell's entropy, its log and pow the costliest operations of the
// scheme, goes to the plane `ent`, from which the stage kernel reads it.
__global__ void __launch_bounds__(KNT) keep_ed_kernel(const __grid_constant__ GridDev gd, int stage,
                                                      const double *buf, double *ent, int ntiles)
{
    __shared__ double sU[4][EPL], sV[4][EPL];
    __shared__ double sh[KNT / 32];
    const int tid = threadIdx.x, n = gd.n;
    const double gam = gd.gam, ygm1 = recip(gam - 1.);
    double m = 0.0;
    grid_dependency();
    // the sensor word of the next stage: nothing reads it during this one
    if (blockIdx.x == 0 && tid == 0) *sensor_word(gd.ctrl, stage % 3 + 1) = 0ull;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int tx0 = (t % gd.tiles_x) * KTX, ty0 = (t / gd.tiles_x) * KTY;
        if (t + (int)gridDim.x >= ntiles) grid_release();
        for (int k = tid; k < EPL; k += KNT) {
            const int r = k / EW, c = k - r * EW, j = ty0 + r, i = tx0 + c;
            double U[4] = {1, 0, 0, 2.5};  // admissible filler beyond the ghost layer
            if (j <= n && i <= n) load_cell(buf, gd, j, i, U);
            double W[4], Uf[4], V[4];
            bool ok = k_prim_near(U, gam, W, Uf);
            if (!ok) k_prim_any(U, gam, W);
            const double sc = k_entropy(W, gam);
            ok = k_evars_near(W, sc, gam, ygm1, V) && ok;
            if (!ok) k_evars_any(W, sc, gam, V);
            for (int q = 0; q < 4; ++q) {
                sU[q][k] = Uf[q];
                sV[q][k] = V[q];
            }
            if (r < KTY && c < KTX && j < n && i < n) put_scalar(gd, ent, j, i, sc);
        }
        __syncthreads();
        for (int k = tid; k < KTX * KTY; k += KNT) {
            const int r = k / KTX, c = k - r * KTX;
            if (ty0 + r >= n || tx0 + c >= n) continue;
            const int b = r * EW + c;
            double ex = 0., ey = 0.;
            for (int q = 0; q < 4; ++q) {
                ex += (sU[q][b + 1] - sU[q][b]) * (sV[q][b + 1] - sV[q][b]);
                ey += (sU[q][b + EW] - sU[q][b]) * (sV[q][b + EW] - sV[q][b]);
            }
            m = fmax(m, fmax(fabs(ex), fabs(ey)));
        }
        __syncthreads();
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((tid & 31) == 0) sh[tid >> 5] = m;
    __syncthreads();
    if (tid == 0) {
        double b = 0.0;
        for (int w = 0; w < KNT / 32; ++w) b = fmax(b, sh[w]);
        atomicMax(sensor_word(gd.ctrl, stage), (unsigned long long)__double_as_longlong(b));
    }
}

// one SSP-RK3 stage of the KEEP scheme               keep_fv_euler_2d.cu:298-393
__global__ void __launch_bounds__(KNT, 2) keep_stage_kernel(const __grid_constant__ GridDev gd, int stage, int ntiles)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *U = reinterpret_cast<double *>(smem_raw);  // [4][KSH][KSW] conserved, rho floored
    double *W = U + 4 * KPL;                           // [3] u, v, floored p
    double *V = W + 3 * KPL;                           // [4] entropy variables (Cartesian)
    double *FX = V + 4 * KPL;                          // [4][KTY][KTX+1]
    double *FY = FX + 4 * KTY * (KTX + 1);             // [4][KTY+1][KTX]
    __shared__ double s_red[KNT / 32];
    const int tid = threadIdx.x, n = gd.n, np = n + 2 * KG;
    const double gam = gd.gam;
    const double *in = (const double *)(stage == 2 ? gd.k1 : stage == 3 ? gd.k2 : gd.st[0]);
    const double *u0 = (const double *)gd.st[0];
    double *out = (double *)(stage == 1 ? gd.k1 : stage == 2 ? gd.k2 : gd.st[0]);
    const double *ent = (const double *)gd.lo[0];  // the stage input's entropies (keep_ed_kernel)
    grid_dependency();
    const double edmax = __longlong_as_double((long long)*sensor_word(gd.ctrl, stage));
    const double inv_h = 1. / gd.h;
    // the step control, the same for every tile
    const TileCtl ctl = tile_control<P64>(gd.ctrl, stage, tid == 0 && blockIdx.x == 0);
    const KFace kf{gam, recip(gam - 1.), edmax, 12. / (edmax + 1e-30)};

    for (int t = blockIdx.x; t < ntiles && ctl.run; t += gridDim.x) {
        const int tx0 = (t % gd.tiles_x) * KTX, ty0 = (t / gd.tiles_x) * KTY;
        // conserved state of the box; primitives and entropy variables of the
        // cells next to a face (the outer ring is the JST stencil's alone)
        for (int k = tid; k < KPL; k += KNT) {
            const int r = k / KSW, c = k - r * KSW, jp = ty0 + r, ip = tx0 + c;
            const bool ring = (unsigned)(r - 1) < (unsigned)(KTY + 2) && (unsigned)(c - 1) < (unsigned)(KTX + 2);
            double Uc[4] = {1, 0, 0, 2.5}, sc = 0.;
            if (jp < np && ip < np) {
                long long e = (long long)jp * gd.pitch + ip + gd.xoff;
#pragma unroll
                for (int q = 0; q < 4; ++q) Uc[q] = in[e + q * gd.plane];
                if (ring) sc = ent[e];
            }
            U[k] = smax<double>(Uc[0], KG_MIN);
            U[KPL + k] = Uc[1];
            U[2 * KPL + k] = Uc[2];
            U[3 * KPL + k] = Uc[3];
            if (!ring) continue;
            double Wc[4], Fc[4], Vc[4];
            bool ok = k_prim_near(Uc, gam, Wc, Fc);
            if (!ok) k_prim_any(Uc, gam, Wc);
            ok = k_evars_near(Wc, sc, gam, kf.ygm1, Vc) && ok;
            if (!ok) k_evars_any(Wc, sc, gam, Vc);
            W[k] = Wc[1];
            W[KPL + k] = Wc[2];
            W[2 * KPL + k] = Wc[3];
#pragma unroll
            for (int q = 0; q < 4; ++q) V[q * KPL + k] = Vc[q];
        }
        __syncthreads();
        // faces: x then y; the face lies between cells a (left/bottom) and
        // b = a + st, with the JST stencil reaching a - st and b + st
        for (int f = tid; f < (KTX + 1) * KTY; f += KNT) {
            const int r = f / (KTX + 1), c = f - r * (KTX + 1);
            const int b = (r + KG) * KSW + (c + KG), a = b - 1;
            double F[4];
            if (!k_face_near<true>(U, W, V, a, b, kf, F)) {
                double A[4];
                k_face_any(U, W, V, a, b, true, gam, edmax, A);
#pragma unroll
                for (int q = 0; q < 4; ++q) F[q] = A[q];
            }
            double *o = FX + f;
#pragma unroll
            for (int q = 0; q < 4; ++q) o[q * KTY * (KTX + 1)] = F[q];
        }
        for (int f = tid; f < KTX * (KTY + 1); f += KNT) {
            const int r = f / KTX, c = f - r * KTX;
            const int b = (r + KG) * KSW + (c + KG), a = b - KSW;
            double F[4];
            if (!k_face_near<false>(U, W, V, a, b, kf, F)) {
                double A[4];
                k_face_any(U, W, V, a, b, false, gam, edmax, A);
#pragma unroll
                for (int q = 0; q < 4; ++q) F[q] = A[q];
            }
            double *o = FY + f;
#pragma unroll
            for (int q = 0; q < 4; ++q) o[q * (KTY + 1) * KTX] = F[q];
        }
        __syncthreads();
        if (t + (int)gridDim.x >= ntiles) grid_release();
        double lmax = 0.0;
        for (int k = tid; k < KTX * KTY; k += KNT) {
            const int r = k / KTX, c = k - r * KTX, i = tx0 + c, j = ty0 + r;
            if (i >= n || j >= n) continue;
            const long long e = (long long)(j + KG) * gd.pitch + (i + KG) + gd.xoff;
            double v[4];
            for (int q = 0; q < 4; ++q) {
                const double *fx = FX + q * KTY * (KTX + 1) + r * (KTX + 1) + c;
                const double *fy = FY + q * (KTY + 1) * KTX + r * KTX + c;
                const double L = -(fx[1] - fx[0] + fy[KTX] - fy[0]) * inv_h;
                const double ua = u0[e + q * gd.plane];  // U0
                const double ub = in[e + q * gd.plane];  // stage input (U0, U1 or U2)
                if (stage == 1) v[q] = 1. * ua + 0. * ua + 1. * ctl.dt * L;
                else if (stage == 2) v[q] = 0.75 * ua + 0.25 * ub + 0.25 * ctl.dt * L;
                else v[q] = (1. / 3.) * ua + (2. / 3.) * ub + (2. / 3.) * ctl.dt * L;
            }
            v[0] = smax<double>(v[0], KG_MIN);
            v[3] = smax<double>(v[3], KG_MIN);
            put_cell<double>(gd, out, j, i, v);
            if (stage == 3) {
                double Wn[4], Fn[4], x;
                bool ok = k_prim_near(v, gam, Wn, Fn);
                double cs = k_snd_near(Wn[0], Wn[3], gam, x);
                if (!(ok && pos_ok(x))) {
                    k_prim_any(v, gam, Wn);
                    cs = k_snd_any(Wn[0], Wn[3], gam);
                }
                lmax = smax<double>((fabs(Wn[1]) + cs) + (fabs(Wn[2]) + cs), lmax);
            }
        }
        if (stage == 3) {
            for (int o = 16; o > 0; o >>= 1) lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
            if ((tid & 31) == 0) s_red[tid >> 5] = lmax;
            __syncthreads();
            if (tid == 0) {
                double m = 0.0;
                for (int w = 0; w < KNT / 32; ++w) m = fmax(m, s_red[w]);
                atomicMax(&gd.ctrl->lam_acc, (unsigned long long)__double_as_longlong(m));
                if (t == 0) leader_finish<P64>(gd.ctrl);
            }
        }
        __syncthreads();
    }
}

// (|u| + c) + (|v| + c) of a conserved state, max into ctrl->lam_acc
__global__ void keep_lam_kernel(const GridDev gd)
{
    __shared__ double sh[32];
    const int n = gd.n;
    const long long n2 = (long long)n * n;
    double m = 0.0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n2;
         k += (long long)blockDim.x * gridDim.x) {
        double U[4], W[4], Fc[4], s;
        load_cell((const double *)gd.st[0], gd, (int)(k / n), (int)(k % n), U);
        k_cell(U, gd.gam, W, Fc, s);
        const double cs = k_snd(W[0], W[3], gd.gam);
        m = fmax(m, (fabs(W[1]) + cs) + (fabs(W[2]) + cs));
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

size_t keep_smem() { return sizeof(double) * (11 * KPL + 4 * KTY * (KTX + 1) + 4 * (KTY + 1) * KTX); }

}  // namespace

void keep_tiles(int n, int &tiles_x, int &tiles)
{
    tiles_x = (n + KTX - 1) / KTX;
    tiles = tiles_x * ((n + KTY - 1) / KTY);
}

// one KEEP stage: the entropy-distance pass, then the fused flux / RK / ghost
// kernel
cudaError_t keep_launch_stage(const GridDev &gd, int stage, int tiles, cudaStream_t s)
{
    LaunchFacts f{};
    cudaError_t e = launch_facts((const void *)keep_stage_kernel, KNT, keep_smem(), f);
    if (e != cudaSuccess) return e;
    const double *in = (const double *)(stage == 2 ? gd.k1 : stage == 3 ? gd.k2 : gd.st[0]);
    double *ent = (double *)gd.lo[0];
    const int eb = tiles < 4 * f.sms ? tiles : 4 * f.sms, cap = f.ctas_per_sm * f.sms;
    void *ea[] = {(void *)&gd, (void *)&stage, (void *)&in, (void *)&ent, (void *)&tiles};
    e = launch_chained((const void *)keep_ed_kernel, eb, KNT, 0, s, ea);
    if (e != cudaSuccess) return e;
    void *sa[] = {(void *)&gd, (void *)&stage, (void *)&tiles};
    return launch_chained((const void *)keep_stage_kernel, tiles < cap ? tiles : cap, KNT, keep_smem(), s, sa);
}

cudaError_t keep_lam_into(const GridDev &gd, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(&gd.ctrl->lam_acc, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    int blocks = (int)(((long long)gd.n * gd.n + 255) / 256);
    if (blocks > 1184) blocks = 1184;
    keep_lam_kernel<<<blocks, 256, 0, s>>>(gd);
    return cudaGetLastError();
}

}  // namespace fvb
