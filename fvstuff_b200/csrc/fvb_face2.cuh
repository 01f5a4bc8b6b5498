// fvb_face2.cuh -- the FP32 face flux of the compensated form, evaluated for
// two faces at once in the packed FP32 pairs of sm_100 (FFMA2 / FADD2 /
// FMUL2: one instruction issues the same operation on both halves of a
// 64-bit register pair).  Lane x and lane y are two independent faces; every
// operation below acts on both, so the arithmetic of two faces issues as one
// instruction stream.  Per-lane work (reciprocals, square roots, compares,
// selects, min / max) stays scalar.
//
// The scheme is the reference's UP7 + Ducros-blended HLLC / HLLE face flux
// (fv_up7_ducros_2d.cu:149-186, :237-328, :433), normal frame, written for
// FP32 throughput:
//   * UP7 weights pre-divided by 420;
//   * HLLC in star variables: one side K is selected (the upwind side of the
//     contact, or of the whole fan when it is supersonic); with S the contact
//     speed (u_K in a supersonic fan), d_K = r_K (S_K - u_K) and
//     q = 1 / (S_K - S): rho* = d_K q, p* = p_K + d_K (S - u_K),
//     E* = q (E_K (S_K - u_K) + (S - u_K)(d_K S + p_K)), and the flux is
//     (rho* S, rho* S^2 + p*, rho* S t_K, (E* + p*) S); c = gp rsqrt(gp rho);
//   * HLLE (Einfeldt's form, SL- = min(SL, 0), SR+ = max(SR, 0)): with
//     a = SR+ / (SR+ - SL-), b = -SL- / (SR+ - SL-), kL = a (uL - SL-) and
//     kR = b (uR - SR+) the average is rho_L kL + rho_R kR, and so on per
//     component; the sensor's weight s is folded into a and b, so the blend is
//     one multiply-add a component;
//   * 99 packed operations two faces (56 the reconstruction), against 118.
// Each rewriting is exact in real arithmetic; in FP32 the results differ from
// the reference's association order by a few ulp, which the compensated
// form's tolerance against the FP64 oracle (1e-6 relative L1) absorbs.
#pragma once
#include <cuda_runtime.h>

#include "fvb_physics.cuh"

namespace fvb {
namespace f2 {

typedef float2 V;

__device__ __forceinline__ V splat(float a) { return make_float2(a, a); }
__device__ __forceinline__ V add(V a, V b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ V mul(V a, V b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ V fma(V a, V b, V c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ V sub(V a, V b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ V vmin(V a, V b) { return make_float2(fminf(a.x, b.x), fminf(a.y, b.y)); }
__device__ __forceinline__ V vmax(V a, V b) { return make_float2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }
__device__ __forceinline__ V rcp(V a) { return make_float2(__fdividef(1.0f, a.x), __fdividef(1.0f, a.y)); }
__device__ __forceinline__ V vrsqrt(V a) { return make_float2(rsqrtf(a.x), rsqrtf(a.y)); }
// sqrt of x >= 1e-14 as x * rsqrt(x)
__device__ __forceinline__ V vsqrt(V a) { return mul(a, vrsqrt(a)); }

// error-free sum of double-floats (hi, lo) and float increments d, as df_add
// (fvb_device.cuh)
__device__ __forceinline__ void df_add(V &hi, V &lo, V d)
{
    const V s = add(hi, d);
    const V bb = sub(s, hi);
    const V err = add(sub(hi, sub(s, bb)), sub(d, bb));
    const V l = add(lo, err);
    const V h2 = add(s, l);
    lo = sub(l, sub(h2, s));
    hi = h2;
}

struct B {
    bool x, y;
};
__device__ __forceinline__ V sel(B c, V a, V b) { return make_float2(c.x ? a.x : b.x, c.y ? a.y : b.y); }

// UP7 face values of a pair of 8-point stencils (face between s[3] and s[4])
__device__ __forceinline__ void upface7(const V s[8], V &vL, V &vR)
{
#define FVB_W7(a) splat((float)((a) / 420.0))
    vL = mul(FVB_W7(-3.), s[0]);
    vL = fma(FVB_W7(25.), s[1], vL);
    vL = fma(FVB_W7(-101.), s[2], vL);
    vL = fma(FVB_W7(319.), s[3], vL);
    vL = fma(FVB_W7(214.), s[4], vL);
    vL = fma(FVB_W7(-38.), s[5], vL);
    vL = fma(FVB_W7(4.), s[6], vL);
    vR = mul(FVB_W7(4.), s[1]);
    vR = fma(FVB_W7(-38.), s[2], vR);
    vR = fma(FVB_W7(214.), s[3], vR);
    vR = fma(FVB_W7(319.), s[4], vR);
    vR = fma(FVB_W7(-101.), s[5], vR);
    vR = fma(FVB_W7(25.), s[6], vR);
    vR = fma(FVB_W7(-3.), s[7], vR);
#undef FVB_W7
}

// the floor 1e-14 on the reconstructed rho and p
__device__ __forceinline__ void floors(V L[4], V R[4])
{
    const V tiny = splat(1e-14f);
    L[0] = vmax(L[0], tiny);
    R[0] = vmax(R[0], tiny);
    L[3] = vmax(L[3], tiny);
    R[3] = vmax(R[3], tiny);
}

// Blended flux of two faces, normal frame.  L, Rv: floored reconstructions
// (rho, un, ut, p); WL, WR: the cell states either side with their sound
// speeds cWL, cWR and energies EWL, EWR.
__device__ __forceinline__ void face_flux(const V L[4], const V Rv[4], const V WL[4], const V WR[4], V cWL,
                                          V cWR, V EWL, V EWR, float gam, float igm1, V F[4])
{
    const V zero = splat(0.0f), one = splat(1.0f), half = splat(0.5f), G = splat(gam), IG = splat(igm1);
    const V cmin = splat(1e-7f);
    // --- HLLC of the reconstructed states, in star variables ---
    V Fh0, Fh1, Fh2, Fh3;
    {
        const V rL = L[0], uL = L[1], tL = L[2], pL = L[3];
        const V rR = Rv[0], uR = Rv[1], tR = Rv[2], pR = Rv[3];
        const V gL = mul(G, pL), gR = mul(G, pR);
        const V cL = vmax(mul(gL, vrsqrt(mul(gL, rL))), cmin), cR = vmax(mul(gR, vrsqrt(mul(gR, rR))), cmin);
        const V SL = vmin(sub(uL, cL), sub(uR, cR)), SR = vmax(add(uL, cL), add(uR, cR));
        const V dL = mul(rL, sub(SL, uL)), eR = mul(rR, sub(uR, SR));  // eR = -dR
        const V Ss = mul(fma(eR, uR, fma(dL, uL, sub(pR, pL))), rcp(add(dL, eR)));
        // side K: by the contact when subsonic, by the fan when supersonic
        const B supL{SL.x >= 0.0f, SL.y >= 0.0f};
        const B sup{supL.x || SR.x <= 0.0f, supL.y || SR.y <= 0.0f};
        const B left{sup.x ? supL.x : Ss.x >= 0.0f, sup.y ? supL.y : Ss.y >= 0.0f};
        const V rK = sel(left, rL, rR), uK = sel(left, uL, uR), tK = sel(left, tL, tR);
        const V pK = sel(left, pL, pR), SK = sel(left, SL, SR);
        const V EK = fma(mul(half, rK), fma(uK, uK, mul(tK, tK)), mul(pK, IG));
        // a supersonic fan: S = uK, and SK - uK and SK - S taken as 1, which
        // gives K's own state exactly (they could be 0 beside a floored c)
        const V S = sel(sup, uK, Ss), w = sel(sup, one, sub(SK, uK));
        const V q = rcp(sel(sup, one, sub(SK, Ss)));
        const V dK = mul(rK, w), du = sub(S, uK);
        const V ps = fma(dK, du, pK);
        const V Es = mul(fma(du, fma(dK, S, pK), mul(EK, w)), q);
        Fh0 = mul(mul(dK, q), S);
        Fh1 = fma(Fh0, S, ps);
        Fh2 = mul(Fh0, tK);
        Fh3 = mul(add(Es, ps), S);
    }
    // --- HLLE of the cell states (Einfeldt form) with the sensor's weight ---
    const V rL = WL[0], uL = WL[1], tL = WL[2], pL = WL[3];
    const V rR = WR[0], uR = WR[1], tR = WR[2], pR = WR[3];
    const V SLm = vmin(vmin(sub(uL, cWL), sub(uR, cWR)), zero);
    const V SRp = vmax(vmax(add(uL, cWL), add(uR, cWR)), zero);
    const V dp = sub(pR, pL), psum = add(pR, pL), dp2 = mul(dp, dp);
    const V sd = mul(dp2, rcp(fma(mul(splat(0.1f), psum), psum, dp2)));
    // (SR+ - SL- >= 2e-7, the cells' sound speeds being at least 1e-7)
    const V w = mul(sd, rcp(sub(SRp, SLm))), om = sub(one, sd);
    const V a = mul(SRp, w), b = mul(SLm, mul(w, splat(-1.0f)));
    const V kL = mul(a, sub(uL, SLm)), kR = mul(b, sub(uR, SRp));
    const V gL = mul(rL, kL), gR = mul(rR, kR);
    const V aP = mul(a, pL), bP = mul(b, pR);
    F[0] = fma(om, Fh0, add(gL, gR));
    F[1] = fma(om, Fh1, fma(uL, gL, fma(uR, gR, add(aP, bP))));
    F[2] = fma(om, Fh2, fma(tL, gL, mul(tR, gR)));
    F[3] = fma(om, Fh3, fma(EWL, kL, fma(EWR, kR, fma(aP, uL, mul(bP, uR)))));
}

}  // namespace f2
}  // namespace fvb
