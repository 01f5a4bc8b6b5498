// fvb_stage.cu -- the fused SSP-RK3 stage kernel of the FP32 form as shipped,
// the choice and the launch of every form's stage kernel (FP64:
// fvb_stage64.cuh, FP32-compensated: fvb_stage32c.cu) and the TMA descriptors.
//
// One launch = one RK stage of one grid (or of every grid of a batch, through
// a tile table).  Per tile of TX x TY interior cells a CTA
//   1. stages the (TX+2g) x (TY+2g) halo tile of the stage-input state into
//      shared memory as primitives,
//   2. evaluates every face of the tile once: UP-ORDER reconstruction of the
//      four primitives on both sides, HLLC of the reconstructed states, HLLE
//      of the two cell averages, Ducros blend,
//   3. per cell: flux divergence, the SSP-RK3 combination with U0, c2p and
//      floors, stores the result into the interior and into every ghost cell
//      that mirrors it (so no separate boundary pass exists), and
//   4. in stage 3, max-reduces |u|+|v|+c of the new state into the grid's
//      step control for the next dt.
// This replaces compute_rhs + rk3_sX + apply_bc (+ reduce_max after stage 3)
// of fv_up7_ducros_2d.cu:370-612, three launches per stage and a host sync
// per step, by one launch per stage and none.
#include <stdint.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "fvb_internal.h"
#include "fvb_physics.cuh"
#include "fvb_device.cuh"
#include "fvb_tma.cuh"
#include "fvb_face32.cuh"

namespace fvb {

// Flux through one face of the working tile W ([4][SH][SW]: rho, u, v, p in
// FP64) whose right/top cell is at `base`, its sound speed at ce[0] and its
// energy for x- and y-faces at ce[CP], ce[2 CP] (the left/bottom cell's cs
// before); XDIR: x-face (normal u),
// else y-face (normal v).  Writes the 4 Cartesian components to
// out[q * ostride].
template <int SW, int PL, int CP, bool XDIR>
__device__ __forceinline__ void face_one(const double *W, int base, const float *ce, int cs, float *out, int ostride,
                                         const f32::Gas &gs)
{
    constexpr int G = 4;
    constexpr int ST = XDIR ? 1 : SW;
    constexpr int EO = XDIR ? CP : 2 * CP;
    constexpr int QN = XDIR ? 1 : 2, QT = XDIR ? 2 : 1;
    constexpr int QS[4] = {0, QN, QT, 3};
    float L[4], Rv[4], WL[4], WR[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const double *v = W + QS[m] * PL + base;
        double s[2 * G];
#pragma unroll
        for (int d = 0; d < 2 * G; ++d) s[d] = v[(d - G) * ST];
        f32::upface7(s, L[m], Rv[m]);
        WL[m] = (float)s[G - 1];
        WR[m] = (float)s[G];
    }
    // (a NaN here may stand for an infinity of the operators)
    const float z = (L[0] + Rv[0]) + (L[1] + Rv[1]) + (L[2] + Rv[2]) + (L[3] + Rv[3]);
    if (z != z) {
#pragma unroll 1
        for (int m = 0; m < 4; ++m) {
            double s[2 * G], tL, tR;
            const double *v = W + (m == 1 ? QN : m == 2 ? QT : m) * PL + base;
#pragma unroll
            for (int d = 0; d < 2 * G; ++d) s[d] = v[(d - G) * ST];
            f32::sums7(s, tL, tR);
            const float l = (float)(tL / 420.0), r = (float)(tR / 420.0);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k == m) {
                    L[k] = l;
                    Rv[k] = r;
                }
        }
    }
    L[0] = f32::fl14(L[0]); Rv[0] = f32::fl14(Rv[0]);
    L[3] = f32::fl14(L[3]); Rv[3] = f32::fl14(Rv[3]);
    float Fn[4], Fh[4], Fl[4];
    f32::hllc(L, Rv, Fh, gs);
    f32::hlle(WL, WR, ce[-cs], ce[0], ce[EO - cs], ce[EO], Fl);
    const float sd = f32::ducros(WL[3], WR[3]);
    const float one_m = 1.f - sd;
#pragma unroll
    for (int q = 0; q < 4; ++q) Fn[q] = one_m * Fh[q] + sd * Fl[q];
    out[0] = Fn[0];
    out[ostride] = Fn[QN];
    out[2 * ostride] = Fn[QT];
    out[3 * ostride] = Fn[3];
}

// shared memory of a tile shape: the box as loaded, the working tile in FP64,
// sound speed and energy of the cells -1 .. TX, -1 .. TY, the fluxes
template <int TX, int TY>
struct L32 {
    static constexpr int SW = TX + 8, SH = TY + 8, PL = SW * SH, CW = TX + 2, CP = CW * (TY + 2);
    static constexpr size_t smem = sizeof(double) * 4 * PL + sizeof(float) * (4 * PL + 3 * CP + 4 * TY * (TX + 1) +
                                                                              4 * (TY + 1) * TX);
};

// The FP32 form as shipped.  What bounds it is instruction issue: per face the
// reference's order asks for 64 FP64 operations of the reconstruction and the
// roundings back, 5 divisions and 2 roots.  The working tile is FP64, so a cell
// is converted once and not by each of its 64 stencil uses (an eighth-rate
// instruction), the divisions by 420 and by the HLLE's span come from
// reciprocals with the same bits (fvb_face32.cuh), and each cell's HLLE sound
// speed and energy are formed once: 3396 -> 2133 instructions a cell on the Sod,
// 34 -> 22 us a stage at 400^2 (351 tiles), bit-identical.
template <int TX, int TY, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) stage32_kernel(const __grid_constant__ StageArgs a)
{
    constexpr int PREC = P32;
    using R = float;
    using LS = L32<TX, TY>;
    constexpr int G = 4, SW = LS::SW, SH = LS::SH, PL = LS::PL, CW = LS::CW, CP = LS::CP;
    constexpr int NXF = (TX + 1) * TY, NYF = TX * (TY + 1);
    constexpr int NW = NT / 32;
    // IN: the tile as loaded (TMA lands here); W: the primitives the faces
    // are computed from, so IN can take the next tile meanwhile
    extern __shared__ __align__(128) unsigned char smem_raw[];
    R *IN = reinterpret_cast<R *>(smem_raw);
    double *W = reinterpret_cast<double *>(IN + 4 * PL);
    R *CE = reinterpret_cast<R *>(W + 4 * PL);  // [3][TY+2][TX+2]
    R *FX = CE + 3 * CP;              // [4][TY][TX+1]
    R *FY = FX + 4 * TY * (TX + 1);   // [4][TY+1][TX]
    __shared__ double s_red[NW];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ int s_err;

    const int tid = threadIdx.x;
    const int ntiles = a.ntiles_static;
    const int cur = a.parity;
    if (tid == 0) {
        mbar_init(&s_bar, 1);
        s_err = 0;
    }
    __syncthreads();
    grid_dependency();

    // every thread waits on the mbarrier itself (the completed phase makes the
    // TMA bytes visible to it); the barrier after the wait also agrees on s_err
    uint32_t phase = 0;
    auto wait_box = [&](bool tma) {
        if (tma) {
            if (mbar_wait(&s_bar, phase)) phase ^= 1;
            else s_err = 1;
        } else {
            cp_async_wait();
        }
        __syncthreads();
    };
    // start the halo-box load of tile t (every thread: the plain path loads
    // cooperatively)
    auto start_single = [&](int t) -> bool {
        if (tid == 0 && a.grid.tmap) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue_tile_load<PREC, G, SW, SH, NT>(a.grid, a.stage, cur, t, IN, &s_bar, tid);
        return a.grid.tmap != nullptr;
    };
    // failure injection (fvb_debug_drop_load): CTA 0 of a single-grid launch
    // issues no first box load, so its bounded wait runs out and the grid's
    // status becomes FVB_ERR_TIMEOUT; the flag is read by every thread of
    // that CTA before thread 0 clears it behind the first barrier
    const bool drop = blockIdx.x == 0 && a.stage > 0 && a.grid.ctrl && a.grid.tmap &&
                      *(volatile int *)&a.grid.ctrl->drop_load;
    const int stride = gridDim.x;
    int t = blockIdx.x;
    if (drop) {
        wait_box(true);  // nothing was issued: the wait runs out
        if (tid == 0) a.grid.ctrl->drop_load = 0;
    } else {
        wait_box(t < ntiles ? start_single(t) : false);
    }
    // the stage-3 wave-speed max is reduced once per CTA, and the step control,
    // the same for every tile, is read once (the leader is CTA 0, whose first
    // tile is tile 0)
    double lacc = 0.0;
    TileCtl ctl{};
    const R ygm1 = __frcp_rn(R(a.grid.gam) - R(1));
    if (t < ntiles) ctl = tile_control<PREC>(a.grid.ctrl, a.stage, tid == 0 && t == 0);
    for (; t < ntiles; t += stride) {
        const bool has_next = t + stride < ntiles;
        const GridDev &gd = a.grid;
        const int tile = t;
        const int n = gd.n;
        const int tx0 = (tile % gd.tiles_x) * TX, ty0 = (tile / gd.tiles_x) * TY;
        const Gas<R> gs{R(gd.gam), R(gd.gam) - R(1)};
        const f32::Gas g32{gs.gam, gs.gm1, ygm1};
        if (s_err) {
            // a halo load never arrived: record it, skip the tile
            if (tid == 0 && gd.ctrl) gd.ctrl->status = FVB_ERR_TIMEOUT;
            break;
        }
        if (ctl.run) {
            for (int k = tid; k < PL; k += NT) {
                const R w0 = IN[k], w1 = IN[PL + k], w2 = IN[2 * PL + k], w3 = IN[3 * PL + k];
                W[k] = w0;
                W[PL + k] = w1;
                W[2 * PL + k] = w2;
                W[3 * PL + k] = w3;
                const int r = k / SW - (G - 1), c = k % SW - (G - 1);
                if ((unsigned)r < (unsigned)(TY + 2) && (unsigned)c < (unsigned)CW) {
                    CE[r * CW + c] = f32::sound(w3, w0, g32);
                    const R pe = f32::over_gm1(w3, g32);
                    CE[CP + r * CW + c] = f32::energy(w0, w1, w2, pe);
                    CE[2 * CP + r * CW + c] = f32::energy(w0, w2, w1, pe);
                }
            }
        }
        __syncthreads();
        // ---- 2. load the next tile into IN (asynchronous through TMA) -------
        // (the fence orders this CTA's reads of IN before the async-proxy writes)
        const bool next_tma = has_next && start_single(t + stride);

        if (!ctl.run) {
            wait_box(next_tma);
            continue;
        }
        const R dt = R(ctl.dt);
        const R hR = R(gd.h);  // a division by h, as the shipped solver does
        // U0 of this thread's cells (stages 2 and 3), loaded now so the loads
        // are in flight while the faces are computed
        constexpr int CPT = (TX * TY + NT - 1) / NT;  // cells per thread
        static_assert(CPT <= 2, "at most two cells a thread");
        R u0v[CPT][4];
        if (a.stage >= 2) {
            const R *u0 = (const R *)gd.st[0];
#pragma unroll
            for (int it = 0; it < CPT; ++it) {
                const int k = tid + it * NT, r = k / TX, c = k - r * TX, i = tx0 + c, j = ty0 + r;
                if (k < TX * TY && i < n && j < n) {
                    const long long e = gidx(gd, 0, j, i);
#pragma unroll
                    for (int q = 0; q < 4; ++q) u0v[it][q] = u0[e + q * gd.plane];
                }
            }
        }

        // ---- 3. face fluxes: x-faces, then y-faces (compile-time strides) ---
        for (int f = tid; f < NXF; f += NT) {
            const int r = f / (TX + 1), c = f - r * (TX + 1);
            face_one<SW, PL, CP, true>(W, (r + G) * SW + (c + G), CE + (r + 1) * CW + c + 1, 1,
                                       FX + r * (TX + 1) + c, TY * (TX + 1), g32);
        }
        for (int f = tid; f < NYF; f += NT) {
            const int r = f / TX, c = f - r * TX;
            face_one<SW, PL, CP, false>(W, (r + G) * SW + (c + G), CE + (r + 1) * CW + c + 1, CW, FY + r * TX + c,
                                        (TY + 1) * TX, g32);
        }
        __syncthreads();

        if (!has_next) grid_release();
        // ---- 4. divergence, RK combination, stores ------------------------
        double lmax = 0.0;
#pragma unroll
        for (int it = 0; it < CPT; ++it) {
            const int k = tid + it * NT;
            if (k >= TX * TY) break;
            int r = k / TX, c = k - r * TX, i = tx0 + c, j = ty0 + r;
            if (i >= n || j >= n) continue;
            R res[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const R *fx = FX + q * TY * (TX + 1) + r * (TX + 1) + c;
                const R *fy = FY + q * (TY + 1) * TX + r * TX + c;
                res[q] = -(fx[1] - fx[0]) / hR - (fy[TX] - fy[0]) / hR;  // fv_up7_ducros_2d.cu:500-503
            }
            const int sc = (r + G) * SW + (c + G);
            if (a.stage == 0) {
                R *rhs = (R *)a.rhs;
                size_t n2 = (size_t)n * n, kk = (size_t)j * n + i;
                for (int q = 0; q < 4; ++q) rhs[q * n2 + kk] = res[q];
                ((R *)a.lam)[kk] = dabs<R>((R)W[PL + sc]) + dabs<R>((R)W[2 * PL + sc]) +
                                   sound<R>((R)W[3 * PL + sc], (R)W[sc], gs);
                continue;
            }
            {
                // the reference's update
                R wk[4], w0[4], c0[4], cv[4], w[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) wk[q] = (R)W[q * PL + sc];
                if (a.stage == 1) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) w0[q] = wk[q];
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) w0[q] = u0v[it][q];
                }
                p2c<R>(w0, c0, gs);
                if (a.stage == 1) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) cv[q] = c0[q] + dt * res[q];
                } else {
                    R ck[4];
                    p2c<R>(wk, ck, gs);
                    if (a.stage == 2) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            cv[q] = FVB_LIT(R, 0.75) * c0[q] + FVB_LIT(R, 0.25) * (ck[q] + dt * res[q]);
                    } else {
                        const R a3 = FVB_LIT(R, 1.) / FVB_LIT(R, 3.), b3 = FVB_LIT(R, 2.) / FVB_LIT(R, 3.);
#pragma unroll
                        for (int q = 0; q < 4; ++q) cv[q] = a3 * c0[q] + b3 * (ck[q] + dt * res[q]);
                    }
                }
                c2p<R>(cv, w, gs);
                w[0] = floor14(w[0]);
                w[3] = floor14(w[3]);
                R *out = (R *)(a.stage == 1 ? gd.k1 : a.stage == 2 ? gd.k2 : gd.st[0]);
                put_cell<R>(gd, out, j, i, w);
                if (a.stage == 3) {
                    const R lam = dabs<R>(w[1]) + dabs<R>(w[2]) + sound<R>(w[3], w[0], gs);
                    // (a NaN lam is skipped, as fmax skips it; one compare-select)
                    lmax = smax<double>((double)lam, lmax);
                }
            }
        }

        // ---- 5. max wave speed of the new state (stage 3) ------------------
        if (a.stage == 3) {
            if (tid == 0 && tile == 0) leader_finish<PREC>(gd.ctrl);
            lacc = fmax(lacc, lmax);
        }
        // ---- 6. next tile's halo box: wait, then release W / FX / FY -------
        wait_box(next_tma);
    }
    if (a.stage == 3) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lacc = fmax(lacc, __shfl_xor_sync(0xffffffffu, lacc, o));
        if ((tid & 31) == 0) s_red[tid >> 5] = lacc;
        __syncthreads();
        if (tid == 0 && a.grid.ctrl) {
            double m = 0.0;
            for (int w = 0; w < NW; ++w) m = fmax(m, s_red[w]);
            if (m > 0.0) atomicMax(&a.grid.ctrl->lam_acc, (unsigned long long)__double_as_longlong(m));
        }
    }
    // a load still in flight after an error: wait for it (bounded) so no
    // copy into this CTA's shared memory outlives it
    if (s_err && gd_has_tma(a)) mbar_wait(&s_bar, phase);
}

// ---------------------------------------------------------------------------
// instantiation table
// ---------------------------------------------------------------------------
template <int SHAPE>
static StageKernel entry32()
{
    constexpr TileShape ts = kTileShapes[SHAPE];
    // three CTAs an SM, the registers' budget (80 at 256 threads)
    return StageKernel{(void *)stage32_kernel<ts.tx, ts.ty, ts.nt, 3>, nullptr, L32<ts.tx, ts.ty>::smem, ts.nt};
}

// the kernel of a form, an order, a tile variant and a solver on the
// reconstructed states; fn null: not built
static StageKernel kernel_for(int prec, int order, int shape, int rs = 0)
{
    if (shape < 0 || shape >= kNumTileShapes) return StageKernel{};
    if (prec == P64) return stage64_kernel_of(order, shape, rs);
    if (order != 7 || rs != 0) return StageKernel{};
    if (prec == P32C) return stage32c_kernel_of(shape);
    switch (shape) {
    case 0: return entry32<0>();
    case 1: return entry32<1>();
    case 2: return entry32<2>();
    case 3: return entry32<3>();
    case 4: return entry32<4>();
    case 5: return entry32<5>();
    default: return entry32<6>();
    }
}

cudaError_t launch_chained(const void *fn, int ctas, int threads, size_t smem, cudaStream_t s, void **args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

cudaError_t launch_facts(const void *fn, int threads, size_t smem, LaunchFacts &out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    static std::mutex mu;
    static std::map<std::tuple<const void *, int, int, size_t>, LaunchFacts> known;
    const auto key = std::make_tuple(fn, dev, threads, smem);
    std::lock_guard<std::mutex> lk(mu);
    const auto it = known.find(key);
    if (it != known.end()) {
        out = it->second;
        return cudaSuccess;
    }
    LaunchFacts f{};
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f.ctas_per_sm, fn, threads, smem);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&f.sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (f.ctas_per_sm <= 0) return cudaErrorInvalidConfiguration;
    known.emplace(key, f);
    out = f;
    return cudaSuccess;
}

// resident CTAs per SM of a kernel: the fewest of its forms
static cudaError_t prepare(const StageKernel &e, int &max_ctas)
{
    LaunchFacts a{}, b{};
    cudaError_t err = launch_facts(e.fn, e.nt, e.smem, a);
    if (err == cudaSuccess && e.fn_queued) {
        err = launch_facts(e.fn_queued, e.nt, e.smem, b);
        a.ctas_per_sm = std::min(a.ctas_per_sm, b.ctas_per_sm);
    }
    if (err == cudaSuccess) err = e.fn_batched ? launch_facts(e.fn_batched, e.nt, e.smem, b) : cudaSuccess;
    if (err != cudaSuccess) return err;
    max_ctas = e.fn_batched ? std::min(a.ctas_per_sm, b.ctas_per_sm) : a.ctas_per_sm;
    return cudaSuccess;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    // looked up once (a function-local static's initialisation is thread-safe)
    static const EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return (EncodeTiledFn)p;
        return (EncodeTiledFn) nullptr;
    }();
    return fn;
}

// Descriptors of the (tx+2g) x (ty+2g) x 4 halo box of each padded buffer and
// of the tx x ty tile of U0 (out[TM_U0]).  The tensor is (x = memory column,
// y = padded row, z = variable plane); x starts at column 0 of the pitched
// row, so a tile's box starts at x = xoff + tx0, or with xo = 1 (where that x
// is odd, FP64) one column earlier and is two columns wider.  Every such x,
// the pitch and the plane stride must be 16-byte multiples; out-of-range
// parts of ragged tiles are zero-filled.
static bool encode_maps(const GridDev &gd, size_t es, int g, int tx, int ty, int xo, CUtensorMap out[TM_COUNT])
{
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    const int np = gd.n + 2 * g, sw = tx + 2 * g + 2 * xo, sh = ty + 2 * g;
    if (((size_t)gd.pitch * es) % 16 || ((size_t)gd.plane * es) % 16 || gd.xoff < xo ||
        ((size_t)(gd.xoff - xo) * es) % 16 || ((size_t)tx * es) % 16 || ((size_t)sw * es) % 16 || sw > 256 || sh > 256)
        return false;
    if (es == 8 && ((size_t)(gd.xoff + g) * es) % 16) return false;
    cuuint64_t dims[3] = {(cuuint64_t)(gd.xoff + np), (cuuint64_t)np, 4};
    cuuint64_t strides[2] = {(cuuint64_t)gd.pitch * es, (cuuint64_t)gd.plane * es};
    cuuint32_t box[3] = {(cuuint32_t)sw, (cuuint32_t)sh, 4};
    cuuint32_t tile[3] = {(cuuint32_t)tx, (cuuint32_t)ty, 4};
    cuuint32_t estr[3] = {1, 1, 1};
    void *bufs[TM_COUNT] = {gd.st[0], gd.st[1] ? gd.st[1] : gd.st[0], gd.k1, gd.k2, gd.st[0]};
    for (int m = 0; m < TM_COUNT; ++m) {
        if (((uintptr_t)bufs[m]) % 16) return false;
        CUresult r = enc(&out[m], es == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                         bufs[m], dims, strides, m == TM_U0 ? tile : box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return false;
    }
    return true;
}

bool encode_tile_maps(const GridDev &gd, int prec, int order, int shape, CUtensorMap out[TM_COUNT])
{
    if (shape < 0 || shape >= kNumTileShapes) return false;
    const TileShape &ts = tile_shape(prec, shape);
    const int g = (order + 1) / 2;
    return encode_maps(gd, prec == P64 ? 8 : 4, g, ts.tx, ts.ty, prec == P64 ? (16 - g) & 1 : 0, out);
}

bool encode_family_maps(const GridDev &gd, int tx, int ty, CUtensorMap out[TM_COUNT])
{
    return encode_maps(gd, 8, gd.g, tx, ty, (16 - gd.g) & 1, out);
}

// Copy a grid's tensor maps into device memory from a kernel parameter, so
// the host copy need not outlive the call (no stream synchronisation).
struct TileMaps {
    CUtensorMap m[TM_COUNT];
};

__global__ void put_maps_kernel(const __grid_constant__ TileMaps maps, CUtensorMap *dst)
{
    constexpr int NV = (int)(sizeof(TileMaps) / 16);
    const int k = threadIdx.x;
    if (k < NV) reinterpret_cast<uint4 *>(dst)[k] = reinterpret_cast<const uint4 *>(&maps)[k];
}

cudaError_t put_tile_maps(const CUtensorMap maps[TM_COUNT], CUtensorMap *dst, cudaStream_t s)
{
    static_assert(sizeof(TileMaps) % 16 == 0 && sizeof(TileMaps) / 16 <= 64, "one small block copies the maps");
    TileMaps tm;
    for (int m = 0; m < TM_COUNT; ++m) tm.m[m] = maps[m];
    put_maps_kernel<<<1, 64, 0, s>>>(tm, dst);
    return cudaGetLastError();
}

int stage_max_ctas_per_sm(int prec, int order, int shape, int rs)
{
    const StageKernel e = kernel_for(prec, order, shape, rs);
    int max_ctas = 0;
    if (!e.fn || prepare(e, max_ctas) != cudaSuccess) return 0;
    return max_ctas;
}

cudaError_t launch_stage(int prec, int order, int shape, const StageArgs &a, int grid_ctas, cudaStream_t s, int rs)
{
    const StageKernel e = kernel_for(prec, order, shape, rs);
    // a queue of tiles from two whole waves up: below, the later box costs more
    // than the balance gives (FP64, us a stage, fixed / queued: 400^2 12.9 / 13.8,
    // 512^2 17.3 / 18.0; 560^2 19.8 / 18.3, 700^2 26.8 / 23.9)
    const bool queued = e.fn_queued && !a.grids && a.grid.tmap && a.stage > 0 && a.ntiles_static > 2 * grid_ctas;
    void *fn = a.grids ? e.fn_batched : queued ? e.fn_queued : e.fn;
    if (!fn) return cudaErrorInvalidValue;
    LaunchFacts f{};
    const cudaError_t err = launch_facts(fn, e.nt, e.smem, f);
    if (err != cudaSuccess) return err;
    if (grid_ctas <= 0) return cudaSuccess;
    void *args[] = {(void *)&a};
    return launch_chained(fn, grid_ctas, e.nt, e.smem, s, args);
}

}  // namespace fvb
