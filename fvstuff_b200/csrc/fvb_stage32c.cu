// fvb_stage32c.cu -- the SSP-RK3 stage kernel of the FP32-compensated form.
//
// Same tile pipeline as the FP64 kernel (fvb_stage64.cuh): persistent CTAs walk
// the tiles of one grid or of a batch's tile table; the halo box of the next
// tile streams in through TMA while the current one is computed; every face
// is evaluated once; the RK combination stores the interior and its ghost
// images; stage 3 max-reduces the wave speed into the step control.
//
// What differs, for FP32 throughput: two faces, or two cells, share the lanes
// of packed FP32 registers (fvb_face2.cuh), so that their arithmetic issues as
// one instruction.  Two forms:
//   * stage32c_kernel pairs x-face p with y-face p, one pair a thread; three
//     CTAs of 256 threads share an SM (71 KB, 80 registers).  It serves small
//     grids and batches.
//   * stage32p_kernel pairs rows half a tile apart and gives a thread four
//     faces of each direction; two CTAs of 256 threads (112 KB, 128
//     registers).  It serves large grids.
// Both give the same bits.  What bounds them is instruction issue and, at 16
// to 24 warps an SM, the latency of dependent instructions, not memory (a
// 2048^2 stage is 34 us at the copy bandwidth).
//
// State: conserved (rho, rho u, rho v, E) as an FP32 hi/lo pair per value;
// the stages form increments d1 = dt L(U0), d2 = (d1 + dt L(U1)) / 4 and add
// U = U0 + 2/3 (d2 + dt L(U2)) to the pair with an error-free sum, so the
// state keeps ~48 bits while all flux arithmetic is FP32.  Ping-pong state
// buffers (parity) keep U0 readable while U is written.
#include <stdint.h>

#include "fvb_internal.h"
#include "fvb_physics.cuh"
#include "fvb_device.cuh"
#include "fvb_tma.cuh"
#include "fvb_face2.cuh"

namespace fvb {

// resident CTAs per SM the kernel is compiled for: 768 threads (24 warps)
// per SM, <= 85 registers a thread
template <int NT> struct MinBlocks32c { static constexpr int v = 768 / NT; };

// The operands of one cell's RK update beside dt L: the stage increment (d1
// in stage 2, d2 in stage 3) and, in stage 3, the hi / lo pair of U0.
struct Operands32c {
    float d[4], h[4], l[4];
};
__device__ __forceinline__ void load_operands32c(const GridDev &gd, int stage, int cur, int j, int i, Operands32c &o)
{
    if (stage == 1) return;
    const unsigned e = cell_index(gd, j, i);
    const float *d = (const float *)(stage == 2 ? gd.k1 : gd.k2);
#pragma unroll
    for (int q = 0; q < 4; ++q) o.d[q] = (d + q * gd.plane)[e];
    if (stage == 3) {
        const float *h = (const float *)gd.st[cur], *l = (const float *)gd.lo[cur];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            o.h[q] = (h + q * gd.plane)[e];
            o.l[q] = (l + q * gd.plane)[e];
        }
    }
}

// The floors on a new state that is at one of them (rho, p >= 1e-14); returns
// its wave speed.
__device__ __noinline__ float floor_cell32c_(float vh0, float vh1, float vh2, float vh3, float gam, float gm1,
                                             float *rho, float *E)
{
    float w[4];
    const float ir = frcp(vh0);
    w[0] = vh0; w[1] = vh1 * ir; w[2] = vh2 * ir;
    w[3] = gm1 * (vh3 - 0.5f * (vh1 * vh1 + vh2 * vh2) * ir);
    *rho = vh0;
    *E = vh3;
    if (!(w[0] > 1e-14f)) { *rho = 1e-14f; w[0] = 1e-14f; }
    if (!(w[3] > 1e-14f)) {
        const float ke = 0.5f * (vh1 * vh1 + vh2 * vh2) / *rho;
        *E = 1e-14f / gm1 + ke;
        w[3] = 1e-14f;
    }
    const float cs2 = gam * w[3] * frcp(w[0]);
    return fabsf(w[1]) + fabsf(w[2]) + fsqrt(cs2 > 1e-14f ? cs2 : 1e-14f);
}
__device__ __forceinline__ float floor_cell32c(float vh[4], float vl[4], float gam, float gm1)
{
    float rho, E;
    const float lam = floor_cell32c_(vh[0], vh[1], vh[2], vh[3], gam, gm1, &rho, &E);
    if (rho != vh[0]) vl[0] = 0.f;
    if (E != vh[3]) vl[3] = 0.f;
    vh[0] = rho;
    vh[3] = E;
    return lam;
}

// The RK update of one cell from dres = dt L(U) (stage 1: d1 = dres; stage
// 2: d2 = (d1 + dres) / 4; stage 3: U0 + 2/3 (d2 + dres) added to the hi /
// lo pair with an error-free sum, floors, stores with ghost images, and the
// cell's wave speed into lmax).
__device__ __forceinline__ void update_cell32c(const GridDev &gd, int stage, int nxt, int j, int i,
                                               const float dres[4], const Operands32c &o, float gam, float gm1,
                                               float &lmax)
{
    if (stage == 1) {
        put_cell<float>(gd, (float *)gd.k1, j, i, dres);
    } else if (stage == 2) {
        float d[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) d[q] = 0.25f * (o.d[q] + dres[q]);
        put_cell<float>(gd, (float *)gd.k2, j, i, d);
    } else {
        float vh[4], vl[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            vh[q] = o.h[q];
            vl[q] = o.l[q];
            df_add(vh[q], vl[q], (2.0f / 3.0f) * (o.d[q] + dres[q]));
        }
        // primitives and wave speed of the new state, floors rho, p >= 1e-14
        const float ir = frcp(vh[0]);
        const float u = vh[1] * ir, v = vh[2] * ir;
        const float ke = __fmul_rn(__fmul_rn(0.5f, __fmaf_rn(vh[1], vh[1], __fmul_rn(vh[2], vh[2]))), ir);
        const float pr = gm1 * __fsub_rn(vh[3], ke);
        const float cs2 = gam * pr * ir;
        const float x = fmaxf(cs2, 1e-14f);
        float lam = fabsf(u) + fabsf(v) + __fmul_rn(x, rsqrtf(x));  // (not fused: as update_pair32c)
        if (!(vh[0] > 1e-14f && pr > 1e-14f)) lam = floor_cell32c(vh, vl, gam, gm1);
        put_cell2<float>(gd, (float *)gd.st[nxt], (float *)gd.lo[nxt], j, i, vh, vl);
        lmax = fmaxf(lmax, lam);  // (NaN skipped; exact in FP64 below)
    }
}

// The same update for two cells in the lanes of packed registers (cells
// (j0, i) and (j1, i); in0 / in1: inside the grid): the arithmetic of
// update_cell32c, one packed operation for both.
__device__ __forceinline__ void update_pair32c(const GridDev &gd, int stage, int nxt, int j0, int j1, int i, bool in0,
                                               bool in1, const f2::V dr[4], const Operands32c &o0,
                                               const Operands32c &o1, float gam, float gm1, float &lmax)
{
    f2::V d[4];
    if (stage == 1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) d[q] = dr[q];
    } else {
        const f2::V c = f2::splat(stage == 2 ? 0.25f : 2.0f / 3.0f);
#pragma unroll
        for (int q = 0; q < 4; ++q) d[q] = f2::mul(c, f2::add(make_float2(o0.d[q], o1.d[q]), dr[q]));
    }
    if (stage <= 2) {
        float *out = (float *)(stage == 1 ? gd.k1 : gd.k2);
        const float a[4] = {d[0].x, d[1].x, d[2].x, d[3].x}, b[4] = {d[0].y, d[1].y, d[2].y, d[3].y};
        if (in0) put_cell<float>(gd, out, j0, i, a);
        if (in1) put_cell<float>(gd, out, j1, i, b);
        return;
    }
    f2::V h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        h[q] = make_float2(o0.h[q], o1.h[q]);
        l[q] = make_float2(o0.l[q], o1.l[q]);
        f2::df_add(h[q], l[q], d[q]);
    }
    // primitives and wave speed of the new state, floors rho, p >= 1e-14
    const f2::V ir = f2::rcp(h[0]);
    const f2::V u = f2::mul(h[1], ir), v = f2::mul(h[2], ir);
    const f2::V ke = f2::mul(f2::mul(f2::splat(0.5f), f2::fma(h[1], h[1], f2::mul(h[2], h[2]))), ir);
    const f2::V pr = f2::mul(f2::splat(gm1), f2::sub(h[3], ke));
    const f2::V cs2 = f2::mul(f2::mul(f2::splat(gam), pr), ir);
    const f2::V cs = f2::vsqrt(f2::vmax(cs2, f2::splat(1e-14f)));
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        if (!(m ? in1 : in0)) continue;
        float vh[4], vl[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            vh[q] = m ? h[q].y : h[q].x;
            vl[q] = m ? l[q].y : l[q].x;
        }
        float lam = fabsf(m ? u.y : u.x) + fabsf(m ? v.y : v.x) + (m ? cs.y : cs.x);
        if (!(vh[0] > 1e-14f && (m ? pr.y : pr.x) > 1e-14f)) lam = floor_cell32c(vh, vl, gam, gm1);
        put_cell2<float>(gd, (float *)gd.st[nxt], (float *)gd.lo[nxt], m ? j1 : j0, i, vh, vl);
        lmax = fmaxf(lmax, lam);
    }
}

template <int TX, int TY, int NT, bool BATCHED>
__global__ void __launch_bounds__(NT, MinBlocks32c<NT>::v) stage32c_kernel(const __grid_constant__ StageArgs a)
{
    constexpr int G = 4;
    constexpr int SW = TX + 2 * G, SH = TY + 2 * G, PL = SW * SH;
    constexpr int NXF = (TX + 1) * TY, NYF = TX * (TY + 1);
    constexpr int NP = NXF > NYF ? NXF : NYF;
    constexpr int NC = TX * TY;
    constexpr int NW = NT / 32;

    // IN: the halo box as loaded (hi + increment planes); W: rho, u, v, p,
    // c, E the faces read; FX / FY: face fluxes
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float *IN = reinterpret_cast<float *>(smem_raw);
    float *W = IN + 8 * PL;
    float *FX = W + 6 * PL;               // [4][TY][TX+1]
    float *FY = FX + 4 * TY * (TX + 1);   // [4][TY+1][TX]
    __shared__ double s_red[NW];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ int s_err;
    __shared__ __align__(16) TileHdr s_hdr[2];
    __shared__ TileRef s_ref_next;  // batched: table entry of the CTA's next tile

    const int tid = threadIdx.x;
    constexpr bool batched = BATCHED;
    const int cur = a.parity, nxt = a.parity ^ 1;
    if (tid == 0) {
        mbar_init(&s_bar, 1);
        s_err = 0;
    }
    __syncthreads();
    const int ntiles = batched ? *a.ntiles : a.ntiles_static;
    BatchHead head{};
    if (batched && tid < 32) head = batch_head(a, &s_hdr[0], ntiles, tid);
    grid_dependency();

    // every thread waits on the mbarrier itself (the completed phase makes the
    // TMA bytes visible to it); the barrier after the wait also agrees on s_err
    uint32_t phase = 0;
    auto wait_box = [&](bool tma) {
        if (tma) {
            if (mbar_wait(&s_bar, phase)) phase ^= 1;
            else s_err = 1;
        }
        __syncthreads();
    };
    // The wait at the end of a tile needs no block barrier when the box came
    // through TMA: the next writes of every buffer are already ordered by
    // the barriers inside the tile (W by the conversion barrier, FX / FY by
    // the face barrier the update follows, IN by the conversion barrier the
    // next load is issued behind; the update reads neither W nor IN), and
    // each thread's own wait makes the box visible to it.  A box loaded by
    // the threads themselves needs the barrier.  A timeout is agreed on at
    // the next conversion barrier.
    auto wait_box_own = [&](bool tma) {
        if (tma) {
            if (mbar_wait(&s_bar, phase)) phase ^= 1;
            else s_err = 1;
        } else {
            __syncthreads();
        }
    };
    // single grid: start the halo-box load of tile t (every thread: the
    // plain path loads cooperatively)
    auto start_single = [&](int t) -> bool {
        if (tid == 0 && a.grid.tmap) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue_tile_load<P32C, G, SW, SH, NT>(a.grid, a.stage, cur, t, IN, &s_bar, tid);
        return a.grid.tmap != nullptr;
    };
    // failure injection (fvb_debug_drop_load): CTA 0 of a single-grid launch
    // issues no first box load, so its bounded wait runs out and the grid's
    // status becomes FVB_ERR_TIMEOUT; the flag is read by every thread of
    // that CTA before thread 0 clears it behind the first barrier
    const bool drop = !batched && blockIdx.x == 0 && a.stage > 0 && a.grid.ctrl && a.grid.tmap &&
                      *(volatile int *)&a.grid.ctrl->drop_load;
    const int stride = gridDim.x;
    int t = blockIdx.x, slot = 0;
    if (t < ntiles && batched) {
        if (tid < 32) {
            const TileRef r0 = head.first;
            start_first_tile<P32C>(a, &s_hdr[0], r0, &s_bar, tid, [&](const TileHdr &h) {
                issue_tile_load<P32C, G, SW, SH, NT>(h.gd, a.stage, cur, r0.tile, IN, &s_bar, 0);
            });
            if (tid == 0) s_ref_next = head.next;
        }
        wait_box(true);
    } else if (drop) {
        wait_box(true);  // nothing was issued: the wait runs out
        if (tid == 0) a.grid.ctrl->drop_load = 0;
    } else {
        wait_box(t < ntiles ? start_single(t) : false);
    }
    double lacc = 0.0;
    // which of this thread's conversion cells (k = tid + it NT) the HLLE
    // reads the sound speed and energy of: the interior rows x columns
    // [G-1, G+TX], and rows G-1, G+TY x the interior columns
    constexpr int NCV = (PL + NT - 1) / NT;
    static_assert(NCV <= 32, "one mask bit per conversion cell");
    unsigned cemask = 0;
#pragma unroll
    for (int it = 0; it < NCV; ++it) {
        const int k = tid + it * NT, r = k / SW, c = k - r * SW;
        const bool ce = ((unsigned)(r - G) < (unsigned)TY && (unsigned)(c - (G - 1)) < (unsigned)(TX + 2)) ||
                        ((r == G - 1 || r == G + TY) && (unsigned)(c - G) < (unsigned)TX);
        cemask |= (ce && k < PL ? 1u : 0u) << it;
    }
    // one grid: the step control is the same for every tile of the launch,
    // read once (the leader is CTA 0, whose first tile is tile 0)
    TileCtl ctl1{};
    if (!batched && t < ntiles) ctl1 = tile_control<P32C>(a.grid.ctrl, a.stage, tid == 0 && t == 0);
    for (; t < ntiles; t += stride, slot ^= 1) {
        // warp 0 of a batched launch: the next tile's descriptor word and the
        // entry of the tile after it, in flight during the conversion
        const bool has_next = t + stride < ntiles;
        unsigned long long wnext = 0ull;
        TileRef ref_next{}, ref_after{};
        if (batched && tid < 32) {
            if (has_next) {
                ref_next = s_ref_next;
                wnext = hdr_word(a, ref_next, tid);
            }
            if (t + 2 * stride < ntiles) ref_after = a.tiles[t + 2 * stride];
        }
        const GridDev &gd = tile_grid<BATCHED>(s_hdr[slot], a);
        const int tile = batched ? s_hdr[slot].tile : t;
        const TileCtl ctl = batched ? s_hdr[slot].ctl : ctl1;
        const int n = gd.n;
        const int tx0 = (tile % gd.tiles_x) * TX, ty0 = (tile / gd.tiles_x) * TY;
        const float gam = (float)gd.gam, gm1 = (float)gd.gam - 1.0f, igm1 = (float)gd.igm1;
        // ---- 1. stage input U0 + d into W as primitives (+ c, E where the
        //         HLLE reads them, cemask) ------------------------------------
        if (ctl.run) {
#pragma unroll
            for (int it = 0; it < NCV; ++it) {
                const int k = tid + it * NT;
                if (k >= PL) break;
                float w0 = IN[k], w1 = IN[PL + k], w2 = IN[2 * PL + k], w3 = IN[3 * PL + k];
                if (a.stage >= 2) {
                    w0 += IN[4 * PL + k]; w1 += IN[5 * PL + k]; w2 += IN[6 * PL + k]; w3 += IN[7 * PL + k];
                }
                const bool ce = (cemask >> it) & 1u;
                const float ir = frcp(w0);
                const float E = w3;
                w1 *= ir;
                w2 *= ir;
                w3 = gm1 * (E - 0.5f * w0 * (w1 * w1 + w2 * w2));
                if (ce) {
                    const float cs2 = gam * w3 * ir;
                    W[4 * PL + k] = fsqrt(cs2 > 1e-14f ? cs2 : 1e-14f);
                    W[5 * PL + k] = E;
                }
                W[k] = w0; W[PL + k] = w1; W[2 * PL + k] = w2; W[3 * PL + k] = w3;
            }
        }
        __syncthreads();
        // a halo load that never arrived (seen by any thread): record it and
        // stop; every thread reads s_err after the same barrier
        if (s_err) {
            if (tid == 0 && gd.ctrl) gd.ctrl->status = FVB_ERR_TIMEOUT;
            break;
        }
        // ---- 2. load the next tile into IN (asynchronous through TMA) -------
        // (in a batched launch warp 0 also fetches that tile's header)
        bool next_tma = false;
        if (has_next) {
            if (batched) {
                if (tid < 32) {
                    start_batched_tile<P32C>(a, &s_hdr[slot ^ 1], ref_next, wnext, &s_bar, tid,
                                             [&](const TileHdr &h) {
                                                 issue_tile_load<P32C, G, SW, SH, NT>(h.gd, a.stage, cur,
                                                                                      ref_next.tile, IN, &s_bar, 0);
                                             });
                    if (tid == 0) s_ref_next = ref_after;
                }
                next_tma = true;
            } else {
                next_tma = start_single(t + stride);
            }
        }
        if (!ctl.run) {
            if (ctl.copy) {
                // skipped step: the next step reads the other buffer
                const float *hi = (const float *)gd.st[cur], *lo = (const float *)gd.lo[cur];
                for (int k = tid; k < NC; k += NT) {
                    int r = k / TX, c = k - r * TX, i = tx0 + c, j = ty0 + r;
                    if (i >= n || j >= n) continue;
                    float vh[4], vl[4];
                    long long e = gidx(gd, 0, j, i);
                    for (int q = 0; q < 4; ++q) { vh[q] = hi[e + q * gd.plane]; vl[q] = lo[e + q * gd.plane]; }
                    put_cell2<float>(gd, (float *)gd.st[nxt], (float *)gd.lo[nxt], j, i, vh, vl);
                }
            }
            wait_box(next_tma);
            continue;
        }
        const float dt = (float)ctl.dt;
        const float dt_h = dt * (float)gd.inv_h;

        // ---- 3. face fluxes, x-face p and y-face p as one packed pair -------
        for (int p = tid; p < NP; p += NT) {
            const int px = p < NXF ? p : NXF - 1, py = p < NYF ? p : NYF - 1;
            const int rx = px / (TX + 1), cx = px - rx * (TX + 1);
            const int ry = py / TX, cy = py - ry * TX;
            const int bx = (rx + G) * SW + (cx + G), by = (ry + G) * SW + (cy + G);
            f2::V L[4], Rv[4], WL[4], WR[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                // x lane: (rho, u, v, p) along x; y lane: (rho, v, u, p) along y
                const float *vx = W + m * PL + bx;
                const float *vy = W + (m == 1 ? 2 : m == 2 ? 1 : m) * PL + by;
                f2::V s[8];
#pragma unroll
                for (int d = 0; d < 8; ++d) s[d] = make_float2(vx[d - G], vy[(d - G) * SW]);
                f2::upface7(s, L[m], Rv[m]);
                WL[m] = s[G - 1];
                WR[m] = s[G];
            }
            f2::floors(L, Rv);
            const float *cex = W + 4 * PL + bx, *cey = W + 4 * PL + by;
            f2::V F[4];
            f2::face_flux(L, Rv, WL, WR, make_float2(cex[-1], cey[-SW]), make_float2(cex[0], cey[0]),
                          make_float2(cex[PL - 1], cey[PL - SW]), make_float2(cex[PL], cey[PL]), gam, igm1, F);
            if (p < NXF) {
                float *o = FX + rx * (TX + 1) + cx;
                constexpr int os = TY * (TX + 1);
                o[0] = F[0].x; o[os] = F[1].x; o[2 * os] = F[2].x; o[3 * os] = F[3].x;
            }
            if (p < NYF) {
                float *o = FY + ry * TX + cy;
                constexpr int os = (TY + 1) * TX;
                // y lane: normal momentum is v, tangential u
                o[0] = F[0].y; o[os] = F[2].y; o[2 * os] = F[1].y; o[3 * os] = F[3].y;
            }
        }
        __syncthreads();

        if (!has_next) grid_release();
        // ---- 4. divergence, RK combination, stores --------------------------
        float lmax = 0.0f;
        for (int k = tid; k < NC; k += NT) {
            const int r = k / TX, c = k - r * TX, i = tx0 + c, j = ty0 + r;
            if (i >= n || j >= n) continue;
            float dres[4];  // dt L
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float *fx = FX + q * TY * (TX + 1) + r * (TX + 1) + c;
                const float *fy = FY + q * (TY + 1) * TX + r * TX + c;
                dres[q] = -((fx[1] - fx[0]) + (fy[TX] - fy[0])) * dt_h;
            }
            Operands32c o;
            load_operands32c(gd, a.stage, cur, j, i, o);
            update_cell32c(gd, a.stage, nxt, j, i, dres, o, gam, gm1, lmax);
        }

        // ---- 5. max wave speed of the new state (stage 3) ------------------
        if (a.stage == 3) {
            // (a batched launch advances each grid's time where its tile 0's header is published)
            if (!batched && tid == 0 && tile == 0) leader_finish<P32C>(gd.ctrl);
            if (batched) {
                // tiles of one CTA belong to different grids: one atomic per
                // warp and tile
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
                if ((tid & 31) == 0 && lmax > 0.0f)
                    atomicMax(&gd.ctrl->lam_acc, (unsigned long long)__double_as_longlong((double)lmax));
            } else {
                lacc = fmax(lacc, (double)lmax);
            }
        }
        // ---- 6. next tile's halo box -----------------------------------------
        wait_box_own(next_tma);
    }
    if (!batched && a.stage == 3) {
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
// Row-pair form of the compensated stage kernel.
//
// The two lanes of every packed register are the same face, or the same
// cell, in two rows HT = TY / 2 apart: the working tile keeps each quantity
// as float2 pairs (box row r, box row r + HT) for r in [0, HT + 2G), so
// x-faces pair with x-faces and y-faces with y-faces (one index pattern and
// component order in both lanes).  On that tile of TX x HT pairs a thread
// takes, as in the FP64 kernel (fvb_stage64.cuh), two neighbouring x-faces and
// two neighbouring y-faces, four faces of each direction: the nine stencil
// points of a variable are five 16-byte loads along x and nine 8-byte ones
// along y for four faces, against sixteen 4-byte ones for two, and the y-fluxes
// stay with the thread that updates their cells.  HT = 2 NK - 1 rows, TX NK
// threads, each updating up to four cells as two packed pairs.  The halo box, the tile walk, the
// step control and the per-cell update are those of stage32c_kernel above; the
// rows the two halves share are converted once per half.
//
// Measured, KH 2048^2, stage 1 / 2 / 3: 109 / 118 / 145 us (430, 480, 570
// instructions a cell) against 119 / 130 / 157 (616 in stage 2) for
// stage32c_kernel; a step 0.347 against 0.376 ms.  In stage 3 the operands of
// two cells are loaded before the barrier and those of the other two after
// the first update (all four before it spill: 181 us), and the lo words,
// which nothing has read yet, are prefetched into L2 at the tile's start
// (145 against 152 us).
// ---------------------------------------------------------------------------
template <int TX, int TY>
struct RowPair {
    static constexpr int G = 4, HT = TY / 2, NK = (HT + 1) / 2, NT = TX * NK;
    static constexpr int SW = TX + 2 * G, SH = TY + 2 * G, PL = SW * SH;
    static constexpr int PR = HT + 2 * G;             // pair rows of the working tile
    static constexpr int P2 = PR * SW;                // pairs per working plane
    static constexpr int CW = TX + 2, C2 = (HT + 2) * CW;  // pairs of the c / E planes: cells -1 .. HT, -1 .. TX
    static constexpr int XP = TX / 2 + 1, FW = 2 * XP;     // x-face pairs of a row, row of FX2
    static constexpr int r16(int v) { return (v + 15) / 16 * 16; }  // in pairs: 128 bytes
    static constexpr int oW = r16(8 * PL / 2), oCE = oW + r16(4 * P2), oFX = oCE + r16(2 * C2),
                         oFY = oFX + r16(4 * HT * FW);
    static constexpr size_t smem = sizeof(float2) * (size_t)(oFY + 4 * NK * TX);
    static constexpr int fit = (int)(227 * 1024 / (smem + 2048)), regs = 512 / NT;
    static constexpr int MINB = fit < regs ? fit : regs;  // resident CTAs an SM, at 128 registers a thread
};

// How a launch's tiles reach its CTAs (as the FP64 kernel's M64_ modes): a fixed
// share each, a table's, or, on single grids of more than two waves, taken
// from the stage's counter (tile_queue) between the x- and the y-faces.
// us a stage, fixed / queued: 1800^2 92.7 / 89.6, 2048^2 116 / 111, 4096^2
// 448 / 406; 1024^2 (3.8 waves) 34.3 / 34.5.  (The x/y pair kernel above, for
// smaller grids, has one face loop, so the box would start with nothing but the
// update left: taken with the conversion, -4 ... +2 %, so it has no such mode.)
enum { M32P_FIXED, M32P_BATCHED, M32P_QUEUED };

template <int TX, int TY, int MODE>
__global__ void __launch_bounds__((RowPair<TX, TY>::NT), (RowPair<TX, TY>::MINB))
    stage32p_kernel(const __grid_constant__ StageArgs a)
{
    using RP = RowPair<TX, TY>;
    static_assert(TY % 2 == 0 && RP::HT % 2 == 1, "two halves of an odd height");
    constexpr int G = RP::G, HT = RP::HT, NK = RP::NK, NT = RP::NT, SW = RP::SW, SH = RP::SH, PL = RP::PL;
    constexpr int P2 = RP::P2, CW = RP::CW, C2 = RP::C2, XP = RP::XP, FW = RP::FW;
    constexpr int NC = TX * TY;
    constexpr int NW = NT / 32;
    constexpr int HS = HT * SW;  // box offset of the upper half's rows

    // IN: the halo box as loaded (hi + increment planes); W2: rho, u, v, p
    // as row pairs; CE2: sound speed and energy as row pairs; FX2 / FY2: face
    // fluxes as row pairs (FY2: the lower face of each thread's two)
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float *IN = reinterpret_cast<float *>(smem_raw);
    float2 *sm2 = reinterpret_cast<float2 *>(smem_raw);
    float2 *W2 = sm2 + RP::oW, *CE2 = sm2 + RP::oCE;
    float2 *FX2 = sm2 + RP::oFX;             // [4][HT][FW]
    float2 *FY2 = sm2 + RP::oFY;             // [4][NK][TX]
    __shared__ double s_red[NW];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ int s_err, s_next;
    __shared__ __align__(16) TileHdr s_hdr[2];
    __shared__ TileRef s_ref_next;

    const int tid = threadIdx.x;
    constexpr bool batched = MODE == M32P_BATCHED, QUEUED = MODE == M32P_QUEUED;
    const int cur = a.parity, nxt = a.parity ^ 1;
    if (tid == 0) {
        mbar_init(&s_bar, 1);
        s_err = 0;
    }
    __syncthreads();
    const int ntiles = batched ? *a.ntiles : a.ntiles_static;
    BatchHead head{};
    if (batched && tid < 32) head = batch_head(a, &s_hdr[0], ntiles, tid);
    grid_dependency();

    uint32_t phase = 0;
    auto wait_box = [&](bool tma) {
        if (tma) {
            if (mbar_wait(&s_bar, phase)) phase ^= 1;
            else s_err = 1;
        }
        __syncthreads();
    };
    // end-of-tile wait without a block barrier for a TMA-fed box, as in
    // stage32c_kernel (W2 / FX2 / FY2 in place of W / FX / FY)
    auto wait_box_own = [&](bool tma) {
        if (tma) {
            if (mbar_wait(&s_bar, phase)) phase ^= 1;
            else s_err = 1;
        } else {
            __syncthreads();
        }
    };
    auto start_single = [&](int t) -> bool {
        if (tid == 0 && a.grid.tmap) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue_tile_load<P32C, G, SW, SH, NT>(a.grid, a.stage, cur, t, IN, &s_bar, tid);
        return a.grid.tmap != nullptr;
    };
    // failure injection (fvb_debug_drop_load), as in stage32c_kernel
    const bool drop = !batched && blockIdx.x == 0 && a.stage > 0 && a.grid.ctrl && a.grid.tmap &&
                      *(volatile int *)&a.grid.ctrl->drop_load;
    const int stride = gridDim.x;
    int t = blockIdx.x, slot = 0;
    if (t < ntiles && batched) {
        if (tid < 32) {
            const TileRef r0 = head.first;
            start_first_tile<P32C>(a, &s_hdr[0], r0, &s_bar, tid, [&](const TileHdr &h) {
                issue_tile_load<P32C, G, SW, SH, NT>(h.gd, a.stage, cur, r0.tile, IN, &s_bar, 0);
            });
            if (tid == 0) s_ref_next = head.next;
        }
        wait_box(true);
    } else if (drop) {
        wait_box(true);
        if (tid == 0) a.grid.ctrl->drop_load = 0;
    } else {
        wait_box(t < ntiles ? start_single(t) : false);
    }
    double lacc = 0.0;
    TileCtl ctl1{};
    if (!batched && t < ntiles) ctl1 = tile_control<P32C>(a.grid.ctrl, a.stage, tid == 0 && t == 0);
    if (QUEUED && tid == 0 && t == 0) clear_tile_queue(a.grid.ctrl, a.stage);
    for (int next; t < ntiles; t = next, slot ^= 1) {
        next = t + stride;
        bool has_next = next < ntiles;
        unsigned long long wnext = 0ull;
        TileRef ref_next{}, ref_after{};
        if (batched && tid < 32) {
            if (has_next) {
                ref_next = s_ref_next;
                wnext = hdr_word(a, ref_next, tid);
            }
            if (t + 2 * stride < ntiles) ref_after = a.tiles[t + 2 * stride];
        }
        const GridDev &gd = tile_grid<batched>(s_hdr[slot], a);
        const int tile = batched ? s_hdr[slot].tile : t;
        const TileCtl ctl = batched ? s_hdr[slot].ctl : ctl1;
        const int n = gd.n;
        const int tx0 = (tile % gd.tiles_x) * TX, ty0 = (tile / gd.tiles_x) * TY;
        const float gam = (float)gd.gam, gm1 = (float)gd.gam - 1.0f, igm1 = (float)gd.igm1;
        // rows of the tile inside the grid: pair rows beyond them are skipped
        const int rows = n - ty0 < HT ? n - ty0 : HT;
        // ---- 1. stage input U0 + d into W2 as primitive row pairs (+ c, E
        //         where the HLLE reads them) -----------------------------------
        if (ctl.run) {
            const f2::V nhalf = f2::splat(-0.5f), G1 = f2::splat(gm1), GA = f2::splat(gam);
            const int np2 = (rows + 2 * G) * SW;
#pragma unroll 2
            for (int k = tid; k < np2; k += NT) {
                f2::V w0 = make_float2(IN[k], IN[k + HS]), w1 = make_float2(IN[PL + k], IN[PL + k + HS]);
                f2::V w2 = make_float2(IN[2 * PL + k], IN[2 * PL + k + HS]);
                f2::V w3 = make_float2(IN[3 * PL + k], IN[3 * PL + k + HS]);
                if (a.stage >= 2) {
                    w0 = f2::add(w0, make_float2(IN[4 * PL + k], IN[4 * PL + k + HS]));
                    w1 = f2::add(w1, make_float2(IN[5 * PL + k], IN[5 * PL + k + HS]));
                    w2 = f2::add(w2, make_float2(IN[6 * PL + k], IN[6 * PL + k + HS]));
                    w3 = f2::add(w3, make_float2(IN[7 * PL + k], IN[7 * PL + k + HS]));
                }
                const f2::V ir = f2::rcp(w0);
                const f2::V E = w3;
                w1 = f2::mul(w1, ir);
                w2 = f2::mul(w2, ir);
                // p = (gamma - 1)(E - rho (u^2 + v^2) / 2)
                w3 = f2::mul(G1, f2::fma(f2::mul(nhalf, w0), f2::fma(w1, w1, f2::mul(w2, w2)), E));
                const int r = k / SW, c = k - r * SW;
                if ((unsigned)(r - (G - 1)) < (unsigned)(HT + 2) && (unsigned)(c - (G - 1)) < (unsigned)CW) {
                    const f2::V cs2 = f2::mul(f2::mul(GA, w3), ir);
                    const int kc = (r - (G - 1)) * CW + (c - (G - 1));
                    CE2[kc] = f2::vsqrt(f2::vmax(cs2, f2::splat(1e-14f)));
                    CE2[C2 + kc] = E;
                }
                W2[k] = w0; W2[P2 + k] = w1; W2[2 * P2 + k] = w2; W2[3 * P2 + k] = w3;
            }
        }
        __syncthreads();
        // a halo load that never arrived (seen by any thread): record it and
        // stop; every thread reads s_err after the same barrier
        if (s_err) {
            if (tid == 0 && gd.ctrl) gd.ctrl->status = FVB_ERR_TIMEOUT;
            break;
        }
        // ---- 2. load the next tile into IN (asynchronous through TMA) -------
        bool next_tma = false;
        if (has_next) {
            if (batched) {
                if (tid < 32) {
                    start_batched_tile<P32C>(a, &s_hdr[slot ^ 1], ref_next, wnext, &s_bar, tid,
                                             [&](const TileHdr &h) {
                                                 issue_tile_load<P32C, G, SW, SH, NT>(h.gd, a.stage, cur,
                                                                                      ref_next.tile, IN, &s_bar, 0);
                                             });
                    if (tid == 0) s_ref_next = ref_after;
                }
                next_tma = true;
            } else if (!QUEUED || !ctl.run) {
                next_tma = start_single(next);
            }
        }
        if (!ctl.run) {
            if (ctl.copy) {
                // skipped step: the next step reads the other buffer
                const float *hi = (const float *)gd.st[cur], *lo = (const float *)gd.lo[cur];
                for (int k = tid; k < NC; k += NT) {
                    int r = k / TX, c = k - r * TX, i = tx0 + c, j = ty0 + r;
                    if (i >= n || j >= n) continue;
                    float vh[4], vl[4];
                    long long e = gidx(gd, 0, j, i);
                    for (int q = 0; q < 4; ++q) { vh[q] = hi[e + q * gd.plane]; vl[q] = lo[e + q * gd.plane]; }
                    put_cell2<float>(gd, (float *)gd.st[nxt], (float *)gd.lo[nxt], j, i, vh, vl);
                }
            }
            wait_box(next_tma);
            continue;
        }
        const float dt = (float)ctl.dt;
        const float dt_h = dt * (float)gd.inv_h;

        if (a.stage == 3) {
            // the lo words come from DRAM: into L2 while the faces are computed
            for (int m = tid; m < 4 * TY; m += NT) {
                const int q = m / TY, j = ty0 + (m - q * TY);
                if (j < n) {
                    const float *pl = (const float *)gd.lo[cur] + gidx(gd, q, j, tx0);
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(pl));
                }
            }
        }
        int taken = ntiles;
        if (QUEUED && tid == 0) taken = stride + atomicAdd(tile_queue(a.grid.ctrl, a.stage), 1);
        // ---- 3. x-faces 2j, 2j + 1 of pair row r -------------------------------
        for (int p = tid; p < XP * rows; p += NT) {
            const int r = p / XP, j = p - r * XP;
            f2::V LA[4], RA[4], LB[4], RB[4], V0[4], V1[4], V2[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const float4 *v = reinterpret_cast<const float4 *>(W2 + m * P2 + (r + G) * SW + 2 * j);
                f2::V s[2 * G + 2];
#pragma unroll
                for (int d = 0; d <= G; ++d) {
                    const float4 x = v[d];
                    s[2 * d] = make_float2(x.x, x.y);
                    s[2 * d + 1] = make_float2(x.z, x.w);
                }
                f2::upface7(s, LA[m], RA[m]);
                f2::upface7(s + 1, LB[m], RB[m]);
                V0[m] = s[G - 1];
                V1[m] = s[G];
                V2[m] = s[G + 1];
            }
            const f2::V *ce = CE2 + (r + 1) * CW + 2 * j;
            f2::V FA[4], FB[4];
            f2::floors(LA, RA);
            f2::floors(LB, RB);
            f2::face_flux(LA, RA, V0, V1, ce[0], ce[1], ce[C2], ce[C2 + 1], gam, igm1, FA);
            f2::face_flux(LB, RB, V1, V2, ce[1], ce[2], ce[C2 + 1], ce[C2 + 2], gam, igm1, FB);
            float4 *o = reinterpret_cast<float4 *>(FX2 + r * FW + 2 * j);
#pragma unroll
            for (int q = 0; q < 4; ++q) o[q * (HT * FW / 2)] = make_float4(FA[q].x, FA[q].y, FB[q].x, FB[q].y);
        }
        if (QUEUED && tid == 0) {
            s_next = taken;
            if (taken < ntiles) start_single(taken);
        }
        // ---- 4. y-faces 2k, 2k + 1 of column c (normal velocity v) ------------
        const int k = tid / TX, c = tid - k * TX, i = tx0 + c;
        f2::V F0[4], F1[4];
        if (2 * k <= rows) {
            f2::V LA[4], RA[4], LB[4], RB[4], V0[4], V1[4], V2[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const f2::V *v = W2 + (m == 1 ? 2 : m == 2 ? 1 : m) * P2 + 2 * k * SW + (c + G);
                f2::V s[2 * G + 1];
#pragma unroll
                for (int d = 0; d <= 2 * G; ++d) s[d] = v[d * SW];
                f2::upface7(s, LA[m], RA[m]);
                f2::upface7(s + 1, LB[m], RB[m]);
                V0[m] = s[G - 1];
                V1[m] = s[G];
                V2[m] = s[G + 1];
            }
            const f2::V *ce = CE2 + 2 * k * CW + c + 1;
            f2::V FA[4], FB[4];
            f2::floors(LA, RA);
            f2::floors(LB, RB);
            f2::face_flux(LA, RA, V0, V1, ce[0], ce[CW], ce[C2], ce[C2 + CW], gam, igm1, FA);
            f2::face_flux(LB, RB, V1, V2, ce[CW], ce[2 * CW], ce[C2 + CW], ce[C2 + 2 * CW], gam, igm1, FB);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int s = q == 1 ? 2 : q == 2 ? 1 : q;  // Cartesian components
                F0[q] = FA[s];
                F1[q] = FB[s];
                FY2[(q * NK + k) * TX + c] = F0[q];
            }
        }
        // the operands of this thread's cells: pair rows 2k, 2k + 1, both halves
        Operands32c ops[2];
        auto load_ops = [&](int h) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int r = 2 * k + h, j = ty0 + r + b * HT;
                if (r < HT && i < n && j < n) load_operands32c(gd, a.stage, cur, j, i, ops[b]);
            }
        };
        load_ops(0);
        __syncthreads();
        if (QUEUED) {
            next = s_next;
            has_next = next_tma = next < ntiles;
        }

        if (!has_next) grid_release();
        // ---- 5. divergence as pairs, then each cell's RK update ---------------
        float lmax = 0.0f;
        const f2::V ndt = f2::splat(-dt_h);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = 2 * k + h;
            if (r >= rows) continue;
            f2::V dr[4];  // dt L of cells (r, c) and (r + HT, c)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const f2::V *fx = FX2 + (q * HT + r) * FW + c;
                const f2::V dy = h == 0 ? f2::sub(F1[q], F0[q]) : f2::sub(FY2[(q * NK + k + 1) * TX + c], F1[q]);
                dr[q] = f2::mul(f2::add(f2::sub(fx[1], fx[0]), dy), ndt);
            }
            const int j = ty0 + r;
            update_pair32c(gd, a.stage, nxt, j, j + HT, i, i < n, i < n && j + HT < n, dr, ops[0], ops[1], gam, gm1,
                           lmax);
            if (h == 0) load_ops(1);
        }

        // ---- 6. max wave speed of the new state (stage 3) ------------------
        if (a.stage == 3) {
            if (!batched && tid == 0 && tile == 0) leader_finish<P32C>(gd.ctrl);
            if (batched) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
                if ((tid & 31) == 0 && lmax > 0.0f)
                    atomicMax(&gd.ctrl->lam_acc, (unsigned long long)__double_as_longlong((double)lmax));
            } else {
                lacc = fmax(lacc, (double)lmax);
            }
        }
        // ---- 7. next tile's halo box -----------------------------------------
        wait_box_own(next_tma);
    }
    if (!batched && a.stage == 3) {
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
    if (s_err && gd_has_tma(a)) mbar_wait(&s_bar, phase);
}

template <int SHAPE>
static StageKernel entry32c()
{
    constexpr TileShape ts = kTileShapes32c[SHAPE];
    if constexpr (row_pairs(ts)) {
        static_assert(ts.nt == RowPair<ts.tx, ts.ty>::NT, "one y-face pair a thread");
        return StageKernel{(void *)stage32p_kernel<ts.tx, ts.ty, M32P_FIXED>,
                           (void *)stage32p_kernel<ts.tx, ts.ty, M32P_BATCHED>, RowPair<ts.tx, ts.ty>::smem, ts.nt,
                           (void *)stage32p_kernel<ts.tx, ts.ty, M32P_QUEUED>};
    } else {
        constexpr int sw = ts.tx + 8, sh = ts.ty + 8;
        constexpr size_t smem = sizeof(float) * ((size_t)14 * sw * sh + 4 * ts.ty * (ts.tx + 1) + 4 * (ts.ty + 1) * ts.tx);
        return StageKernel{(void *)stage32c_kernel<ts.tx, ts.ty, ts.nt, false>,
                           (void *)stage32c_kernel<ts.tx, ts.ty, ts.nt, true>, smem, ts.nt};
    }
}

StageKernel stage32c_kernel_of(int shape)
{
    static_assert(kNumTileShapes == 7, "one entry a shape");
    switch (shape) {
    case 0: return entry32c<0>();
    case 1: return entry32c<1>();
    case 2: return entry32c<2>();
    case 3: return entry32c<3>();
    case 4: return entry32c<4>();
    case 5: return entry32c<5>();
    case 6: return entry32c<6>();
    default: return StageKernel{};
    }
}

}  // namespace fvb
