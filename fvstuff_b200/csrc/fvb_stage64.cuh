// fvb_stage64.cuh -- the SSP-RK3 stage kernel of the FP64 plain method.
//
// The pipeline of fvb_stage.cu (persistent CTAs over the tiles of one grid or
// of a batch's tile table; TMA halo boxes; every face once; RK update with
// ghost images; stage-3 wave-speed max), laid out for FP64:
//
//   * The state is primitive, so the faces read the TMA box itself; two boxes
//     alternate, and the next tile's load has a whole tile to arrive.  Only
//     each cell's sound speed and energy (for the HLLE) are formed before the
//     faces.
//   * A thread evaluates two neighbouring x-faces, then two neighbouring
//     y-faces: the nine cells of both stencils are loaded once (five 16-byte
//     loads a variable along x, nine 8-byte ones along y, against sixteen),
//     and the two fluxes are independent instruction streams.  With TX columns
//     and NK row pairs there are TX NK threads, exactly one y-pair each, and
//     TY = 2 NK - 1 rows (an even number of y-face rows).
//   * The thread of a y-pair updates the two cells above its faces: its own
//     fluxes stay in registers, only the lower one of each pair goes through
//     shared memory to the pair below it.
//   * U0 of the tile (stages 2 and 3) arrives by TMA during the faces.
//
// What bounds it: instruction issue and the FP64 pipe together (a 2048^2
// stage is 55 us of memory at the copy bandwidth).  Against one face a
// thread, a copied working tile and U0 through registers, a cell takes 826
// instructions instead of 1097 and 405 FP64 ones instead of 480, and a 2048^2
// stage 179 us instead of 231; 801 and 164 with queued tiles (below), 833 and 165
// with floors that compare all bits (fvb_face64.cuh).
#pragma once
#include <stdint.h>

#include "fvb_internal.h"
#include "fvb_device.cuh"
#include "fvb_tma.cuh"
#include "fvb_face64.cuh"

namespace fvb {

// A tile shape's layout.  NT = TX (TY + 1) / 2 threads take pairs of faces, as
// above; with NT >= 2 TX (TY + 1) (the split form) the lower half of the
// threads takes one x-face each while the upper half takes one y-face each,
// and a thread updates one cell: a quarter of the serial work, for grids whose
// tiles are fewer than the SMs.
template <int ORDER, int TX, int TY, int NT>
struct L64 {
    static constexpr int G = (ORDER + 1) / 2;
    static constexpr int NK = (TY + 1) / 2;
    static constexpr bool SPLIT = NT >= 2 * TX * (TY + 1);
    static_assert(SPLIT || (NT == TX * NK && TY == 2 * NK - 1), "one y-pair a thread");
    static_assert(!SPLIT || NT / 2 >= (TX + 1) * TY, "one x-face a thread");
    static constexpr int NFY = SPLIT ? TY + 1 : NK;             // y-face rows kept in shared memory
    // a TMA box starts on an even column (16 bytes); with an odd ghost width
    // the tile's first column is odd, so the box starts one column earlier
    static constexpr int XO = (16 - G) & 1;
    static constexpr int SW = TX + 2 * G + 2 * XO, SH = TY + 2 * G, PL = SW * SH;
    static constexpr int CW = TX + 2, CP = (TY + 2) * CW;       // cells -1 .. TX, -1 .. TY
    static constexpr int XP = TX / 2 + 1, FW = 2 * XP;          // x-face pairs of a row, row of FX
    static constexpr int r16(int v) { return (v + 15) / 16 * 16; }
    static constexpr int BOX = r16(4 * PL);
    static constexpr bool U0S = ORDER != 9;  // UP9's wider boxes leave no room for U0 beside two CTAs
    static constexpr int oCE = 2 * BOX, oFX = oCE + r16(2 * CP), oFY = oFX + 4 * TY * FW, oU0 = r16(oFY + 4 * NFY * TX);
    static constexpr size_t smem = sizeof(double) * (size_t)(oU0 + (U0S ? 4 * TY * TX : 0));
    // resident CTAs an SM is compiled for, at 128 registers a thread
    static constexpr int fit = (int)(227 * 1024 / (smem + 1024));
    static constexpr int regs = 512 / NT;
    static constexpr int MINB = fit < regs ? fit : regs;
};

// How a launch's tiles reach its CTAs.  FIXED: each CTA a fixed share, in turn,
// the next box loaded from the top of a tile.  QUEUED (single grids on tensor
// maps): a CTA takes its next tile (tile_queue) when it comes to its
// y-faces, so that none is left with a whole tile while others are done; the
// box has the y-faces and the update to arrive.  us a stage, fixed / queued:
// 2048^2 179 / 164, 1024^2 50.5 / 47.2, 777^2 33.0 / 28.9.  BATCHED: a fixed
// share of a tile table.
enum { M64_FIXED, M64_BATCHED, M64_QUEUED };

template <int ORDER, int TX, int TY, int NT, int MODE, int RS>
__global__ void __launch_bounds__(NT, (L64<ORDER, TX, TY, NT>::MINB)) stage64_kernel(const __grid_constant__ StageArgs a)
{
    constexpr bool BATCHED = MODE == M64_BATCHED, QUEUED = MODE == M64_QUEUED;
    using P = L64<ORDER, TX, TY, NT>;
    constexpr bool SPLIT = P::SPLIT;
    constexpr int G = P::G, NK = P::NK, XO = P::XO, SW = P::SW, SH = P::SH, PL = P::PL;
    constexpr int CW = P::CW, CP = P::CP, XP = P::XP, FW = P::FW, NW = (NT + 31) / 32;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    double *sm = reinterpret_cast<double *>(smem_raw);
    double *CE = sm + P::oCE;  // [2][TY+2][TX+2] sound speed, energy
    double *FX = sm + P::oFX;  // [4][TY][FW]
    double *FY = sm + P::oFY;  // [4][NFY][TX] the lower face of each pair (split: every face)
    double *U0 = sm + P::oU0;  // [4][TY][TX]
    __shared__ double s_red[NW];
    __shared__ __align__(8) uint64_t s_bar[3];  // two boxes, U0
    __shared__ int s_err, s_next;
    __shared__ __align__(16) TileHdr s_hdr[2];
    __shared__ TileRef s_ref_next;  // batched: table entry of the CTA's next tile

    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int m = 0; m < 3; ++m) mbar_init(&s_bar[m], 1);
        s_err = 0;
    }
    __syncthreads();
    const int ntiles = BATCHED ? *a.ntiles : a.ntiles_static;
    BatchHead head{};
    if (BATCHED && tid < 32) head = batch_head(a, &s_hdr[0], ntiles, tid);
    grid_dependency();

    // every thread waits on the mbarrier itself (the completed phase makes the
    // TMA bytes visible to it); the barrier after the wait also agrees on s_err
    uint32_t phase = 0;  // bit m: the phase of s_bar[m] to wait for
    uint32_t lost = 0;   // bit m: a wait on s_bar[m] gave up
    auto wait_bar = [&](int m) -> bool {
        if (!mbar_wait(&s_bar[m], (phase >> m) & 1u)) {
            s_err = 1;
            lost |= 1u << m;
            return false;
        }
        phase ^= 1u << m;
        return true;
    };
    auto wait_box = [&](int m, bool tma) {
        if (tma) wait_bar(m);
        else cp_async_wait();
        __syncthreads();
    };
    // single grid: start the halo-box load of tile t (every thread: the
    // plain path loads cooperatively)
    auto start_single = [&](int t, int m) -> bool {
        if (tid == 0 && a.grid.tmap) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue_tile_load64<G, TX, TY, SW, XO, NT>(a.grid, a.stage, t, sm + m * P::BOX, &s_bar[m], tid);
        return a.grid.tmap != nullptr;
    };
    // failure injection (fvb_debug_drop): CTA 0 of a single-grid launch
    // issues no first box load, or no U0 load for its first tile, so its bounded
    // wait runs out and the grid's status becomes FVB_ERR_TIMEOUT; the flag is
    // read by every thread of that CTA before thread 0 clears it behind the
    // first barrier
    const int armed = !BATCHED && blockIdx.x == 0 && a.stage > 0 && a.grid.ctrl && a.grid.tmap
                          ? *(volatile int *)&a.grid.ctrl->drop_load : 0;
    const bool drop = armed == FVB_DROP_BOX, drop_u0 = armed == FVB_DROP_U0 && a.stage >= 2;
    const int stride = gridDim.x;
    int t = blockIdx.x, buf = 0;
    if (t < ntiles && BATCHED) {
        if (tid < 32) {
            const TileRef r0 = head.first;
            start_first_tile<P64>(a, &s_hdr[0], r0, &s_bar[0], tid, [&](const TileHdr &h) {
                issue_tile_load64<G, TX, TY, SW, XO, NT>(h.gd, a.stage, r0.tile, sm, &s_bar[0], 0);
            });
            if (tid == 0) s_ref_next = head.next;
        }
        wait_box(0, true);
    } else if (drop) {
        wait_box(0, true);  // nothing was issued: the wait runs out
        if (tid == 0) a.grid.ctrl->drop_load = 0;
    } else {
        wait_box(0, t < ntiles ? start_single(t, 0) : false);
    }
    // single grid: the stage-3 wave-speed max is reduced once per CTA, and the
    // step control, the same for every tile, is read once (the leader is CTA
    // 0, whose first tile is tile 0)
    if (drop_u0 && tid == 0) a.grid.ctrl->drop_load = 0;
    double lacc = 0.0;
    TileCtl ctl1{};
    if (!BATCHED && t < ntiles) ctl1 = tile_control<P64>(a.grid.ctrl, a.stage, tid == 0 && t == 0);
    if (QUEUED && tid == 0 && t == 0) clear_tile_queue(a.grid.ctrl, a.stage);
    if (QUEUED && !ctl1.run && !s_err) t = ntiles;
    for (int next; t < ntiles; t = next, buf ^= 1) {
        next = t + stride;
        // warp 0 of a batched launch: the next tile's descriptor word and the
        // entry of the tile after it, in flight while c and E are formed
        bool has_next = next < ntiles;
        unsigned long long wnext = 0ull;
        TileRef ref_next{}, ref_after{};
        if (BATCHED && tid < 32) {
            if (has_next) {
                ref_next = s_ref_next;
                wnext = hdr_word(a, ref_next, tid);
            }
            if (t + 2 * stride < ntiles) ref_after = a.tiles[t + 2 * stride];
        }
        const GridDev &gd = tile_grid<BATCHED>(s_hdr[buf], a);
        const int tile = BATCHED ? s_hdr[buf].tile : t;
        const TileCtl ctl = BATCHED ? s_hdr[buf].ctl : ctl1;
        const int n = gd.n;
        const int tx0 = (tile % gd.tiles_x) * TX, ty0 = (tile / gd.tiles_x) * TY;
        const f64::Gas gf{gd.gam, gd.igm1, gd.gam - 1.0};
        if (s_err) {
            // a load never arrived: no tile of this CTA from here on is computed;
            // record it for their grids, stop
            if constexpr (BATCHED) {
                for (int k = t + tid * stride; k < ntiles; k += NT * stride)
                    a.ctrls[a.tiles[k].grid].status = FVB_ERR_TIMEOUT;
            } else if (tid == 0 && gd.ctrl) {
                gd.ctrl->status = FVB_ERR_TIMEOUT;
            }
            break;
        }
        // ---- 1. start the next tile's box (its buffer was last read before
        //         the barrier that ended the previous tile) and this tile's U0 --
        bool next_tma = false;
        if (!BATCHED && !QUEUED && has_next) next_tma = start_single(next, buf ^ 1);
        const bool u0_tma = P::U0S && ctl.run && a.stage >= 2 && gd.tmap;
        if (u0_tma && tid == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (!drop_u0) {
                mbar_expect_tx(&s_bar[2], 4u * TY * TX * sizeof(double));
                tma_load3(U0, gd.tmap + TM_U0, gd.xoff + G + tx0, G + ty0, 0, &s_bar[2]);
            }
        }
        // ---- 2. sound speed and energy of the cells the HLLE reads ----------
        const double *IN = sm + buf * P::BOX;
        if (ctl.run) {
            for (int k = tid; k < CP; k += NT) {
                const int r = k / CW, c = k - r * CW, e = (r + G - 1) * SW + (c + G - 1 + XO);
                const double rho = IN[e], u = IN[PL + e], v = IN[2 * PL + e], p = IN[3 * PL + e];
                CE[k] = f64::snd(gf.gam * p, rho);
                CE[CP + k] = f64::energy(rho, u, v, p, gf);
            }
        }
        __syncthreads();
        if (BATCHED && has_next) {
            if (tid < 32) {
                start_batched_tile<P64>(a, &s_hdr[buf ^ 1], ref_next, wnext, &s_bar[buf ^ 1], tid,
                                        [&](const TileHdr &h) {
                                            issue_tile_load64<G, TX, TY, SW, XO, NT>(
                                                h.gd, a.stage, ref_next.tile, sm + (buf ^ 1) * P::BOX,
                                                &s_bar[buf ^ 1], 0);
                                        });
                if (tid == 0) s_ref_next = ref_after;
            }
            next_tma = true;
        }
        if (!ctl.run) {
            wait_box(buf ^ 1, next_tma);
            continue;
        }

        int taken = ntiles;
        if (QUEUED && tid == 0) taken = stride + atomicAdd(tile_queue(a.grid.ctrl, a.stage), 1);
        // the box of the tile taken: its buffer was last read before the barrier that ended the previous tile
        auto start_taken = [&] {
            if (!QUEUED || tid != 0) return;
            s_next = taken;
            if (taken < ntiles) start_single(taken, buf ^ 1);
        };
        double F0[4], F1[4];  // this thread's y-pair
        if constexpr (SPLIT) {
            // ---- 3s. one face a thread: x-faces in the lower half of the
            //      threads, y-faces in the upper ------------------------------
            const bool xf = tid < NT / 2;
            const int f = xf ? tid : tid - NT / 2, w = xf ? TX + 1 : TX;
            const int r = f / w, c = f - r * w;
            if (f < (xf ? (TX + 1) * TY : TX * (TY + 1))) {
                const int st = xf ? 1 : SW;
                const double *v0 = IN + (xf ? (r + G) * SW + c + XO : r * SW + c + G + XO);
                double L[4], R[4], WL[4], WR[4], F[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const double *v = v0 + (xf || m == 0 || m == 3 ? m : 3 - m) * PL;
                    double s[2 * G];
#pragma unroll
                    for (int d = 0; d < 2 * G; ++d) s[d] = v[d * st];
                    f64::upface<ORDER>(s, L[m], R[m]);
                    WL[m] = s[G - 1];
                    WR[m] = s[G];
                }
                const int e = xf ? (r + 1) * CW + c : r * CW + c + 1, es = xf ? 1 : CW;
                f64::face_flux<RS>(L, R, WL, WR, CE[e], CE[e + es], CE[CP + e], CE[CP + e + es], gf, F);
                double *o = xf ? FX + r * FW + c : FY + r * TX + c;
                const int os = xf ? TY * FW : (TY + 1) * TX;
                o[0] = F[0];
                o[os] = xf ? F[1] : F[2];
                o[2 * os] = xf ? F[2] : F[1];
                o[3 * os] = F[3];
            }
        } else {
            // ---- 3. x-faces 2j, 2j + 1 of row r -----------------------------------
            for (int p = tid; p < XP * TY; p += NT) {
                const int r = p / XP, j = p - r * XP;
                double LA[4], RA[4], LB[4], RB[4], W0[4], W1[4], W2[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const double2 *v = reinterpret_cast<const double2 *>(IN + m * PL + (r + G) * SW + 2 * j);
                    double s[2 * G + 2];
#pragma unroll
                    for (int d = 0; d <= G; ++d) {
                        const double2 x = v[d];
                        s[2 * d] = x.x;
                        s[2 * d + 1] = x.y;
                    }
                    f64::upface<ORDER>(s + XO, LA[m], RA[m]);
                    f64::upface<ORDER>(s + XO + 1, LB[m], RB[m]);
                    W0[m] = s[XO + G - 1];
                    W1[m] = s[XO + G];
                    W2[m] = s[XO + G + 1];
                }
                const double *ce = CE + (r + 1) * CW + 2 * j;
                const double2 c01 = *reinterpret_cast<const double2 *>(ce), e01 = *reinterpret_cast<const double2 *>(ce + CP);
                const double c2 = ce[2], e2 = ce[CP + 2];
                double FA[4], FB[4];
                f64::face_pair<RS>(LA, RA, LB, RB, W0, W1, W2, c01.x, c01.y, c2, e01.x, e01.y, e2, gf, FA, FB);
                double2 *o = reinterpret_cast<double2 *>(FX + r * FW + 2 * j);
#pragma unroll
                for (int q = 0; q < 4; ++q) o[q * (TY * FW / 2)] = make_double2(FA[q], FB[q]);
            }
            start_taken();
            // ---- 4. y-faces 2k, 2k + 1 of column c (normal velocity v) ------------
            {
                const int k = tid / TX, c = tid - k * TX;
                double LA[4], RA[4], LB[4], RB[4], W0[4], W1[4], W2[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const double *v = IN + (m == 1 ? 2 : m == 2 ? 1 : m) * PL + 2 * k * SW + (c + G + XO);
                    double s[2 * G + 1];
#pragma unroll
                    for (int d = 0; d <= 2 * G; ++d) s[d] = v[d * SW];
                    f64::upface<ORDER>(s, LA[m], RA[m]);
                    f64::upface<ORDER>(s + 1, LB[m], RB[m]);
                    W0[m] = s[G - 1];
                    W1[m] = s[G];
                    W2[m] = s[G + 1];
                }
                const double *ce = CE + 2 * k * CW + c + 1;
                double FA[4], FB[4];
                f64::face_pair<RS>(LA, RA, LB, RB, W0, W1, W2, ce[0], ce[CW], ce[2 * CW], ce[CP], ce[CP + CW],
                                   ce[CP + 2 * CW], gf, FA, FB);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int s = q == 1 ? 2 : q == 2 ? 1 : q;  // Cartesian components
                    F0[q] = FA[s];
                    F1[q] = FB[s];
                    FY[(q * NK + k) * TX + c] = F0[q];
                }
            }
        }
        __syncthreads();
        if (QUEUED) {
            next = s_next;
            has_next = next_tma = next < ntiles;
        }

        if (!has_next) grid_release();
        // ---- 5. divergence, RK combination, stores: cells 2k and 2k + 1 of
        //      column c (split: one cell) -----------------------------------
        double lmax = 0.0;
        const double inv_h = gd.inv_h, dth = ctl.dt * inv_h;
        // (a lost U0 is recorded here: there may be no next tile)
        const bool u0_ok = !u0_tma || wait_bar(2);
        if (!u0_ok && gd.ctrl) gd.ctrl->status = FVB_ERR_TIMEOUT;
        const int k = tid / TX, c = tid - k * TX, i = tx0 + c;
#pragma unroll
        for (int h = 0; h < (SPLIT ? 1 : 2); ++h) {
            const int r = SPLIT ? k : 2 * k + h, j = ty0 + r;
            if (r >= TY || i >= n || j >= n || !u0_ok) continue;
            double div[4];  // h times the flux divergence
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double *fx = FX + (q * TY + r) * FW + c;
                const double *fy = FY + (q * P::NFY + k) * TX + c;
                const double dy = SPLIT ? fy[TX] - fy[0] : h == 0 ? F1[q] - F0[q] : fy[TX] - F1[q];
                div[q] = (fx[1] - fx[0]) + dy;
            }
            const int e = (r + G) * SW + (c + G + XO);
            const double rk = IN[e], uk = IN[PL + e], vk = IN[2 * PL + e], pk = IN[3 * PL + e];
            if (a.stage == 0) {
                double *rhs = (double *)a.rhs;
                const size_t n2 = (size_t)n * n, kk = (size_t)j * n + i;
#pragma unroll
                for (int q = 0; q < 4; ++q) rhs[q * n2 + kk] = -(div[q] * inv_h);
                ((double *)a.lam)[kk] = fabs(uk) + fabs(vk) + f64::snd(gf.gam * pk, rk);
                continue;
            }
            // U_k - dt div of the conserved variables, then the combination
            double cv[4] = {fma(-dth, div[0], rk), fma(-dth, div[1], rk * uk), fma(-dth, div[2], rk * vk),
                            fma(-dth, div[3], f64::energy(rk, uk, vk, pk, gf))};
            if (a.stage >= 2) {
                double w0[4];
                if (u0_tma) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) w0[q] = U0[(q * TY + r) * TX + c];
                } else {
                    const double *u0 = (const double *)gd.st[0] + gidx(gd, 0, j, i);
#pragma unroll
                    for (int q = 0; q < 4; ++q) w0[q] = u0[q * gd.plane];
                }
                const double c0[4] = {w0[0], w0[0] * w0[1], w0[0] * w0[2], f64::energy(w0[0], w0[1], w0[2], w0[3], gf)};
                const double wa = a.stage == 2 ? 0.75 : 1. / 3., wb = a.stage == 2 ? 0.25 : 2. / 3.;
#pragma unroll
                for (int q = 0; q < 4; ++q) cv[q] = fma(wa, c0[q], wb * cv[q]);
            }
            const double ir = frcp(cv[0]);
            double w[4];
            w[1] = cv[1] * ir;
            w[2] = cv[2] * ir;
            w[3] = gf.gm1 * fma(-0.5, fma(cv[1], w[1], cv[2] * w[2]), cv[3]);
            w[0] = f64::fl14(cv[0]);
            w[3] = f64::fl14(w[3]);
            put_cell<double>(gd, (double *)(a.stage == 1 ? gd.k1 : a.stage == 2 ? gd.k2 : gd.st[0]), j, i, w);
            // (a NaN is skipped, as fmax skips it)
            if (a.stage == 3) lmax = smax<double>(fabs(w[1]) + fabs(w[2]) + f64::snd(gf.gam * w[3], w[0]), lmax);
        }

        // ---- 6. max wave speed of the new state (stage 3) ------------------
        if (a.stage == 3) {
            // (a batched launch advances each grid's time where its tile 0's header is published)
            if (!BATCHED && tid == 0 && tile == 0) leader_finish<P64>(gd.ctrl);
            if (BATCHED) {
                // tiles of one CTA belong to different grids: one atomic per
                // warp and tile
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
                if ((tid & 31) == 0 && lmax > 0.0)
                    atomicMax(&gd.ctrl->lam_acc, (unsigned long long)__double_as_longlong(lmax));
            } else {
                lacc = fmax(lacc, lmax);
            }
        }
        // ---- 7. the next box: wait, then release this tile's buffers ---------
        wait_box(buf ^ 1, next_tma);
    }
    if (!BATCHED && a.stage == 3) {
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
    // a load whose wait gave up may still be in flight: wait once more
    // (bounded) so no copy into this CTA's shared memory outlives it
    if (lost && !drop && !drop_u0)
        for (int m = 0; m < 3; ++m)
            if ((lost >> m) & 1u) mbar_wait(&s_bar[m], (phase >> m) & 1u);
}

template <int ORDER, int RS, int SHAPE>
static StageKernel entry64()
{
    constexpr TileShape ts = kTileShapes64[SHAPE];
    void *batched = nullptr;
    if constexpr (ORDER == 7 && RS == 0) batched = (void *)stage64_kernel<ORDER, ts.tx, ts.ty, ts.nt, M64_BATCHED, RS>;
    // (the split form is for grids of few tiles: no queue)
    void *queued = nullptr;
    if constexpr (!L64<ORDER, ts.tx, ts.ty, ts.nt>::SPLIT)
        queued = (void *)stage64_kernel<ORDER, ts.tx, ts.ty, ts.nt, M64_QUEUED, RS>;
    return StageKernel{(void *)stage64_kernel<ORDER, ts.tx, ts.ty, ts.nt, M64_FIXED, RS>, batched,
                       L64<ORDER, ts.tx, ts.ty, ts.nt>::smem, ts.nt, queued};
}

template <int ORDER, int RS>
static StageKernel pick64(int shape)
{
    static_assert(kNumTileShapes == 7, "one entry a shape");
    switch (shape) {
    case 0: return entry64<ORDER, RS, 0>();
    case 1: return entry64<ORDER, RS, 1>();
    case 2: return entry64<ORDER, RS, 2>();
    case 3: return entry64<ORDER, RS, 3>();
    case 4: return entry64<ORDER, RS, 4>();
    case 5: return entry64<ORDER, RS, 5>();
    case 6: return entry64<ORDER, RS, 6>();
    default: return StageKernel{};
    }
}

// the kernels are built in three translation units
StageKernel stage64_up7(int shape);
StageKernel stage64_up7_rs(int shape, int rs);
StageKernel stage64_orders(int order, int shape);

}  // namespace fvb
