// fvb_internal.h -- device-side data structures shared by the kernels and
// the host library.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fvb.h"

namespace fvb {

// Device-resident step control of one grid.  The stage kernels read and
// update it themselves, so a run of steps needs no host round trip:
//   stage 1 : every CTA derives dt from lam_acc (max wave speed of the
//             current state), t and t_stop, identically; the CTA holding
//             tile 0 ("leader") publishes dt / active
//   stage 2 : leader clears lam_acc
//   stage 3 : every CTA max-reduces lam of the new state into lam_acc;
//             leader advances t and step
// Fields a stage writes are never read by another CTA of the same stage.
struct Ctrl {
    double t;                   // simulated time (always FP64)
    double t_stop;              // steps stop when t >= t_stop
    double dt;                  // dt of the step in progress
    double cfl, h;              // dt = cfl * h / lam
    unsigned long long lam_acc; // bit pattern of max lam (non-negative double)
    unsigned long long lam_cur; // lam_acc that set the current dt
    long long step;
    int active;                 // the step in progress runs
    int status;                 // fvb_status of the step control
    int clamped;                // dt was clamped to land on t_stop
    int drop_load;              // failure-injection hook (fvb_debug_drop): CTA 0 of the next
                                // single-grid stage that makes that load does not issue it
                                // (its wait must run out)
    unsigned long long aux;     // KEEP: bit pattern of the entropy-distance max of stage 1's
                                // input; rec3: count of 2x2 blocks given the brutal mean fix
    unsigned long long aux23[2];  // KEEP: the same of stages 2 and 3; else: tile counters of the stages (tile_queue)
};

// Device view of one grid.  Element (q, jp, ip) of a padded buffer, padded
// coordinates jp, ip in [0, n + 2g), sits at q*plane + jp*pitch + xoff + ip.
// The IDX_P layout of the reference is pitch = n + 2g, xoff = 0,
// plane = pitch * (n + 2g).
struct GridDev {
    int n, g;
    int pitch, xoff;
    long long plane;
    int bcx, bcy;
    double h, gam;
    double inv_h, igm1;  // 1 / h, 1 / (gam - 1)
    void *st[2];    // state: prim (F64/F32, st[0] only) or conserved hi (F32C, ping-pong)
    void *lo[2];    // F32C: lo words of the conserved state; KEEP: lo[0] holds the cells' entropies
    void *k1, *k2;  // stage outputs: U1/U2 primitives (F64/F32) or increments d1/d2 (F32C)
    Ctrl *ctrl;
    const CUtensorMap *tmap;  // TMA descriptors of st[0], st[1], k1, k2 for the kernel's halo
                              // box and of st[0] for a tile (device memory); null: plain loads
    int tiles_x;    // tiles along x for the kernel's tile width
    int pad;
};

inline void set_scales(GridDev &gd, double h, double gam)
{
    gd.h = h;
    gd.gam = gam;
    gd.inv_h = 1.0 / h;
    gd.igm1 = 1.0 / (gam - 1.0);
}

// TM_U0: the FP64 kernel's U0 tile (no halo) of st[0]
enum { TM_ST0 = 0, TM_ST1 = 1, TM_K1 = 2, TM_K2 = 3, TM_U0 = 4, TM_COUNT = 5 };

// Tile-table entry of the batched launch: grid index and tile index.
struct TileRef {
    int grid;
    int tile;
};

enum Prec { P64 = 0, P32 = 1, P32C = 2 };

// Step control of one grid for one RK stage: the dt the stage uses, whether
// its tiles compute, and (FP32c stage 3 of a grid that stopped) whether they
// carry the state to the other buffer.
struct TileCtl {
    double dt;
    int run;
    int copy;
};

struct StageArgs {
    GridDev grid;              // single-grid launches
    const GridDev *grids;      // batched launches: grid descriptors
    Ctrl *ctrls;               // batched launches: step control of each grid (indexed like grids)
    const TileRef *tiles;      // batched launches: tile table
    const int *ntiles;         // batched launches: live tile count (device)
    int ntiles_static;         // single-grid launches: tiles
    int stage;                 // 1, 2, 3; 0 = residual only (reference contract)
    int parity;                // F32C: index of the current state buffer
    void *rhs, *lam;           // stage 0 outputs, (4, n, n) and (n, n) unpadded
};

// Tile shapes the stage kernel is instantiated for (tile width x height,
// threads per CTA).  Chosen so the face count (TX+1)TY + TX(TY+1) is close
// to a multiple of the thread count.
struct TileShape {
    int tx, ty, nt;
};
constexpr int kNumTileShapes = 7;
constexpr TileShape kTileShapes[kNumTileShapes] = {
    {32, 15, 256}, {32, 7, 128}, {64, 7, 256}, {16, 15, 256}, {32, 9, 256}, {32, 16, 256}, {32, 14, 256}};
// the FP64 kernel's shapes of the same variant numbers (fvb_stage64.cuh): pairs
// of faces and of cells a thread, NT = TX (TY + 1) / 2, or the split form, one
// face a thread, NT = 2 TX (TY + 1)
constexpr TileShape kTileShapes64[kNumTileShapes] = {
    {32, 15, 256}, {32, 7, 128}, {64, 7, 256}, {16, 7, 256}, {16, 7, 64}, {32, 7, 512}, {16, 3, 128}};
// the FP32-compensated kernels' (fvb_stage32c.cu): row pairs where the height
// is even and NT = TX (TY / 2 + 1) / 2, else an x-face and a y-face a thread
constexpr TileShape kTileShapes32c[kNumTileShapes] = {
    {32, 30, 256}, {32, 7, 128}, {64, 14, 256}, {16, 15, 256}, {32, 14, 128}, {32, 16, 256}, {32, 22, 192}};
constexpr bool row_pairs(const TileShape &t) { return t.ty % 4 == 2 && t.nt == t.tx * (t.ty / 2 + 1) / 2; }
constexpr const TileShape &tile_shape(int prec, int shape)
{
    return prec == P64 ? kTileShapes64[shape] : prec == P32C ? kTileShapes32c[shape] : kTileShapes[shape];
}

// TMA descriptors (fvb_stage.cu): encode the TM_COUNT maps of a grid for
// a tile shape into host memory; false if this grid cannot use TMA
bool encode_tile_maps(const GridDev &gd, int prec, int order, int shape, CUtensorMap out[TM_COUNT]);
// the same for the kernels of BoxPipe (fvb_tma.cuh) with tx x ty tiles
bool encode_family_maps(const GridDev &gd, int tx, int ty, CUtensorMap out[TM_COUNT]);
// stream-ordered copy of encoded maps into device memory (dst 64-byte aligned)
cudaError_t put_tile_maps(const CUtensorMap maps[TM_COUNT], CUtensorMap *dst, cudaStream_t s);

// a stage kernel as launched: for one grid, for a tile table (null where the
// batched form is not built), its dynamic shared memory and threads
struct StageKernel {
    void *fn, *fn_batched;
    size_t smem;
    int nt;
    void *fn_queued = nullptr;  // single grids on tensor maps, tiles taken as CTAs come free
};
// the FP64 stage kernel of an order, a tile variant and a solver on the
// reconstructed states (fvb_stage64.cuh); fn null: not built
StageKernel stage64_kernel_of(int order, int shape, int rs);

// the FP32-compensated stage kernel of a tile variant (fvb_stage32c.cu)
StageKernel stage32c_kernel_of(int shape);

// launchers (fvb_stage.cu).  rs: the solver on the reconstructed states of
// the FP64 UP7 kernel -- 0 HLLC, 1 HLL, 2 Roe
cudaError_t launch_stage(int prec, int order, int shape, const StageArgs &a, int grid_ctas,
                         cudaStream_t s, int rs = 0);
int stage_max_ctas_per_sm(int prec, int order, int shape, int rs = 0);

// What a persistent launch of kernel `fn` with `threads` threads and `smem`
// bytes of dynamic shared memory needs on the current device: the shared-
// memory opt-in is applied and the resident CTAs per SM and the SM count
// are read once per (kernel, device, threads, smem), under a lock, so
// solvers on several host threads or devices set it up safely
// (fvb_stage.cu).  An error if not even one CTA fits on an SM.
struct LaunchFacts {
    int ctas_per_sm;
    int sms;
};
// a launch whose CTAs may start, up to their grid_dependency(), while the
// kernel before it in the stream ends (fvb_stage.cu)
cudaError_t launch_chained(const void *fn, int ctas, int threads, size_t smem, cudaStream_t s, void **args);
cudaError_t launch_facts(const void *fn, int threads, size_t smem, LaunchFacts &out);

}  // namespace fvb
