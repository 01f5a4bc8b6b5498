// fvb_tune.cpp -- choice of the stage-kernel tile variant (halo-tile shape
// and threads per tile) by measurement.
//
// On first use for a (device, precision, order, grid-size class) the tuner
// builds a scratch grid of a representative size (the grid's own size, at
// most 2048^2), fills it with a smooth state, and times a few SSP-RK3 steps
// of every tile variant that can be resident on the device with CUDA
// events; the fastest wins and is cached for the process.  FVB_TILE=<k>
// forces variant k; FVB_AUTOTUNE=0 selects variant 0 without measuring;
// FVB_AUTOTUNE_LOG=1 prints each variant's time and the choice to stderr.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <tuple>

#include "fvb_host.h"

namespace fvb {
namespace {

std::mutex g_mu;
std::map<std::tuple<int, int, int, int>, int> g_cache;

// <=64, <=96, <=128, <=192, ... <=1024, larger: below about 512^2 cells the
// choice turns on how the tiles fill the SMs, which changes within a factor
// of two in n
int size_class(int n)
{
    int c = 0;
    for (int m = 64; m < n && c < 9; ++c) m = c & 1 ? m / 3 * 4 : m / 2 * 3;
    return c;
}

// time `steps` steps of variant `shape` on a scratch grid; < 0 on failure
float time_shape(int prec, int order, int n, int shape, cudaStream_t s)
{
    const int g = (order + 1) / 2;
    Geometry G = make_geometry(n, g, prec == P64 ? FVB_PREC_F64 : prec == P32 ? FVB_PREC_F32 : FVB_PREC_F32C);
    const size_t ctrl_off = (G.bytes + 255) / 256 * 256, map_off = ctrl_off + 256;
    const size_t stage_bytes = (size_t)4 * n * n * sizeof(double);
    void *block = nullptr, *stage = nullptr;
    if (cudaMalloc(&block, map_off + TM_COUNT * sizeof(CUtensorMap)) != cudaSuccess) return -1.f;
    if (cudaMalloc(&stage, stage_bytes) != cudaSuccess) { cudaFree(block); return -1.f; }
    float ms = -1.f;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    do {
        GridDev gd{};
        grid_pointers(gd, block, G, prec == P64 ? FVB_PREC_F64 : prec == P32 ? FVB_PREC_F32 : FVB_PREC_F32C);
        gd.bcx = gd.bcy = FVB_BC_PERIODIC;
        set_scales(gd, 1.0 / n, 1.4);
        gd.ctrl = (Ctrl *)((char *)block + ctrl_off);
        int tiles;
        tile_dims(prec, shape, n, gd.tiles_x, tiles);
        CUtensorMap maps[TM_COUNT];
        gd.tmap = nullptr;
        if (encode_tile_maps(gd, prec, order, shape, maps)) {
            CUtensorMap *dm = (CUtensorMap *)((char *)block + map_off);
            if (cudaMemcpy(dm, maps, sizeof maps, cudaMemcpyHostToDevice) != cudaSuccess) break;
            gd.tmap = dm;
        }
        fvb_case c;
        case_defaults(&c, FVB_CASE_KH, 0.0, 0.0, 1.0);
        const int internal = prec_internal(prec == P64 ? FVB_PREC_F64 : prec == P32 ? FVB_PREC_F32 : FVB_PREC_F32C);
        ExtView ev{1, g, n + 2 * g, FVB_LAYOUT_PRIM, FVB_F64};
        BufView v = view_of(gd);
        // (the step control too: its tile counters and its lost-load flag are
        // read by the first launches and set by nothing before them)
        if (cudaMemsetAsync(block, 0, ctrl_off + sizeof(Ctrl), s) != cudaSuccess) break;
        if (init_case_prim64((double *)stage, n, 0.0, 0.0, gd.h, 1.4, c, s) != cudaSuccess) break;
        if (import_state(stage, ev, gd.st[0], gd.lo[0], v, internal, 1.4, s) != cudaSuccess) break;
        cudaError_t e = internal == INT_PRIM64 ? bc_fill<double>((double *)gd.st[0], v, 1, 1, s)
                                               : bc_fill<float>((float *)gd.st[0], v, 1, 1, s);
        if (e == cudaSuccess && internal == INT_CONS_HILO) e = bc_fill<float>((float *)gd.lo[0], v, 1, 1, s);
        if (e == cudaSuccess) e = lam_into(gd.st[0], v, internal, 1.4, &gd.ctrl->lam_acc, s);
        if (e == cudaSuccess) e = ctrl_set(gd.ctrl, 1e300, 1, 0.0, 0.4, gd.h, s);
        if (e != cudaSuccess) break;
        int per_sm = stage_max_ctas_per_sm(prec, order, shape), sms = 0, dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (per_sm <= 0) break;
        const int ctas = tiles < per_sm * sms ? tiles : per_sm * sms;
        StageArgs a{};
        a.grid = gd;
        a.ntiles_static = tiles;
        auto run = [&](int steps) {
            int parity = 0;
            for (int k = 0; k < steps; ++k) {
                for (int stage = 1; stage <= 3; ++stage) {
                    a.stage = stage;
                    a.parity = parity;
                    if (launch_stage(prec, order, shape, a, ctas, s) != cudaSuccess) return false;
                }
                if (prec == P32C) parity ^= 1;
            }
            return true;
        };
        if (!run(2)) break;  // warm-up (even: F32C ends on its start buffer)
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        // the best of three timings of four steps: variants differ by a few
        // per cent, about the run-to-run spread of a single timing
        bool ok = true;
        for (int rep = 0; rep < 3 && ok; ++rep) {
            cudaEventRecord(e0, s);
            ok = run(4);
            cudaEventRecord(e1, s);
            float t = -1.f;
            if (ok && cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&t, e0, e1) == cudaSuccess)
                ms = (ms < 0.f || t < ms) ? t : ms;
            else
                ok = false;
        }
        if (!ok) ms = -1.f;
    } while (0);
    cudaStreamSynchronize(s);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(stage);
    cudaFree(block);
    cudaGetLastError();  // a failed variant must not poison later calls
    return ms;
}

}  // namespace

// FVB_TILE's variant, FVB_AUTOTUNE=0's, or -1
static int forced_shape()
{
    if (const char *f = std::getenv("FVB_TILE")) {
        const int k = std::atoi(f);
        if (k >= 0 && k < kNumTileShapes) return k;
    }
    const char *a = std::getenv("FVB_AUTOTUNE");
    return a && a[0] == '0' ? 0 : -1;
}

// Tile variant of a batch, fixed before its grids are known.  FP32c: 32 x 16
// (three CTAs an SM): grids of 64 ... 512 cells a side fill its 16 rows better
// than the 30 of the row-pair tile that wins on one large grid.  us a stage on
// B200, 32 x 16 against 32 x 30: 24 grids of 64-128 15 / 17, 32 of 100-200
// 35 / 38, 64 of 64-256 74 / 82, 32 of 64-512 111 / 110, 128 of 64-512
// 415 / 409.  FP64: as one large grid (32 x 15 was best on all of these).
int batch_shape(int prec)
{
    const int f = forced_shape();
    return f >= 0 ? f : prec == P32C ? 5 : autotune_shape(prec, 7, 4096);
}

int autotune_shape(int prec, int order, int n)
{
    const int forced = forced_shape();
    if (forced >= 0) return forced;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(dev, prec, order, size_class(n));
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_cache.find(key);
    if (it != g_cache.end()) return it->second;
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return 0;
    const int nt = n < 2048 ? (n < 16 ? 16 : n) : 2048;
    int best = 0;
    float best_ms = -1.f;
    const bool log = std::getenv("FVB_AUTOTUNE_LOG") != nullptr;
    for (int shape = 0; shape < kNumTileShapes; ++shape) {
        float ms = time_shape(prec, order, nt, shape, s);
        if (log)
            std::fprintf(stderr, "fvb autotune: precision %d order %d n %d: tile %d (%dx%d, %d threads) %.4f ms\n",
                         prec, order, nt, shape, tile_shape(prec, shape).tx, tile_shape(prec, shape).ty,
                         tile_shape(prec, shape).nt, ms);
        if (ms > 0 && (best_ms < 0 || ms < best_ms)) {
            best_ms = ms;
            best = shape;
        }
    }
    if (log) std::fprintf(stderr, "fvb autotune: -> tile %d\n", best);
    cudaStreamDestroy(s);
    g_cache[key] = best;
    return best;
}

}  // namespace fvb
