"""The tile tuner's host code (fvb_tune.cpp) built against a stand-in for the
CUDA runtime, whose allocations come back full of old bytes as a device's do:
every stage launch of a variant's timing must find a cleared step control
(no tile counted as taken, no lost load asked for).  No GPU needed."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

STAND_IN = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "fvb_host.h"
static int g_launches = 0, g_dirty = 0;
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) { *p = std::malloc(n); std::memset(*p, 0xa5, n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { *t = 1.f; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
}
namespace fvb {
int prec_internal(int p) { return p; }
Geometry make_geometry(int n, int g, int)
{
    Geometry G{};
    G.n = n; G.g = g; G.np = n + 2 * g; G.pitch = n + 32; G.xoff = 16 - g;
    G.plane = (long long)G.pitch * G.np; G.elem = 8; G.nbuf = 3;
    G.bytes = 96 * (size_t)G.plane;
    return G;
}
void grid_pointers(GridDev &gd, void *p, const Geometry &G, int)
{
    gd.n = G.n; gd.g = G.g; gd.pitch = G.pitch; gd.plane = G.plane;
    gd.st[0] = gd.st[1] = gd.lo[0] = gd.lo[1] = gd.k1 = gd.k2 = p;
}
BufView view_of(const GridDev &) { return BufView{}; }
void tile_dims(int prec, int shape, int n, int &tx, int &t)
{
    const TileShape &s = tile_shape(prec, shape);
    tx = (n + s.tx - 1) / s.tx;
    t = tx * ((n + s.ty - 1) / s.ty);
}
void case_defaults(fvb_case *, int, double, double, double) {}
bool encode_tile_maps(const GridDev &, int, int, int, CUtensorMap *) { return true; }
cudaError_t init_case_prim64(double *, int, double, double, double, double, const fvb_case &, cudaStream_t) { return cudaSuccess; }
cudaError_t import_state(const void *, const ExtView &, void *, void *, const BufView &, int, double, cudaStream_t) { return cudaSuccess; }
template <class R> cudaError_t bc_fill(R *, const BufView &, int, int, cudaStream_t) { return cudaSuccess; }
template cudaError_t bc_fill<double>(double *, const BufView &, int, int, cudaStream_t);
template cudaError_t bc_fill<float>(float *, const BufView &, int, int, cudaStream_t);
cudaError_t lam_into(const void *, const BufView &, int, double, unsigned long long *acc, cudaStream_t) { *acc = 1; return cudaSuccess; }
cudaError_t ctrl_set(Ctrl *c, double ts, int, double t0, double cfl, double h, cudaStream_t)
{
    c->t = t0; c->dt = 0; c->step = 0; c->status = c->active = c->clamped = 0; c->cfl = cfl; c->h = h; c->t_stop = ts;
    return cudaSuccess;
}
int stage_max_ctas_per_sm(int, int, int, int) { return 2; }
cudaError_t launch_stage(int, int, int, const StageArgs &a, int, cudaStream_t, int)
{
    const Ctrl &c = *a.grid.ctrl;
    ++g_launches;
    g_dirty += c.aux23[0] != 0 || c.aux23[1] != 0 || c.drop_load != 0;
    return cudaSuccess;
}
}
int main(int argc, char **argv)
{
    const int prec = std::atoi(argv[1]), n = std::atoi(argv[2]);  // n 0: a batch
    const int shape = n ? fvb::autotune_shape(prec, 7, n) : fvb::batch_shape(prec);
    std::printf("%d %d %d\n", shape, g_launches, g_dirty);
    return 0;
}
"""


@pytest.fixture(scope="module")
def tuner(tmp_path_factory):
    d = tmp_path_factory.mktemp("tuner")
    src, exe = d / "stand_in.cpp", d / "tuner"
    src.write_text(STAND_IN)
    csrc = ROOT / "fvstuff_b200" / "csrc"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CUDA), "-I", str(ROOT / "include"), "-I", str(csrc),
                    "-o", str(exe), str(src), str(csrc / "fvb_tune.cpp"), "-ldl"], check=True)

    def run(prec, n, **env):
        base = {k: v for k, v in os.environ.items() if not k.startswith("FVB_")}
        out = subprocess.run([str(exe), str(prec), str(n)], env={**base, **env}, capture_output=True, text=True,
                             check=True).stdout
        return [int(x) for x in out.split()]

    return run


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_timed_launches_find_a_cleared_step_control(tuner, prec):
    _, launches, dirty = tuner(prec, 640)
    assert launches == 7 * (2 + 3 * 4) * 3  # variants x (warm-up + timed steps) x stages
    assert dirty == 0


@pytest.mark.parametrize("n", [0, 640])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_knobs_hold_for_grids_and_batches(tuner, prec, n):
    assert tuner(prec, n, FVB_AUTOTUNE="0") == [0, 0, 0]
    assert tuner(prec, n, FVB_AUTOTUNE="0", FVB_TILE="3") == [3, 0, 0]
    assert tuner(prec, n, FVB_TILE="4") == [4, 0, 0]


def test_an_fp32c_batch_is_not_timed(tuner):
    assert tuner(2, 0) == [5, 0, 0]
