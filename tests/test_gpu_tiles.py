"""Where the tiled kernels can go wrong: grids one cell around a tile's edge,
smaller than a tile, with a last tile of one row, and just above two waves of
CTAs, where a stage's tiles are taken from its counter instead of in fixed
shares (so the counters are cleared and counted again over several steps).
Against the oracle at the bars of the form's own parity tests; variants of one
form, which share their face arithmetic, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import fvstuff_b200 as F
import oracle as O
from cases import kh, pad, prim_to_cons, rel_linf, smooth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _up64(n, bc, steps, tile, order=7):
    g = (order + 1) // 2
    U = pad(smooth(n, seed=n), g)
    O.bc(U, n, g, bc)
    s = F.Solver(n, order=order, bc=["reflect", "periodic", "transmissive"][bc], tile=tile)
    s.set_state(U)
    s.step(steps)
    assert s.sync().steps == steps
    return U, s.get_state()


# widths 16, 32, 64 and heights 3, 7, 15 (variants: 32x15, 32x7, 64x7, 16x7 split,
# 16x7, 32x7 split, 16x3 split)
@pytest.mark.parametrize("tile", range(7))
@pytest.mark.parametrize("n,bc,order", [(8, 0, 7), (15, 1, 7), (16, 2, 5), (33, 0, 7), (61, 1, 9), (65, 2, 3)])
def test_f64_tile_edges(tile, n, bc, order):
    U, got = _up64(n, bc, 3, tile, order)
    g = (order + 1) // 2
    ref = U.copy()
    O.up_run(ref, n, 1.0 / n, 0.4, bc, 3, order=order)
    inner = slice(g, g + n)
    assert rel_linf(prim_to_cons(got[:, inner, inner]), prim_to_cons(ref[:, inner, inner])) <= 1e-12
    assert rel_linf(got, ref) <= 1e-12  # the ghost ring as well


def test_f64_taken_tiles_equal_fixed_shares():
    """601^2: 779 tiles of 32x15 against 592 in two waves; the split variant
    always runs fixed shares"""
    _, taken = _up64(601, 1, 4, 0)
    _, fixed = _up64(601, 1, 4, 3)
    assert np.array_equal(taken, fixed)


# variants 0, 2, 4, 6: row pairs of 30, 14 and 22 rows; 3: 16x15 and 5: 32x16 pair x- with y-faces
@pytest.mark.parametrize("tile", [0, 1, 2, 3, 4, 6])
@pytest.mark.parametrize("n,bc", [(8, "reflect"), (15, "periodic"), (16, "transmissive"), (31, "reflect"),
                                  (45, "periodic"), (67, "transmissive")])
def test_f32c_tile_edges(tile, n, bc):
    w = smooth(n, seed=n)
    out = []
    for t in (5, tile):
        s = F.Solver(n, precision="f32c", bc=bc, tile=t)
        s.set_state(w, interior=True)
        s.step(3)
        out.append(s.get_state())
    assert np.array_equal(out[0], out[1])


def test_f32c_taken_tiles_equal_fixed_shares():
    """781^2: 675 row-pair tiles of 32x30 against 592 in two waves; a step
    skipped at the stop time copies the state through the same tiles"""
    out = []
    for t in (0, 5):
        s = F.Solver(781, precision="f32c", bc="periodic", tile=t)
        s.set_state(kh(781), interior=True)
        s.step(5)
        s.step(3, s.sync().t)  # stopped: every stage copies
        s.step(2)
        out.append(s.get_state())
    assert np.array_equal(out[0], out[1])


# the residual's tile rule changes above 119 / 360 (FP64) and 315 (FP32) on 148 SMs; odd n: 8-byte rows
@pytest.mark.parametrize("n,dtype,tol", [(119, np.float64, 1e-13), (128, np.float64, 1e-13), (360, np.float64, 1e-13),
                                         (361, np.float64, 1e-13), (315, np.float32, 2e-5), (321, np.float32, 2e-5)])
def test_up_rhs_tile_rule(n, dtype, tol):
    U = pad(smooth(n, seed=n).astype(dtype), 4)
    O.bc(U, n, 4, 0)
    Qd = torch.from_numpy(U).cuda()
    rhs = torch.empty((4, n, n), dtype=Qd.dtype, device="cuda")
    lam = torch.empty((n, n), dtype=Qd.dtype, device="cuda")
    F.up_rhs(Qd, rhs, lam, n, n + 8, 1.0 / n)
    torch.cuda.synchronize()
    R, l = O.up_rhs(U, n, 1.0 / n)
    assert rel_linf(rhs.cpu().numpy(), R) <= tol
    assert rel_linf(lam.cpu().numpy()[None], l[None]) <= tol


@pytest.mark.parametrize("n", [15, 31, 33, 46])
def test_keep_tile_edges(n):
    U = O.keep_ic(n, 1.0 / n, False)
    O.bc(U, n, 2, 1)
    s = F.Solver(n, flux="keep", bc="periodic", cfl=0.2)
    s.set_state(U, layout="cons")
    s.step(2)
    ref = U.copy()
    O.keep_run(ref, n, 1.0 / n, 0.2, 2)
    assert rel_linf(s.get_state(layout="cons")[:, 2:-2, 2:-2], ref[:, 2:-2, 2:-2]) <= 1e-12


# 32x14 tiles; 400^2: 377 tiles against 296 CTAs
@pytest.mark.parametrize("n,steps", [(14, 6), (30, 6), (34, 6), (400, 3)])
def test_rec3_tile_edges_and_taken_tiles(n, steps):
    U = O.rec3_ic(n, 1.0 / n, "sod", 0.0)
    O.rec3_limit(U, n)
    O.bc(U, n, 2, 1)
    s = F.Solver(n, flux="rec3", bc="periodic", cfl=0.4)
    s.set_state(U, layout="cons")
    s.step(steps)
    ref = U.copy()
    O.rec3_run(ref, n, 1.0 / n, 0.4, steps)
    assert rel_linf(s.get_state(layout="cons")[:, 2:-2, 2:-2], ref[:, 2:-2, 2:-2]) <= 1e-13


# 32x8 tiles; 600^2: 1425 tiles, more than two waves at up to four CTAs an SM
@pytest.mark.parametrize("n,order,steps", [(9, 5, 4), (31, 7, 4), (33, 9, 4), (600, 5, 2)])
def test_d2av_tile_edges_and_taken_tiles(n, order, steps):
    g = O.d2av_ghost(order)
    U = O.d2av_ic_sod(n, 1.0 / n, order)
    O.bc(U, n, g, 0)
    s = F.Solver(n, order=order, flux="up_hllc_d2av", bc="reflect", cfl=0.4)
    s.set_state(U[:, g:-g, g:-g].copy(), layout="cons", interior=True)
    s.step(steps)
    ref = U.copy()
    O.d2av_run(ref, n, 1.0 / n, 0.4, 0, steps, 1e30, order, 0.5, 0.0, 0.05)
    assert rel_linf(s.get_state(layout="cons", interior=True), ref[:, g:-g, g:-g]) <= 1e-13


@pytest.mark.parametrize("precision,n", [("f64", 601), ("f32c", 781)])
def test_taken_tiles_after_a_lost_load(precision, n):
    """A stage that stops early (its first load is not issued, so the bounded
    wait runs out) leaves tiles untaken; the stages after it clear its counter,
    so the solver given a new state advances as a fresh one."""
    w = smooth(n, seed=n)
    out = []
    for lost in (True, False):
        s = F.Solver(n, precision=precision, bc="periodic", tile=0)
        s.set_state(w, interior=True)
        if lost:
            s.debug_drop_load()
            s.step(1)
            assert s.sync().status != 0
            s.set_state(w, interior=True)
        s.step(3)
        assert s.sync().steps == 3
        out.append(s.get_state())
    assert np.array_equal(out[0], out[1])
