"""Tile edges of the single-precision kernels on the solver's own path (boxes
through tensor maps, ghost images), against the oracle: FP32 as shipped against
the FP32 oracle at the form's 2e-5, all tile variants bit for bit; FP32c against
the FP64 oracle at its 1e-6 relative L1, a variant of either kernel."""
from __future__ import annotations

import numpy as np
import pytest

import fvstuff_b200 as F
import oracle as O
from cases import pad, prim_to_cons, rel_linf, smooth

pytestmark = pytest.mark.gpu

BCS = ["reflect", "periodic", "transmissive"]


def _oracle(n, bc, dtype):
    U = pad(smooth(n, seed=n).astype(dtype), 4)
    O.bc(U, n, 4, bc)
    ref = U.copy()
    O.up_run(ref, n, 1.0 / n, 0.4, bc, 3)
    return U, ref


# below, at and one above the variants' widths (16, 32, 64) and heights (7 to 16)
@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("n", [8, 15, 33, 65])
def test_f32_tile_edges(n, bc):
    U, ref = _oracle(n, bc, np.float32)
    first = None
    for tile in range(7):
        s = F.Solver(n, precision="f32", bc=BCS[bc], tile=tile)
        s.set_state(U)
        s.step(3)
        got = s.get_state(dtype=np.float32)
        first = got if first is None else first
        assert np.array_equal(got, first), tile
    assert rel_linf(first.astype(np.float64), ref.astype(np.float64)) <= 2e-5  # the ghost ring as well


@pytest.mark.parametrize("tile", [0, 5])  # row pairs; x- with y-faces
@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("n", [8, 15, 33, 65])
def test_f32c_tile_edges_against_the_oracle(n, bc, tile):
    U, ref = _oracle(n, bc, np.float64)
    s = F.Solver(n, precision="f32c", bc=BCS[bc], tile=tile)
    s.set_state(U)
    s.step(3)
    got, want = s.get_state(layout="cons", interior=True), prim_to_cons(ref[:, 4:-4, 4:-4])
    for q in range(4):
        assert np.sum(np.abs(got[q] - want[q])) <= 1e-6 * np.sum(np.abs(want[q]))
