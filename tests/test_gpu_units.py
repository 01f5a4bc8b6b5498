"""States in units in which a sound speed is far from one (velocities V times,
pressures V^2 times those of an order-one state; dt follows through h).  The
schemes have no scale of their own above their floors, so each form holds at
every V the bar it holds at one: FP64 1e-12 of the oracle, FP32c 1e-6 relative
L1 of FP64.  Mean flows of Mach 0 and about 4 (2.5 along each axis), so that
every face's fan is subsonic or supersonic, to either side.

UP9 is left out: its published left-biased weights sum to 4217/2520, so in a
mean flow to the right the scheme itself turns one ulp of the input into 2e-11
within these four steps, at V = 1 as at 1e7."""
from __future__ import annotations

import numpy as np
import pytest

import fvstuff_b200 as F
import oracle as O
from cases import pad, prim_to_cons, rel_linf, smooth

pytestmark = pytest.mark.gpu

N, STEPS = 48, 4


def _state(V, mean):
    w = smooth(N, seed=7)
    w[1] += mean
    w[2] -= mean
    return w * np.array([1.0, V, V, V * V])[:, None, None]


def _run(w, **kw):
    s = F.Solver(N, bc="periodic", tile=0, **kw)
    s.set_state(w, interior=True)
    s.step(STEPS)
    assert s.sync().steps == STEPS
    return s


@pytest.mark.parametrize("V", [1.0, 1e3, 1e5, 1e7])
@pytest.mark.parametrize("mean", [0.0, 3.0])
@pytest.mark.parametrize("riemann,order", [("hllc", 3), ("hllc", 5), ("hllc", 7), ("hll", 7), ("roe", 7)])
def test_f64_against_the_oracle(V, mean, riemann, order):
    w = _state(V, mean)
    s = _run(w, order=order, flux="up_ducros" + ("" if riemann == "hllc" else "_" + riemann))
    g = s.g
    ref = pad(w, g)
    O.bc(ref, N, g, 1)
    O.up_run(ref, N, 1.0 / N, 0.4, 1, STEPS, order=order, riemann=riemann)
    got = s.get_state(interior=True)
    assert rel_linf(prim_to_cons(got), prim_to_cons(ref[:, g:-g, g:-g])) <= 1e-12


@pytest.mark.parametrize("V", [1.0, 1e3, 1e5, 1e7])
@pytest.mark.parametrize("mean", [0.0, 3.0])
def test_f32c_against_f64(V, mean):
    w = _state(V, mean)
    a, b = (_run(w, precision=p).get_state(layout="cons", interior=True) for p in ("f32c", "f64"))
    for q in range(4):
        assert np.sum(np.abs(a[q] - b[q])) <= 1e-6 * np.sum(np.abs(b[q]))


@pytest.mark.parametrize("tile", [0, 3])
def test_f64_just_above_the_floors(tile):
    """A resting gas whose pressure, or whose squared sound speed, is 5e-7 of
    itself above the floor of 1e-14 stays what it is, and is not taken for the
    floor.  (Each step rounds p / (gamma - 1) and back: a few ulp.)"""
    over = 1e-14 * (1 + 5e-7)
    for rho, p in ((1.0, over), (1.4, over)):  # the second: c^2 = 1.4 p / rho = over
        w = np.stack([np.full((N, N), x) for x in (rho, 0.0, 0.0, p)])
        s = F.Solver(N, bc="periodic", tile=tile)
        s.set_state(w, interior=True)
        s.step(3)
        got, st = s.get_state(interior=True), s.sync()
        assert st.steps == 3
        assert np.max(np.abs(got[3] - p)) <= 1e-14 * p
        assert abs(st.lam_max - np.sqrt(1.4 * p / rho)) <= 1e-14 * st.lam_max
