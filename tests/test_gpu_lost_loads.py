"""A U0 tile or a rec3 halo box that never arrives (fvb_debug_drop: the copy is
not issued, so the kernel's bounded wait of one second runs out and the kernel
ends normally) is an error of the step, on the last tile of a CTA as on any
other; the solver given a new state then advances as a fresh one."""
from __future__ import annotations

import numpy as np
import pytest

import fvstuff_b200 as F
from cases import smooth

pytestmark = pytest.mark.gpu

FVB_ERR_TIMEOUT = 7


# 96^2 and 64^2: one tile a CTA, so the lost load is that of its last tile;
# 601^2 (variant 0) and rec3's 400^2: several, taken from the stage's counter
@pytest.mark.parametrize("flux,n,tile,load", [
    ("up_ducros", 96, 0, "u0"), ("up_ducros", 96, 3, "u0"), ("up_ducros", 601, 0, "u0"), ("up_ducros", 96, 0, "box"),
    ("rec3", 64, -1, "u0"), ("rec3", 64, -1, "box"), ("rec3", 400, -1, "u0"), ("rec3", 400, -1, "box")])
def test_a_lost_load_is_reported(flux, n, tile, load):
    w = smooth(n, seed=n)
    out = []
    for lost in (True, False):
        s = F.Solver(n, flux=flux, bc="periodic", tile=tile)
        s.set_state(w, interior=True)
        if lost:
            s.debug_drop(load)
            s.step(1)
            assert s.sync().status == FVB_ERR_TIMEOUT
            s.step(2)
            assert s.sync().status == FVB_ERR_TIMEOUT  # it stays stopped
            s.set_state(w, interior=True)
        s.step(3)
        st = s.sync()
        assert st.status == 0 and st.steps == 3
        out.append(s.get_state())
    assert np.array_equal(out[0], out[1])


def test_loads_a_form_does_not_make_are_refused():
    for kw, load in ((dict(flux="keep"), "box"), (dict(flux="up_hllc_d2av"), "box"), (dict(precision="f32c"), "u0"),
                     (dict(precision="f32"), "u0"), (dict(order=9), "u0")):
        s = F.Solver(32, tile=0, **kw)
        with pytest.raises(F.FvbError):
            s.debug_drop(load)
    with pytest.raises(F.FvbError):
        F.Solver(32, flux="rec3", bc="periodic").debug_drop_load()
