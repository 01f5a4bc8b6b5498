"""Quotients from shared reciprocals on the device against plain division:
through fvb_rk3_stage, whose stage 1 with a resting U0 returns
(dt L) / rho as the new velocity, over the operands of the whole FP64 range,
and through the families that reproduce their reference operation for
operation, on momenta so small that remainders, squares or the quotients
themselves underflow (the oracle divides)."""
from __future__ import annotations

import numpy as np
import pytest

import fvstuff_b200 as F
import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N, G = 256, 4


def _quotients(a, b):
    pad = lambda x, fill: np.pad(x, G, constant_values=fill)
    zero = pad(np.copysign(0.0, a), 0.0)  # rho * 0 + a keeps the sign of a zero a
    U0 = np.stack([pad(b, 1.0), zero, zero, pad(np.ones_like(b), 1.0)])
    L = np.stack([np.zeros_like(a), a, a, np.zeros_like(a)])
    Uo = torch.empty((4, N + 2 * G, N + 2 * G), dtype=torch.float64, device="cuda")
    F.rk3_stage(1, Uo, torch.from_numpy(U0).cuda(), None, torch.from_numpy(L).cuda(), 1.0, N, N + 2 * G)
    return Uo.cpu().numpy()[1:3, G:-G, G:-G]


def _operands(name):
    r = np.random.default_rng(5)
    mag = lambda lo, hi: np.ldexp(r.uniform(1, 2, (N, N)), r.integers(lo, hi, (N, N)))
    sign = lambda x: np.where(r.random((N, N)) < 0.5, -x, x)
    ones = np.ldexp(1.0 - 2.0 ** -53, r.integers(-300, 200, (N, N)))  # all significand bits set
    return {"ordinary": lambda: (sign(mag(-60, 60)), mag(-60, 60)),
            "tiny": lambda: (sign(mag(-1074, -700)), mag(-40, 40)),
            "subnormal": lambda: (sign(r.integers(1, 1000, (N, N)) * 5e-324), mag(-3, 3)),
            "zeros": lambda: (sign(np.zeros((N, N))), mag(-500, 230)),
            "whole range": lambda: (sign(mag(-1074, 1023)), mag(-1000, 1000)),
            "all ones": lambda: (sign(np.ldexp(r.integers(1, 9, (N, N)) * 1.0, r.integers(-300, 300, (N, N)))), ones)}[name]()


@pytest.mark.parametrize("name", ["ordinary", "tiny", "subnormal", "zeros", "whole range", "all ones"])
def test_rk3_velocities_are_plain_quotients(name):
    a, b = _operands(name)
    with np.errstate(all="ignore"):
        want = a / b
    for got in _quotients(a, b):
        assert np.array_equal(np.ascontiguousarray(got).view(np.int64), want.view(np.int64))


@pytest.mark.parametrize("scale", [1e-80, 1e-160, 1e-240, 1e-300, 1e-318])
@pytest.mark.parametrize("order", [3, 5, 7, 9])
def test_d2av_small_momenta_equal_the_oracle(order, scale):
    n, g = 40, O.d2av_ghost(order)
    r = np.random.default_rng(order)
    U = np.zeros((4, n + 2 * g, n + 2 * g))
    U[0], U[3] = 1.25, 2.5
    U[1:3, g:-g, g:-g] = scale * r.uniform(-1, 1, (2, n, n))
    O.bc(U, n, g, 1)
    s = F.Solver(n, order=order, flux="up_hllc_d2av", bc="periodic")
    s.set_state(U[:, g:-g, g:-g].copy(), layout="cons", interior=True)
    s.step(3)
    ref = U.copy()
    O.d2av_run(ref, n, 1.0 / n, 0.4, 1, 3, 1e30, order, 0.5, 0.0, 0.05)
    assert np.array_equal(s.get_state(layout="cons", interior=True), ref[:, g:-g, g:-g])


@pytest.mark.parametrize("scale", [1e-80, 1e-160, 1e-240, 1e-300, 1e-318])
def test_rec3_small_momenta_equal_the_oracle(scale):
    n = 40
    r = np.random.default_rng(1)
    U = np.zeros((4, n + 4, n + 4))
    U[0], U[3] = 1.25, 2.5
    U[1:3, 2:-2, 2:-2] = scale * r.uniform(-1, 1, (2, n, n))
    O.bc(U, n, 2, 1)
    s = F.Solver(n, flux="rec3", bc="periodic", cfl=0.4)
    s.set_state(U, layout="cons")
    s.step(3)
    ref = U.copy()
    O.rec3_run(ref, n, 1.0 / n, 0.4, 3)
    assert np.array_equal(s.get_state(layout="cons")[:, 2:-2, 2:-2], ref[:, 2:-2, 2:-2])
