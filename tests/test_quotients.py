"""The shared-reciprocal quotients of the kernels (fvb_ieee.cuh) compiled for
the host: wherever a caller's range tests hold, the value has the bits of the
operator's, the sign of a zero included, and the tests hold for every zero
numerator.  No GPU needed; the device's reciprocal seed is the host's exact one
here (test_gpu_quotients.py has the device's).  Also the FP64 face's floors.
"""
from __future__ import annotations

import ctypes as C
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

HOST = r"""
#include <cmath>
#include <cstring>
#include <stdint.h>
#include <cuda_runtime.h>
using std::fma; using std::fabs; using std::sqrt;
static inline unsigned max(unsigned a, unsigned b) { return a > b ? a : b; }
static inline unsigned min(unsigned a, unsigned b) { return a < b ? a : b; }
static inline long long __double_as_longlong(double x) { long long v; std::memcpy(&v, &x, 8); return v; }
static inline int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
static inline int __double2loint(double x) { return (int)__double_as_longlong(x); }
static inline double __hiloint2double(int h, int l)
{
    const long long v = ((long long)h << 32) | (unsigned)l;
    double x;
    std::memcpy(&x, &v, 8);
    return x;
}
static inline unsigned __float_as_uint(float x) { unsigned v; std::memcpy(&v, &x, 4); return v; }
using std::rint; using std::copysign;
static inline double __drcp_rn(double x) { return 1.0 / x; }
static inline float __frcp_rn(float x) { return 1.0f / x; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fdividef(float a, float b) { return a / b; }
static inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }
#define FVB_EXACT_RCP_SQRT 1
#include "fvb_ieee.cuh"
#include "fvb_face32.cuh"
#include "fvb_face64.cuh"
extern "C" {
// 1: the range tests hold, and q is the kernels' quotient
void quot64(int n, const double *a, const double *b, double *q, int *ok)
{
    for (int i = 0; i < n; ++i) {
        q[i] = fvb::quot(a[i], b[i], fvb::recip(b[i]));
        ok[i] = fvb::num_ok(a[i]) && fvb::den_ok(b[i]) && b[i] > 0;
    }
}
// the FP32 face's p / (gamma - 1), and HLLE with its quotients as operators
void over_gm1_32(int n, const float *p, float gm1, float *e, float *floored, float *plain)
{
    const fvb::f32::Gas gs{gm1 + 1.0f, gm1, __frcp_rn(gm1)};
    for (int i = 0; i < n; ++i) {
        e[i] = fvb::f32::over_gm1(p[i], gs);
        floored[i] = fvb::f32::over_gm1_floored(p[i], gs);
        plain[i] = p[i] / gm1;
    }
}
void hlle32(int n, const float *L, const float *R, const float *c, const float *E, float *F, float *P)
{
    for (int i = 0; i < n; ++i) {
        const float *l = L + 4 * i, *r = R + 4 * i, cL = c[2 * i], cR = c[2 * i + 1], EL = E[2 * i], ER = E[2 * i + 1];
        fvb::f32::hlle(l, r, cL, cR, EL, ER, F + 4 * i);
        float *o = P + 4 * i;
        const float FL[4] = {l[0] * l[1], l[0] * l[1] * l[1] + l[3], l[0] * l[1] * l[2], (EL + l[3]) * l[1]};
        const float FR[4] = {r[0] * r[1], r[0] * r[1] * r[1] + r[3], r[0] * r[1] * r[2], (ER + r[3]) * r[1]};
        const float U[4] = {l[0], l[0] * l[1], l[0] * l[2], EL}, V[4] = {r[0], r[0] * r[1], r[0] * r[2], ER};
        const float SL = std::fmin(l[1] - cL, r[1] - cR), SR = std::fmax(l[1] + cL, r[1] + cR);
        const float dS = std::fmax(SR - SL, 1e-10f), SRL = SR * SL;
        for (int q = 0; q < 4; ++q)
            o[q] = SL >= 0.f ? FL[q] : SR <= 0.f ? FR[q] : (SR * FL[q] - SL * FR[q] + SRL * (V[q] - U[q])) / dS;
    }
}
// the FP64 face's floors: of rho and p, and of a sound speed whose square is p / r
void floors64(int n, const double *x, double *f, double *c)
{
    for (int i = 0; i < n; ++i) {
        f[i] = fvb::f64::fl14(x[i]);
        c[i] = fvb::f64::snd(x[i], 1.0);
    }
}
void small64(int n, const double *a, const double *b, double *q, int *ok)
{
    for (int i = 0; i < n; ++i) {
        q[i] = fvb::small_quot(a[i], b[i], fvb::recip(b[i]));
        ok[i] = (fvb::is_small(a[i]) || a[i] == 0) && fvb::den_ok(b[i]);
    }
}
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("quot")
    src, so = d / "host.cpp", d / "host.so"
    src.write_text(HOST)
    subprocess.run(["g++", "-std=c++17", "-O1", "-mfma", "-ffp-contract=off", "-fPIC", "-shared", "-I", str(CUDA),
                    "-I", str(ROOT / "include"), "-I", str(ROOT / "fvstuff_b200" / "csrc"), "-o", str(so), str(src)],
                   check=True)
    return C.CDLL(str(so))


RNG = np.random.default_rng(20)
N = 200000


def _mag(lo, hi, dtype=np.float64):
    with np.errstate(over="ignore", under="ignore"):
        return np.ldexp(RNG.uniform(1, 2, N), RNG.integers(lo, hi, N)).astype(dtype)


def _signed(x):
    return np.where(RNG.random(N) < 0.5, -x, x).astype(x.dtype)


def _ints(k):
    return RNG.integers(1, k, N).astype(np.float64) * 2.0 ** RNG.integers(-1074, 960, N).astype(np.float64)


OPERANDS64 = {
    "ordinary": lambda: (_signed(_mag(-60, 60)), _mag(-60, 60)),
    "tiny numerators": lambda: (_signed(_mag(-1074, -700)), _mag(-40, 40)),
    "subnormal numerators": lambda: (_signed(RNG.integers(1, 1000, N) * 5e-324), _mag(-3, 3)),
    "zeros": lambda: (_signed(np.zeros(N)), _mag(-500, 99)),
    "whole range": lambda: (_signed(_mag(-1074, 1023)), _mag(-1000, 1000)),
    "beside powers of two": lambda: (_signed(_ints(9)), np.ldexp(1.0 + RNG.integers(-4, 5, N) * 2.0 ** -53,
                                                                 RNG.integers(-20, 20, N))),
}


@pytest.mark.parametrize("name", list(OPERANDS64))
def test_fp64_quotient_where_its_range_tests_hold(host, name):
    a, b = (np.ascontiguousarray(x, np.float64) for x in OPERANDS64[name]())
    q, ok = np.empty(N), np.empty(N, np.int32)
    p = lambda x: x.ctypes.data_as(C.c_void_p)
    host.quot64(N, p(a), p(b), p(q), p(ok))
    with np.errstate(all="ignore"):
        want = a / b
    ok = ok.astype(bool)
    assert np.array_equal(q[ok].view(np.int64), want[ok].view(np.int64))
    if name in ("ordinary", "zeros"):
        assert ok.all()  # the usual path


@pytest.mark.parametrize("name", list(OPERANDS64) + ["ties"])
def test_fp64_quotient_of_small_numerators(host, name):
    """Below num_ok's range, subnormal quotients and their ties included, for
    denominators of either sign."""
    if name == "ties":  # (k + 1/2) 2^-1074, exactly, just above and just below
        b = 2.0 * RNG.integers(1, 1 << 20, N)
        a = ((2 * RNG.integers(0, 1 << 20, N) + 1) * (b / 2) + RNG.integers(-1, 2, N)) * 5e-324
        a = _signed(a)
    else:
        a, b = OPERANDS64[name]()
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(_signed(np.asarray(b, np.float64)))
    q, ok = np.empty(N), np.empty(N, np.int32)
    p = lambda x: x.ctypes.data_as(C.c_void_p)
    host.small64(N, p(a), p(b), p(q), p(ok))
    with np.errstate(all="ignore"):
        want = a / b
    ok = ok.astype(bool) & ~((a == 0) & np.signbit(a) & (b > 0))  # (squot: a zero numerator is +0)
    assert np.array_equal(q[ok].view(np.int64), want[ok].view(np.int64))
    if name in ("ties", "subnormal numerators"):
        assert ok.all()


def _f32(*x):
    return [np.ascontiguousarray(a, np.float32) for a in x]


def _same32(got, want):
    nan = np.isnan(got) & np.isnan(want)
    return np.array_equal(got.view(np.int32)[~nan], want.view(np.int32)[~nan]) and not np.isnan(got[~nan]).any()


@pytest.mark.parametrize("gm1", [0.4, 2.0 / 3.0, 0.0625, 1e-5])
def test_fp32_pressure_over_gamma_minus_one(host, gm1):
    """Pressures over all of FP32, infinities among them; floored ones (1e-14 and
    up) by the form without a range test."""
    p, = _f32(_mag(-149, 128))
    p[:100], p[100:200], p[200:300] = np.inf, 0.0, np.nan
    e, f, plain = (np.empty(N, np.float32) for _ in range(3))
    ptr = lambda x: x.ctypes.data_as(C.c_void_p)
    host.over_gm1_32(N, ptr(p), C.c_float(gm1), ptr(e), ptr(f), ptr(plain))
    assert _same32(e, plain)
    up = p >= np.float32(1e-14)
    assert _same32(f[up], plain[up])


@pytest.mark.parametrize("vel", [(-20, 4), (-120, -90), (-149, -120), None])
@pytest.mark.parametrize("unit", [0, 12, 26])
def test_fp32_hlle(host, vel, unit):
    """Cell velocities down to subnormal and zero, sound speeds near 1, 2^12 and
    2^26: numerators and quotients that underflow."""
    z = np.zeros(N)
    w = [[_mag(-2, 2), _signed(_mag(*vel) * 2.0 ** unit if vel else z), _signed(_mag(*vel) * 2.0 ** unit if vel else z),
          _mag(-2, 2) * 4.0 ** unit] for _ in range(2)]
    same = RNG.random(N) < 0.5  # equal densities and pressures: nothing but the small terms
    for q in (0, 3):
        w[1][q] = np.where(same, w[0][q], w[1][q])
    L, R = (np.ascontiguousarray(np.stack(x, 1), np.float32) for x in w)
    c = np.ascontiguousarray(np.stack([np.sqrt(1.4 * x[3] / x[0]) for x in w], 1), np.float32)
    E = np.ascontiguousarray(np.stack([2.5 * x[3] for x in w], 1), np.float32)
    F, P = np.empty((N, 4), np.float32), np.empty((N, 4), np.float32)
    ptr = lambda x: x.ctypes.data_as(C.c_void_p)
    host.hlle32(N, ptr(L), ptr(R), ptr(c), ptr(E), ptr(F), ptr(P))
    assert _same32(F, P)


def test_fp64_floors(host):
    """x > 1e-14 ? x : 1e-14 to the last bit, for numbers beside the floor, of
    either sign, infinite and NaN; the sound speed's at 1e-7 likewise."""
    near = 1e-14 * (1 + RNG.uniform(-4e-6, 4e-6, N // 4))
    ulps = 1e-14 + RNG.integers(-4, 5, N // 4) * np.spacing(1e-14)
    x = np.concatenate([near, ulps, -near, _mag(-1074, 1023)[: N // 4]])
    x[:5] = [0.0, -0.0, np.inf, -np.inf, np.nan]
    f, c = np.empty_like(x), np.empty_like(x)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    host.floors64(len(x), p(x), p(f), p(c))
    assert np.array_equal(f, np.where(x > 1e-14, x, 1e-14))
    with np.errstate(invalid="ignore"):
        r = np.sqrt(x)
    assert np.array_equal(c, np.where(r > 1e-7, r, 1e-7))
