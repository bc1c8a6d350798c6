"""Host check of the per-step coefficients of the fixed-point advect
(fidibench_gb300/csrc/fixed_point.cuh step_qcoeff, step_qcoeff_carry) and of
the six-product cell update they allow (fixed_update6), against exact integers.
Compiled with g++ into a throwaway library; CPU only."""
from __future__ import annotations

import ctypes
import os
import subprocess
import tempfile
from fractions import Fraction

import numpy as np
import pytest

from conftest import ROOT

SRC = r"""
#include <stdint.h>
#include "fixed_point.cuh"
extern "C" {
void t_qcoeff(double a, int32_t* q) {
  fdb::QCoeff r = fdb::make_qcoeff(a); q[0] = r.a1; q[1] = r.a0;
}
void t_step(const int32_t* q, int64_t n, int last, int32_t* out) {
  fdb::QCoeff c{q[0], q[1]};
  c = fdb::step_qcoeff(c, n, last != 0);
  out[0] = c.a1; out[1] = c.a0;
}
void t_carry(const int32_t* q, int64_t* carry, int last, int32_t* out) {
  fdb::QCoeff c{q[0], q[1]};
  c = fdb::step_qcoeff_carry(c, carry, last != 0);
  out[0] = c.a1; out[1] = c.a0;
}
int64_t t_update6(int64_t c, int64_t zb, int64_t up, int64_t left, const int32_t* a) {
  return fdb::fixed_update6(c, zb, up, left, a[0], a[1], a[2]);
}
int64_t t_update9(int64_t c, int64_t zb, int64_t up, int64_t left, const int32_t* a) {
  return fdb::fixed_update(c, zb, up, left, fdb::QCoeff{a[0], 0}, fdb::QCoeff{a[1], 0},
                           fdb::QCoeff{a[2], 0});
}
}
"""


@pytest.fixture(scope="module")
def fx():
    d = tempfile.mkdtemp()
    src = os.path.join(d, "t.cpp")
    so = os.path.join(d, "t.so")
    with open(src, "w") as fh:
        fh.write(SRC)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "fidibench_gb300", "csrc"), src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    i32p, i64p = ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_int64)
    lib.t_qcoeff.argtypes = [ctypes.c_double, i32p]
    lib.t_step.argtypes = [i32p, ctypes.c_int64, ctypes.c_int, i32p]
    lib.t_carry.argtypes = [i32p, i64p, ctypes.c_int, i32p]
    for f in (lib.t_update6, lib.t_update9):
        f.argtypes = [ctypes.c_int64] * 4 + [i32p]
        f.restype = ctypes.c_int64
    return lib


A = [0.0, 1.0, 0.5, 0.1, 1.0 / 3.0, 0.999999999, 1e-7, 1e-18, 2.0 ** -31, 3.0 * 2.0 ** -32]


def _q(fx, a):
    q = (ctypes.c_int32 * 2)()
    fx.t_qcoeff(a, q)
    return q, (q[0] << 32) + q[1]


@pytest.mark.parametrize("a", A)
@pytest.mark.parametrize("steps", [1, 2, 3, 100, 1001])
def test_steps_sum_to_the_coefficient(fx, a, steps):
    """The coefficients of an advect's steps sum to steps * a exactly, every
    partial sum within 2^-31, every one of them in [0, 2^30] units of 2^-30
    with a0 = 0 but for the last; the carried form gives the same."""
    q, full = _q(fx, a)
    total, carry = 0, ctypes.c_int64(0)
    out, out2 = (ctypes.c_int32 * 2)(), (ctypes.c_int32 * 2)()
    for n in range(1, steps + 1):
        last = n == steps
        fx.t_step(q, n, last, out)
        fx.t_carry(q, ctypes.byref(carry), last, out2)
        assert list(out) == list(out2)
        assert 0 <= out[0] <= 1 << 30 and (last or out[1] == 0)
        total += (out[0] << 32) + out[1]
        assert abs(total - n * full) <= 1 << 31
    assert total == steps * full


def test_one_step_keeps_the_coefficient(fx):
    for a in A:
        q, _ = _q(fx, a)
        out = (ctypes.c_int32 * 2)()
        fx.t_step(q, 1, 1, out)
        assert list(out) == list(q)


def test_far_steps_stay_in_range(fx):
    for a in A:
        q, full = _q(fx, a)
        out = (ctypes.c_int32 * 2)()
        for n in (1 << 20, (1 << 31) - 1):
            for last in (0, 1):
                fx.t_step(q, n, last, out)
                assert 0 <= out[0] <= 1 << 30
                assert abs((out[0] << 32) - full) <= 1 << 32


@pytest.mark.parametrize("a", [(1 << 30, 1 << 30, 1 << 30), (0, 0, 0), (1, 0, 1 << 29),
                               (357913941, 357913942, 357913941), (1073741823, 5, 7)])
def test_six_products(fx, a):
    """fixed_update6 gives fixed_update's integer for a0 = 0, within 2 units of
    the exact value, also at the range limits; exactly F when every difference
    is 0."""
    av = (ctypes.c_int32 * 3)(*a)
    lim = (1 << 59) + (1 << 39)
    rng = np.random.default_rng(7)
    cases = [tuple(int(x) for x in rng.integers(-lim, lim, size=4, endpoint=True))
             for _ in range(400)]
    cases += [(lim, -lim, -lim, -lim), (-lim, lim, lim, lim), (0, lim, -lim, lim),
              (lim,) * 4, (-lim,) * 4, (0,) * 4]
    for c, zb, up, left in cases:
        got = fx.t_update6(c, zb, up, left, av)
        assert got == fx.t_update9(c, zb, up, left, av)
        exact = c + Fraction(sum(x * (u - c) for x, u in zip(a, (zb, up, left))), 1 << 30)
        assert abs(got - exact) <= 2
        if zb == up == left == c:
            assert got == c
