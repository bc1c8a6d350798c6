"""The fixed-point advect's 30-bit coefficients (all steps but the last, the error
carried from step to step) where they leave most: the highest frequency, undamped
(sum_j a_j = 1), coefficients halfway between multiples of 2^-30, many steps."""
from __future__ import annotations

import ctypes
from fractions import Fraction

import numpy as np
import pytest

from test_step_coeffs_host import _q, fx  # noqa: F401

U30 = 2.0 ** -30
# per axis (z, y, x): sums of 1 to rounding
COEFFS = [
    (0.25 + 0.49 * U30, 0.25 + 0.49 * U30, 0.5 - 0.98 * U30),
    (1 / 3, 1 / 3, 1 / 3),
    (0.30 + 0.5 * U30, 0.45 - 0.4995 * U30, 0.25),
    (0.0, 0.6 + 0.47 * U30, 0.4 - 0.46 * U30),
]


@pytest.mark.parametrize("phi", [0.0, 1e-4, 0.02, 0.25, 0.4999, 0.5, -0.3, -0.4999])
@pytest.mark.parametrize("steps", [2, 7, 100, 1000])
def test_squared_errors_of_the_steps(fx, phi, steps):  # noqa: F811
    """What the carried errors leave is -1/2 sum_n (sum_j e_n,j D_j)^2: per axis
    their squares sum to at most S / 4 + 1 units of 2^-60."""
    q, full = _q(fx, 0.3 + phi * U30)
    out = (ctypes.c_int32 * 2)()
    total = Fraction(0)
    for n in range(1, steps + 1):
        fx.t_step(q, n, n == steps, out)
        total += Fraction((out[0] << 32) + out[1] - full, 1 << 32) ** 2
    assert total <= Fraction(steps, 4) + 1


@pytest.mark.gpu
@pytest.mark.parametrize("a", COEFFS)
@pytest.mark.parametrize("steps", [3, 100, 400])
@pytest.mark.parametrize("plain", [True, False])
def test_undamped_highest_frequency(fdb, a, steps, plain):
    n = (16, 18, 20)
    axes = [j for j in range(3) if a[j] != 0.0]
    par = sum(np.indices(n)[j] for j in axes) % 2
    f0 = np.where(par, 1.0, -1.0)
    if not plain:
        f0 = f0 * (1.0 + 0.1 * np.random.default_rng(9).random(n))
    # a_j = dt v_j / dx_j with dt = 1, dx_j = 1 / n_j
    v = tuple(a[j] / n[j] for j in range(3))
    up = fdb.Upwind(v, (1.0, 1.0, 1.0), n, arith="fixed")
    up.f = f0
    up.advect(steps, 1.0)
    got = up.f
    up.close()
    # the coefficients as the library rounds them: (dt v_j) / dx_j
    c = [np.longdouble((1.0 * v[j]) / (1.0 / n[j])) for j in range(3)]
    f = f0.astype(np.longdouble)
    for _ in range(steps):
        f = f + sum(c[j] * (np.roll(f, 1, j) - f) for j in range(3))
    # rounding: 2 units a step, one unit at most 2^-56 of max|f| (two guard bits);
    # the remainder: 1/2 (2 sum_j |e_j|)^2 <= 6 sum_j e_j^2, three axes of
    # (S / 4 + 1) 2^-60; the last conversion
    tol = steps * 2.0 ** -55 + 18 * (steps / 4 + 1) * 2.0 ** -60 + 2.0 ** -53
    assert np.max(np.abs(got.reshape(n) - f)) <= tol * np.max(np.abs(f0))
