"""Several FP64 steps per launch (small grids) against the same steps one call at
a time, which run one launch each: the cell arithmetic is the same, so the
fields agree bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one cell, fewer cells than a halo, one tile, remainders on every axis, one
# long axis, 2-D, a grid above what takes several steps per launch
GRIDS = [(1,), (7,), (2000,), (5, 9), (3, 700), (1, 1, 1), (2, 2, 2), (12, 12, 12), (3, 17, 33),
         (16, 9, 25), (40, 41, 42)]


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("arith", ["fma", "exact"])
def test_steps_per_launch_keep_the_bits(n, arith):
    import fidibench_gb300 as fdb
    rng = np.random.default_rng(sum(n))
    f0 = rng.standard_normal(int(np.prod(n)))
    for sign in (1.0, -1.0):
        v = tuple(sign * x for x in (0.9, -0.6, 0.3)[:len(n)])
        dt = 0.3 / max(n)
        for steps in (2, 3, 11, 24):
            up = fdb.Upwind(v, (1.0,) * len(n), n, arith=arith)
            up.f = f0
            up.advect(steps, dt)
            a = up.f
            up.f = f0
            for _ in range(steps):
                up.advect(1, dt)
            assert np.array_equal(a, up.f), (n, arith, sign, steps)
            up.close()
