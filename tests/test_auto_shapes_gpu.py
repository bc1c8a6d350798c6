"""The launches the automatic choice makes (4-warp CTAs of 8, 6 or 4 rows,
z-slabs by the remaining planes) against a CTA shape asked for: the integer
update does not depend on the tiling, so the fields agree bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (nz, ny, nx): fewer rows or columns than a tile; one past a tile; less than
# half a wave of tiles (4 rows); 8-, 6- and 4-row tiles; more z-slabs than the
# slab table holds at 8 planes each; a single plane
GRIDS = [(9, 5, 3), (17, 30, 31), (40, 33, 61), (616, 58, 58), (416, 63, 58), (620, 42, 59),
         (1300, 20, 20), (1, 64, 70)]


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("depth,steps", [(2, 5), (3, 7), (4, 9), (0, 1), (3, 1)])
def test_auto_choice_is_tiling_independent(n, depth, steps):
    import fidibench_gb300 as fdb
    rng = np.random.default_rng(sum(n) + steps)
    f0 = rng.standard_normal(n).reshape(-1)
    v = (0.7, -1.0, 0.4)
    dt = 0.4 / max(n)
    out = []
    for shape in (-1, 4):
        up = fdb.Upwind(v, (1.0, 1.0, 1.0), n, arith="fixed", depth=depth)
        up.set_shape(shape)
        up.f = f0
        up.advect(steps, dt)
        out.append(up.f)
        up.close()
    assert np.array_equal(out[0], out[1])
