"""The z-slabs of the automatic choice (a single wave of equal ones; short ones
on grids that fill few CTAs) against slabs of a height asked for: the integer
update does not depend on the slabs, so the fields agree bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# equal slabs: many columns of tiles, few, the least height of 8, velocity signs
# on a ragged grid; short slabs: heights 3 to 7, fewer planes than a slab
GRIDS = [(180, 180, 180), (240, 90, 75), (130, 150, 170), (257, 120, 33), (64, 64, 64),
         (40, 50, 60), (83, 80, 80), (2, 40, 40), (1, 9, 7)]


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("depth,steps", [(2, 5), (3, 7), (4, 9), (0, 1)])
def test_slabs_do_not_change_the_field(n, depth, steps):
    import fidibench_gb300 as fdb
    rng = np.random.default_rng(sum(n) + steps)
    f0 = rng.standard_normal(n).reshape(-1)
    v = (-0.7, 1.0, 0.4)
    dt = 0.4 / max(n)
    out = []
    for tile_z in (0, 5, 10000):
        up = fdb.Upwind(v, (1.0, 1.0, 1.0), n, arith="fixed", depth=depth)
        up.set_tile_z(tile_z)
        up.f = f0
        up.advect(steps, dt)
        out.append(up.f)
        up.close()
    assert np.array_equal(out[0], out[1])
    assert np.array_equal(out[0], out[2])
