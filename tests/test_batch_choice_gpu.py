"""The batched launch's automatic form (CTA shape and z-ranges chosen from the
instances) against whole columns of the 4 x 8 shape: the integer update does not
depend on the tiling, so equal depths give equal bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# few and many instances, extents around the 6 x 4 and 4 x 8 tiles' outputs
BATCHES = [[(64, 22, 30), (70, 21, 29)], [(40, 64, 64)] * 6, [(96, 96, 96)] * 3,
           [(9, 8, 7), (130, 20, 45), (33, 47, 31), (16, 90)], [(24, 30, 28)] * 40]


@pytest.mark.parametrize("shapes", BATCHES)
@pytest.mark.parametrize("depth,steps", [(2, 7), (3, 8), (0, 1)])
def test_automatic_form_is_tiling_independent(shapes, depth, steps):
    import fidibench_gb300 as fdb
    rng = np.random.default_rng(len(shapes) + steps)
    inst = [(tuple(rng.uniform(-1, 1, len(n))), (1.0,) * len(n), n) for n in shapes]
    dts = [0.3 * min(1.0 / k / abs(x) for k, x in zip(n, v)) for v, _, n in inst]
    out = []
    f = rng.standard_normal(sum(int(np.prod(n)) for n in shapes))
    for kw in ({"depth": depth}, {"depth": depth or 2, "shape": 4, "tile_z": 1 << 20}):
        b = fdb.Batch(inst)
        b.set_tuning(**kw)
        b.set_fields(f)
        b.advect(steps, dts)
        out.append(b.get_fields())
        b.close()
    assert np.array_equal(out[0], out[1])
