"""The automatic form of batches that leave most of the GPU idle (4 steps per
block, ranges of 8 planes) against whole columns of the same depth: the integer
update does not depend on the tiling, so the fields agree bit for bit; and
against depth 2, whose time blocks rescale at other steps: 40 roundings of at
most 8 units of 2^-58 max|f| each, on either side."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BATCHES = [[(32, 32, 32)] * 8, [(24, 40, 31), (5, 6, 7), (33, 29, 30)], [(64, 64, 64)] * 4,
           [(48, 30)], [(28, 28, 8), (29, 29, 9)]]


@pytest.mark.parametrize("shapes", BATCHES)
@pytest.mark.parametrize("steps", [1, 4, 40])
def test_small_batches(shapes, steps):
    import fidibench_gb300 as fdb
    rng = np.random.default_rng(len(shapes) + steps)
    inst = [(tuple(rng.uniform(-1, 1, len(n))), (1.0,) * len(n), n) for n in shapes]
    dts = [0.3 * min(1.0 / k / abs(x) for k, x in zip(n, v)) for v, _, n in inst]
    out = []
    f = rng.uniform(-1, 1, sum(int(np.prod(n)) for n in shapes))
    for kw in ({"depth": 0}, {"depth": 4, "shape": 4, "tile_z": 1 << 20}, {"depth": 2}):
        b = fdb.Batch(inst)
        b.set_tuning(**kw)
        b.set_fields(f)
        b.advect(steps, dts)
        out.append(b.get_fields())
        b.close()
    assert np.array_equal(out[0], out[1])
    assert np.abs(out[0] - out[2]).max() <= 2 * steps * 8 * 2.0 ** -58 + 2.0 ** -52
