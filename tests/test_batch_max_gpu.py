"""The batched max|f| pass: the largest value and a NaN are found wherever they
lie (instance, chunk edge), also when one instance is far larger than the rest."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_every_place_counts(fdb):
    sizes = [(1,), (1023,), (1024,), (1025,), (2049,), (160, 160, 160)] + [(7, 5, 3)] * 1500
    dt = [0.1 / max(n) for n in sizes]
    b = fdb.Batch([((0.5,) * len(n), (1.0,) * len(n), n) for n in sizes])
    total = sum(b.sizes)
    start = np.concatenate([[0], np.cumsum(b.sizes)])
    places = [start[0], start[1] + 1022, start[2] + 1023, start[3] + 1024, start[4] + 2048,
              start[5], start[5] + 1024, start[6] - 1, start[7], total - 1]
    rng = np.random.default_rng(8)
    for p in places:
        f = rng.standard_normal(total)
        f[p] = np.nan
        b.set_fields(f)
        b.advect(2, dt)
        with pytest.raises(fdb.FdbError) as ei:
            b.checksums()
        assert ei.value.code == 6, p
    # a value far above the rest sets the scale: a missed one overflows the fixed point
    for p in places:
        f = rng.standard_normal(total)
        f[p] = 2.0 ** 40
        b.set_fields(f)
        b.advect(1, [0.0] * b.count)
        assert np.max(np.abs(b.get_fields() - f)) <= 2.0 ** (40 - 53), p
    b.close()
