"""The FP64 step of fields on either side of the lines where it takes more CTAs:
bit-identical to the oracle, whatever the share of a CTA."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,v", [((143, 144, 145), (0.7, -0.4, 0.3)),   # 2,985,840 cells
                                 ((120, 125, 200), (-0.7, 0.4, -0.3)),  # 3,000,000
                                 ((2828, 2828), (0.6, -0.5)),           # 7,997,584
                                 ((200, 199, 203), (-0.2, -0.4, 0.8)),  # 8,079,400
                                 ((8000000,), (1.0,)), ((3000011,), (-1.0,))])
@pytest.mark.parametrize("steps", [1, 3])
def test_shares_of_the_cells(fdb, port, n, v, steps):
    L = (1.0,) * len(n)
    dt = 0.3 / max(n)
    f0 = np.random.default_rng(5).standard_normal(int(np.prod(n)))
    up = fdb.Upwind(v, L, n, arith="exact")
    up.f = f0
    up.advect(steps, dt)
    assert np.array_equal(up.f, port.advect(n, v, L, f0, steps, dt))
    up.close()
