"""Batch.set_fields / get_fields on device tensors (one launch for all
instances) against the per-instance calls, over instances stored in every kind
of axis order and extents off the 32 x 32 tile of the transposition."""
from __future__ import annotations

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXTENTS = [(16, 65, 260), (33, 128, 64), (300, 40, 31), (97, 64, 47), (8, 181, 182)]


def test_all_orders_round_trip():
    import torch

    import fidibench_gb300 as fdb
    shapes = [p for e in EXTENTS for p in itertools.permutations(e)]
    shapes += [(5, 6, 7), (40, 90), (7,), (64, 64, 64)]  # stored as described
    b = fdb.Batch([((0.5,) * len(n), (1.0,) * len(n), n) for n in shapes])
    orders = {b.storage_order(i) for i in range(b.count)}
    assert (0, 1, 2) in orders and {o[2] for o in orders} == {0, 1, 2}, orders
    rng = np.random.default_rng(11)
    f = rng.standard_normal(sum(b.sizes))
    dev = torch.tensor(f, device="cuda")
    b.set_fields(dev)
    at = 0
    for i, n in enumerate(b.sizes):
        assert np.array_equal(b.get_field(i), f[at:at + n]), (shapes[i], b.storage_order(i))
        b.set_field(i, -f[at:at + n])
        at += n
    out = torch.zeros_like(dev)
    b.get_fields(out)
    assert torch.equal(out, -dev)
    # host arrays take the same order
    b.set_fields(f)
    assert np.array_equal(b.get_fields(), f)
    b.close()
