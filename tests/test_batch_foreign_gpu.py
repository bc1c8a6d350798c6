"""Batch transfers with a caller's device memory that only copies can reach
(another GPU's): no kernel gets such a pointer, and the fields arrive as through
the one-launch path.  FDB_FAULT=foreign makes every pointer but the batch's own
count as such memory, so that one GPU shows the route."""
from __future__ import annotations

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_foreign_pointers_are_staged(monkeypatch):
    import torch

    import fidibench_gb300 as fdb
    shapes = list(itertools.permutations((16, 65, 260))) + [(5, 6, 7), (40, 90), (64, 64, 64)]
    b = fdb.Batch([((0.5,) * len(n), (1.0,) * len(n), n) for n in shapes])
    assert any(b.storage_order(i) != (0, 1, 2) for i in range(b.count))
    f = torch.tensor(np.random.default_rng(12).standard_normal(sum(b.sizes)), device="cuda")
    dt = [0.1 / max(n) for n in shapes]
    want = b.advect_transposed(7, dt, f)
    monkeypatch.setenv("FDB_FAULT", "foreign")
    b.set_fields(f)
    out = torch.zeros_like(f)
    b.get_fields(out)
    assert torch.equal(out, f)
    assert torch.equal(b.advect_transposed(7, dt, f), want)
    monkeypatch.delenv("FDB_FAULT")
    at = 0
    for i, n in enumerate(b.sizes):
        assert np.array_equal(b.get_field(i), f[at:at + n].cpu().numpy()), i
        at += n
    b.close()
