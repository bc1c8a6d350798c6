"""Launch tables built in host memory that ends with the call: the kernels read
what the call built, also when the heap is reused right away by the next one."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_new_tables_on_every_call():
    """dt changes from call to call, so each advect and gradient uploads tables
    of its own while the earlier ones' launches run; fresh handles that do one
    call each give the same bits."""
    import torch

    import fidibench_gb300 as fdb
    from fidibench_gb300.batch import random_instances
    specs = random_instances(200, 5, 20, 40)
    desc = [(s["v"], s["L"], s["n"]) for s in specs]
    one = fdb.Batch(desc)
    f = torch.randn(sum(one.sizes), dtype=torch.float64, device="cuda",
                    generator=torch.Generator("cuda").manual_seed(1))
    lam = torch.randn_like(f)
    one.set_fields(f)
    got = []
    for k in range(4):
        dts = [s["dt"] * (1.0 - 0.1 * k) for s in specs]
        g, gv = one.adjoint(5, dts, lam)
        one.advect(5, dts)
        out = torch.empty_like(f)
        one.get_fields(out)
        got.append((g.clone(), gv.copy(), out))
    one.close()
    x = f
    for k in range(4):
        dts = [s["dt"] * (1.0 - 0.1 * k) for s in specs]
        b = fdb.Batch(desc)
        b.set_fields(x)
        g, gv = b.adjoint(5, dts, lam)
        assert torch.equal(g, got[k][0]) and np.array_equal(gv, got[k][1]), k
        b.advect(5, dts)
        out = torch.empty_like(f)
        b.get_fields(out)
        assert torch.equal(out, got[k][2]), k
        x = out
        b.close()
