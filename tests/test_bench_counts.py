"""The operation counts that bench.py divides by (CPU)."""
from __future__ import annotations

import pytest

from fidibench_gb300.filter import laplacian_stencil


@pytest.mark.parametrize("stencil,issued", [
    (laplacian_stencil(2), 4), (laplacian_stencil(3), 7), ({(0,): 0.5, (1,): 0.5}, 4),
    ({(0, 0): 2.0, (0, 1): -8.0}, 3)])
def test_issued_fp64_of_the_filter(stencil, issued):
    import bench
    assert bench.filter_fp64_issued(stencil) == issued
