"""The Filter's fused terms (weights +-2^k), its unrolled stencils and its share
of cells per thread against the CPU restatement, bit for bit: weights that fuse
and that do not at every position, 1 to 9 terms, offsets beyond an extent, and
values whose products overflow, underflow or are not finite."""
from __future__ import annotations

import numpy as np
import pytest

from test_filter_gpu import oracle_applies, run_filter

pytestmark = pytest.mark.gpu

FUSED = [1.0, -1.0, 2.0, -4.0, 2.0 ** 40, -2.0 ** 999]
GENERAL = [0.5, -6.0, 0.0, 3.0, 2.0 ** -1000, 1.0e300]


def same(out, ref):
    return (np.array_equal(out, ref, equal_nan=True)
            and np.array_equal(np.signbit(out[~np.isnan(ref)]), np.signbit(ref[~np.isnan(ref)])))


@pytest.mark.parametrize("nterms", range(1, 10))
@pytest.mark.parametrize("mix", ["fused", "centre", "any"])
def test_weights_at_every_position(port, nterms, mix):
    rng = np.random.default_rng(10 * nterms + len(mix))
    for dims in ((37, 11), (9, 8, 13), (300,)):
        nd = len(dims)
        offs = set()
        while len(offs) < nterms:
            offs.add(tuple(int(x) for x in rng.integers(-3, 4, size=nd - 1)) +
                     (int(rng.integers(-6, 7)),))
        offs = sorted(offs)
        w = []
        for k in range(nterms):
            pool = FUSED if mix == "fused" or (mix == "centre" and k != nterms // 2) else GENERAL
            if mix == "any":
                pool = FUSED + GENERAL
            w.append(float(rng.choice(pool)))
        n = int(np.prod(dims))
        f = rng.standard_normal(n) * 10.0 ** rng.integers(-320, 308, size=n)
        f[rng.integers(0, n, size=4)] = [np.inf, -np.inf, 0.0, -0.0]
        f[rng.integers(0, n, size=4)] = [1.7e308, -1.7e308, 5e-324, -2.3e-308]
        for periodic in (False, True):
            with np.errstate(all="ignore"):
                out, _ = run_filter(dims, list(zip(offs, w)), f, periodic)
                ref = oracle_applies(port, dims, list(zip(offs, w)), f, periodic)
            assert same(out, ref), (dims, offs, w, periodic)


@pytest.mark.parametrize("dims", [(3, 2), (2, 3, 2), (1, 5), (700, 700), (2, 400000)])
def test_offsets_beyond_an_extent_and_strides(port, dims):
    nd = len(dims)
    rng = np.random.default_rng(sum(dims))
    offs = [(0,) * nd, (7,) + (0,) * (nd - 1), (-9,) + (1,) * (nd - 1), (0,) * (nd - 1) + (-5,)]
    f = rng.standard_normal(int(np.prod(dims)))
    st = list(zip(offs, [-4.0, 1.0, 0.3, -1.0]))
    for periodic in (False, True):
        out, _ = run_filter(dims, st, f, periodic)
        assert same(out, oracle_applies(port, dims, st, f, periodic)), (dims, periodic)
