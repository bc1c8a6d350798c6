"""Block chains whose time step or velocity changes: within the parity tolerance
of the oracle, or refused with the chain unchanged where planes were exchanged."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu

N, L = (24, 20, 32), (1.0, 1.0, 1.0)
FIELD_TOL = 1e-13


def _open(fdb, v, dt, f0):
    from fidibench_gb300._capi import FDB_OK, lib
    up = fdb.Upwind(v, L, N, arith="fixed", depth=3)
    up.f = f0
    fixed = ctypes.c_int()
    assert lib.fdb_upwind_block_begin(up._h, dt, ctypes.byref(fixed)) == FDB_OK and fixed.value
    return up, lib


def _field(seed=6):
    # the highest frequency, which a change of coefficient feeds most
    z, y, x = np.indices(N)
    rng = np.random.default_rng(seed)
    return (np.where((z + y + x) % 2, 1.0, -1.0) * (1 + 0.1 * rng.random(N))).ravel()


# dt of each block (steps), from a = 0.1 on the x axis to 0.9
CHAINS = [
    [(3, 0.1), (3, 0.9)],
    [(3, 0.1), (3, 0.1), (2, 0.9), (3, 0.9), (1, 0.3)],
    [(1, 0.1), (3, 0.9), (3, 0.2)],
    [(3, 0.5), (3, 0.25), (2, 0.5)],  # multiples of 2^-30: nothing to settle
]


@pytest.mark.parametrize("blocks", CHAINS)
@pytest.mark.parametrize("v", [(0.0, 0.0, 1.0), (0.05, -0.03, 1.0)])
def test_chain_with_changing_dt(fdb, port, blocks, v):
    f0 = _field()
    up, lib = _open(fdb, v, blocks[0][1] / 32, f0)
    ref = f0
    for k, (steps, a) in enumerate(blocks):
        st = lib.fdb_upwind_advect_block(up._h, steps, a / 32, int(k == len(blocks) - 1))
        assert st == 0, lib.fdb_last_error()
        ref = port.advect(N, v, L, ref, steps, a / 32)
    assert rel_maxnorm(up.f, ref) <= FIELD_TOL
    up.advect(4, 0.1 / 32)  # and the handle goes on
    assert rel_maxnorm(up.f, port.advect(N, v, L, ref, 4, 0.1 / 32)) <= FIELD_TOL
    up.close()


def test_chain_with_changing_velocity(fdb, port):
    f0, dt = _field(7), 0.1 / 32
    v0, v1 = (0.0, 0.0, 1.0), (0.0, 0.0, -1.0)
    up, lib = _open(fdb, v0, dt, f0)
    assert lib.fdb_upwind_advect_block(up._h, 3, dt, 0) == 0
    v = np.array(v1)
    assert lib.fdb_upwind_set_velocity(up._h, v.ctypes.data) == 0
    assert lib.fdb_upwind_advect_block(up._h, 3, dt, 1) == 0
    ref = port.advect(N, v1, L, port.advect(N, v0, L, f0, 3, dt), 3, dt)
    assert rel_maxnorm(up.f, ref) <= FIELD_TOL
    up.close()


def test_exchanged_chain_refuses_the_change(fdb, port):
    from fidibench_gb300._capi import FDB_ERR_INVALID
    f0, v, dt = _field(8), (0.3, 0.2, 1.0), 0.1 / 32
    up, lib = _open(fdb, v, dt, f0)
    assert lib.fdb_upwind_advect_block(up._h, 3, dt, 0) == 0
    plane = np.empty(N[1] * N[2])
    assert lib.fdb_upwind_get_planes(up._h, 2, 1, plane.ctypes.data, 0) == 0
    assert lib.fdb_upwind_set_planes(up._h, 2, 1, plane.ctypes.data, 0) == 0
    assert lib.fdb_upwind_advect_block(up._h, 3, 2 * dt, 0) == FDB_ERR_INVALID
    assert lib.fdb_upwind_advect_block(up._h, 2, dt, 1) == 0  # the chain as it was
    ref = port.advect(N, v, L, f0, 5, dt)
    assert rel_maxnorm(up.f, ref) <= FIELD_TOL
    up.close()
