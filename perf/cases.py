"""The calls whose speed is measured: upwind advection of one field, of many
uneven fields at once, its gradients, and the stencil Filter, each through the
public entry points (fidibench_gb300.Upwind / Batch / batch_advect_fn / Filter,
and the C-ABI of include/fdb_filter.h for device-resident Filter fields).

A case is a dict of plain values; "kind" names the call:
  advect  set_field, advect(steps, dt), checksum, get_field on one handle
  calls   as advect, with one advect(dt) call per step (the Python class's loop)
  adjoint Upwind.adjoint: dL/df0 and dL/dv of a loss given dL/df_T
  batch   Batch.set_fields, advect, get_fields: many uneven problems
  grad    batch_advect_fn forward and torch's backward, dL/df0
  filter  one or several applications of the laplacian driver's stencil
"""
from __future__ import annotations

import numpy as np
import torch

from fidibench_gb300 import Batch, Upwind
from fidibench_gb300._capi import check, lib
from fidibench_gb300.autograd import batch_advect_fn
from fidibench_gb300.batch import random_instances
from fidibench_gb300.filter import Filter, laplacian_stencil

DEV = "cuda"


def _one(name, kind, n, v, cfl, steps, arith="auto"):
    c = {"kind": kind, "steps": steps, "cfl": cfl, "arith": arith, "ndims": len(n)}
    for j, (nj, vj) in enumerate(zip(n, v)):
        c["n%d" % j] = nj
        c["v%d" % j] = vj
    return dict(c, name=name) if name else c


def _many(name, kind, count, nmin, nmax, steps, mix):
    c = {"kind": kind, "count": count, "nmin": nmin, "nmax": nmax, "steps": steps, "mix": mix}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the drivers' smallest grids (ctest and the drivers' default cube):
        # launches and latency count
        _one("advect_32cube", "advect", (32, 32, 32), (1.0, 1.0, 1.0), 0.1, 100),
        # the reference charts' 128^3 x 100 run
        _one("advect_128cube", "advect", (128, 128, 128), (1.0, 1.0, 1.0), 0.1, 100),
        # the Python driver's loop, one advect(dt) call per step
        _one("calls_256cube", "calls", (256, 256, 256), (1.0, 1.0, 1.0), 0.1, 10),
        # extents that fit no tile, every sign of the velocity
        _one("advect_ragged", "advect", (333, 190, 417), (-0.6, 0.9, -0.4), 0.4, 50),
        # the headline benchmark: 512^3, 100 steps
        _one("advect_512cube", "advect", (512, 512, 512), (1.0, -0.7, 0.3), 0.5, 100),
        # a 2-D problem
        _one("advect_2d", "advect", (2048, 2048), (0.8, -0.5), 0.5, 50),
        # bit parity with the reference's operation order
        _one("exact_192cube", "advect", (192, 192, 192), (1.0, -0.7, 0.3), 0.5, 20, "exact"),
        # the gradient benchmark: 256^3, 200 steps, dL/df0 and dL/dv
        _one("adjoint_256cube", "adjoint", (256, 256, 256), (0.8, 0.5, -0.6), 0.4, 200),
        # the batched benchmark: 256 uneven problems, axes in [32, 160]
        _many("batch_256", "batch", 256, 32, 160, 50, 20261203),
        # initial-field recovery: 64 fields of 128^3, forward and backward
        _many("grad_64x128cube", "grad", 64, 128, 128, 100, 1),
        # the laplacian driver's default, 2-D 8000 x 8000
        {"name": "filter_8000sq", "kind": "filter", "ndims": 2, "n0": 8000, "n1": 8000,
         "iters": 1},
        # a 3-D laplacian applied repeatedly, extents that fit no tile
        {"name": "filter_3d", "kind": "filter", "ndims": 3, "n0": 301, "n1": 222, "n2": 187,
         "iters": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _velocity(rng, nd):
    return [round(rng.uniform(0.1, 1.0), 3) * rng.choice((-1.0, 1.0)) for _ in range(nd)]


def draw(rng):
    kind = rng.choice(("small", "advect", "advect", "calls", "advect2", "exact", "adjoint",
                       "batch", "batch", "grad", "filter2", "filter3"))
    if kind == "small":
        n = [rng.randint(12, 63) for _ in range(3)]
        return _one(None, "advect", n, _velocity(rng, 3), 0.3, _log_int(rng, 10, 200))
    if kind == "advect":
        n = [_log_int(rng, 64, 512) for _ in range(3)]
        return _one(None, "advect", n, _velocity(rng, 3), 0.33, _log_int(rng, 5, 100))
    if kind == "calls":
        n = [_log_int(rng, 64, 320) for _ in range(3)]
        return _one(None, "calls", n, _velocity(rng, 3), 0.33, rng.randint(2, 20))
    if kind == "advect2":
        n = [_log_int(rng, 200, 4000) for _ in range(2)]
        return _one(None, "advect", n, _velocity(rng, 2), 0.5, _log_int(rng, 5, 100))
    if kind == "exact":
        n = [_log_int(rng, 24, 256) for _ in range(3)]
        return _one(None, "advect", n, _velocity(rng, 3), 0.33, _log_int(rng, 4, 40), "exact")
    if kind == "adjoint":
        n = [_log_int(rng, 48, 256) for _ in range(3)]
        return _one(None, "adjoint", n, _velocity(rng, 3), 0.33, _log_int(rng, 10, 200))
    if kind == "batch":
        nmin = rng.randint(24, 64)
        return _many(None, "batch", _log_int(rng, 8, 256), nmin, nmin + rng.randint(8, 96),
                     _log_int(rng, 5, 50), rng.randint(1, 1 << 20))
    if kind == "grad":
        n = rng.randint(48, 128)
        return _many(None, "grad", _log_int(rng, 4, 64), n, n, _log_int(rng, 10, 100),
                     rng.randint(1, 1 << 20))
    if kind == "filter2":
        return {"kind": "filter", "ndims": 2, "n0": _log_int(rng, 500, 8000),
                "n1": _log_int(rng, 500, 8000), "iters": rng.randint(1, 4)}
    return {"kind": "filter", "ndims": 3, "n0": _log_int(rng, 64, 400),
            "n1": _log_int(rng, 64, 400), "n2": _log_int(rng, 64, 400),
            "iters": rng.randint(1, 12)}


# ---- what a case describes -----------------------------------------------------


def _shape(case):
    return tuple(case["n%d" % j] for j in range(case["ndims"]))


def _problem(case):
    n = _shape(case)
    v = tuple(case["v%d" % j] for j in range(case["ndims"]))
    dt = case["cfl"] * min(1.0 / nj / abs(vj) for nj, vj in zip(n, v))
    return n, v, dt


def _instances(case):
    """(shape, velocity, dt) of each instance: the benchmark's uneven mix, or
    the recovery workload's equal cubes with dt = 0.5 dx / sum |v|."""
    if case["kind"] == "batch":
        return [(s["n"], s["v"], s["dt"]) for s in
                random_instances(case["count"], case["mix"], case["nmin"], case["nmax"])]
    rng = np.random.default_rng(case["mix"])
    n = case["nmin"]
    out = []
    for _ in range(case["count"]):
        v = tuple(float(x) for x in rng.uniform(-1.0, 1.0, size=3))
        out.append(((n, n, n), v, 0.5 / n / sum(abs(x) for x in v)))
    return out


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _sphere(n, g, noise):
    """A sphere of ones (seeded centre and radius) plus uniform noise."""
    u = torch.rand(len(n) + 1, generator=g, device=DEV, dtype=torch.float64)
    r2 = torch.zeros(n, device=DEV, dtype=torch.float64)
    for j, nj in enumerate(n):
        x = (torch.arange(nj, device=DEV, dtype=torch.float64) + 0.5) / nj
        shape = [1] * len(n)
        shape[j] = nj
        r2 += ((x - (0.3 + 0.4 * u[j])) ** 2).view(shape)
    f = (r2 < (0.1 + 0.15 * u[-1]) ** 2).to(torch.float64)
    if noise:
        f += noise * torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    return f.reshape(-1)


def _normal(count, g):
    return torch.randn(count, generator=g, device=DEV, dtype=torch.float64)


def _inputs(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("advect", "calls"):
        return {"f0": _sphere(_shape(case), g, 0.01)}
    if kind == "adjoint":
        f0 = _sphere(_shape(case), g, 0.01)
        return {"f0": f0, "lam": _normal(f0.numel(), g)}
    if kind in ("batch", "grad"):
        f0 = torch.cat([_sphere(n, g, 0.01) for n, _, _ in _instances(case)])
        return {"f0": f0, "lam": _normal(f0.numel(), g)} if kind == "grad" else {"f0": f0}
    # filter: the driver's smooth input with a seeded phase, axis 0 fastest
    ph = torch.rand(case["ndims"], generator=g, device=DEV, dtype=torch.float64)
    f = torch.ones(1, device=DEV, dtype=torch.float64)
    for j, nj in enumerate(_shape(case)):
        x = (torch.arange(nj, device=DEV, dtype=torch.float64) + 0.5) / nj
        s = torch.sin(2.0 * np.pi * (x + ph[j]))
        f = (s[:, None] * f[None, :]).reshape(-1)
    return {"f": f}


# ---- the measured interface ----------------------------------------------------


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind in ("advect", "calls", "adjoint"):
        n, v, s["dt"] = _problem(case)
        s["up"] = Upwind(v, (1.0,) * len(n), n, arith=case["arith"])
        s["out"] = torch.empty_like(s["f0"])
    elif kind == "batch":
        inst = _instances(case)
        s["batch"] = Batch([(v, (1.0,) * 3, n) for n, v, _ in inst])
        s["dts"] = [dt for _, _, dt in inst]
        s["out"] = torch.empty_like(s["f0"])
    elif kind == "grad":
        inst = _instances(case)
        s["shapes"] = [n for n, _, _ in inst]
        s["vel"] = torch.tensor([v for _, v, _ in inst], dtype=torch.float64)
        s["dts"] = [dt for _, _, dt in inst]
        s["f0"].requires_grad_(True)
    else:
        nd = case["ndims"]
        s["filter"] = Filter(_shape(case), [0.0] * nd, [1.0] * nd, laplacian_stencil(nd))
        s["out"] = torch.empty_like(s["f"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "advect":
        s["up"].set_field(s["f0"])
        s["up"].advect(case["steps"], s["dt"])
        total = s["up"].checksum()
        return [s["up"].get_field(s["out"]), total]
    if kind == "calls":
        s["up"].set_field(s["f0"])
        for _ in range(case["steps"]):
            s["up"].advect(s["dt"])
        total = s["up"].checksum()
        return [s["up"].get_field(s["out"]), total]
    if kind == "adjoint":
        s["up"].set_field(s["f0"])
        gf, gv = s["up"].adjoint(case["steps"], s["dt"], s["lam"], s["out"])
        return [gf, gv]
    if kind == "batch":
        s["batch"].set_fields(s["f0"])
        s["batch"].advect(case["steps"], s["dts"])
        return s["batch"].get_fields(s["out"])
    if kind == "grad":
        out = batch_advect_fn(s["f0"], s["vel"], s["shapes"], case["steps"], s["dts"])
        (grad,) = torch.autograd.grad(out, s["f0"], s["lam"])
        return [out.detach(), grad]
    flt = s["filter"]
    flt.set_in_data(s["f"])
    if case["iters"] == 1:
        flt.applyFilter()
    else:
        flt.iterate(case["iters"])
    check(lib.fdb_filter_get_data(flt._h, 1, s["out"].data_ptr(), 1))
    return s["out"]


def work(case):
    """Bytes: every FP64 input read once and every output written once.
    Operations: per cell and step one multiply and one multiply-add per axis
    in the folded form; the Filter's multiply and adds per term."""
    kind = case["kind"]
    if kind == "filter":
        cells = int(np.prod(_shape(case)))
        return {"bytes": 16.0 * cells, "flops": (2.0 * case["ndims"] + 1) * cells * case["iters"]}
    if kind in ("batch", "grad"):
        cells = sum(int(np.prod(n)) for n, _, _ in _instances(case))
        back = 2.0 if kind == "grad" else 1.0
        return {"bytes": 16.0 * cells * back, "flops": 7.0 * cells * case["steps"] * back}
    nd = case["ndims"]
    cells = int(np.prod(_shape(case)))
    step = (2.0 * nd + 1) * cells * case["steps"]
    if kind == "adjoint":
        # f0 and dL/df_T in, dL/df0 out; the transposed steps and the forward
        return {"bytes": 24.0 * cells, "flops": 2.0 * step + 3.0 * nd * cells}
    return {"bytes": 16.0 * cells, "flops": step}


# ---- the same in plain torch ---------------------------------------------------


def _coeffs(n, v, dt):
    """c_j = dt v_j up_j / dx_j and up_j on the unit cube."""
    up = [1 if vj < 0.0 else -1 for vj in v]
    return [dt * vj * u / (1.0 / nj) for nj, vj, u in zip(n, v, up)], up


def _step(f, c, up, sign=1):
    """One upwind step; sign = -1: its transpose."""
    t = f.clone()
    for j, (cj, uj) in enumerate(zip(c, up)):
        t -= cj * (torch.roll(f, -uj * sign, dims=j) - f)
    return t


def _advect(f, n, v, dt, steps, sign=1):
    c, up = _coeffs(n, v, dt)
    f = f.reshape(n)
    for _ in range(steps):
        f = _step(f, c, up, sign)
    return f.reshape(-1)


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("advect", "calls"):
        n, v, dt = _problem(case)
        f = _advect(s["f0"], n, v, dt, case["steps"])
        return [f, float(f.sum())]
    if kind == "adjoint":
        n, v, dt = _problem(case)
        c, up = _coeffs(n, v, dt)
        states = [s["f0"].reshape(n)]
        for _ in range(case["steps"] - 1):
            states.append(_step(states[-1], c, up))
        lam = s["lam"].reshape(n)
        gv = np.zeros(len(n))
        while states:
            f = states.pop()
            for j, uj in enumerate(up):
                d = torch.roll(f, -uj, dims=j) - f
                gv[j] -= float((lam * d).sum()) * dt * uj * n[j]
            lam = _step(lam, c, up, -1)
        return [lam.reshape(-1), gv]
    if kind == "batch" or kind == "grad":
        out, back, at = [], [], 0
        for n, v, dt in _instances(case):
            size = int(np.prod(n))
            out.append(_advect(s["f0"][at:at + size], n, v, dt, case["steps"]))
            if kind == "grad":
                back.append(_advect(s["lam"][at:at + size], n, v, dt, case["steps"], -1))
            at += size
        return [torch.cat(out), torch.cat(back)] if kind == "grad" else torch.cat(out)
    # column-major field; an index of -1 wraps to (2^64 - 1) mod n, as the
    # reference's unsigned arithmetic gives it
    nd = case["ndims"]
    f = s["f"].reshape(tuple(reversed(_shape(case))))
    for _ in range(case["iters"]):
        t = -2.0 * nd * f
        for j, nj in enumerate(_shape(case)):
            i = torch.arange(nj, device=DEV)
            lo = i - 1
            lo[0] = (2 ** 64 - 1) % nj
            hi = (i + 1) % nj
            d = nd - 1 - j
            t += f.index_select(d, lo) + f.index_select(d, hi)
        f = t
    return f.reshape(-1)
