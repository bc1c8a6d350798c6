"""Kernels launched as programmatic dependents start before the launch whose
output they read has ended, so that memory is not read-only for their lifetime:
they must not read it through the read-only path (__ldg, or a const __restrict__
parameter, which the compiler may read that way).  Checked on the source, since
what goes wrong depends on the compiler's order of the loads.  CPU only."""
from __future__ import annotations

import glob
import os
import re

from conftest import ROOT

# tables that the host has uploaded, and waited for, before the chain of launches
TABLES = {"insts", "items", "groups", "offs", "sizes", "first"}


def _kernels():
    """(name, parameters, body) of every __global__ function under csrc/."""
    for path in sorted(glob.glob(os.path.join(ROOT, "fidibench_gb300", "csrc", "*.cu*"))):
        with open(path) as fh:
            src = re.sub(r"//[^\n]*", "", fh.read())
        for m in re.finditer(r"__global__\s+void\b(?:\s+__launch_bounds__\((?:[^()]|\([^()]*\))*\))?"
                             r"\s*(\w+)\s*\(([^)]*)\)\s*\{", src):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
            yield m.group(1), m.group(2), src[m.end():end]


def test_dependent_kernels_use_ordinary_loads():
    seen = set()
    for name, params, body in _kernels():
        if "cudaGridDependencySynchronize" not in body:
            continue
        seen.add(name)
        assert "__ldg" not in body, name
        for p in params.split(","):
            if "__restrict__" in p and re.search(r"\bconst\b", p.split("__restrict__")[0]):
                assert p.split()[-1] in TABLES, (name, p)
    assert {"k_advect_fixed", "k_absmax_bits", "k_step3", "k_steps_tile", "k_filter3",
            "k_batch_fixed", "k_batch_absmax"} <= seen


def test_tile_loader_uses_ordinary_loads():
    """The loads of the fixed-point kernels are in advance_tile (step_fixed.cuh)."""
    with open(os.path.join(ROOT, "fidibench_gb300", "csrc", "step_fixed.cuh")) as fh:
        src = re.sub(r"//[^\n]*", "", fh.read())
    assert "__ldg" not in src and not re.search(r"const int64_t\*\s*__restrict__", src)
