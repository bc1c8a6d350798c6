"""Host check of the work items of the batched max|f| pass
(fidibench_gb300/csrc/batch_max.h), compiled with g++ into a throwaway library:
every cell in one chunk, and no more chunks than the cells ask for, at counts
where a product of 32 bits overflows.  CPU only."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r"""
#include "batch_max.h"
extern "C" uint64_t t_chunks(const uint64_t* sizes, int count, uint64_t* first) {
  const auto m = fdb::bt::max_chunks(std::vector<uint64_t>(sizes, sizes + count));
  for (int i = 0; i <= count; ++i) first[i] = m.first[i];
  return m.cells;
}
"""


@pytest.fixture(scope="module")
def chunks(tmp_path_factory):
    d = tmp_path_factory.mktemp("max")
    src, so = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as fh:
        fh.write(SRC)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "fidibench_gb300", "csrc"), src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.t_chunks.restype = ctypes.c_uint64

    def run(sizes):
        sizes = np.asarray(sizes, dtype=np.uint64)
        first = np.empty(sizes.size + 1, dtype=np.uint64)
        cells = lib.t_chunks(sizes.ctypes.data_as(ctypes.c_void_p), ctypes.c_int(sizes.size),
                             first.ctypes.data_as(ctypes.c_void_p))
        return int(cells), first.astype(object)
    return run


@pytest.mark.parametrize("sizes", [
    [1], [1023], [1024], [1025], [64 ** 3] * 8, [160 ** 3] * 256,
    [512 ** 3] + [1] * 1999,
    [1 << 27] + [1] * 524287,          # 524,288 x 4096 is 2^31
    [1 << 30] * 3 + [8191, 8192, 8193] * 1000,
    [1 << 34, 5],
])
def test_chunks_cover_the_cells(chunks, sizes):
    cells, first = chunks(sizes)
    assert 1024 <= cells <= 8192
    for s, n in zip(sizes, np.diff(first)):
        assert (n - 1) * cells < s <= n * cells
    assert first[0] == 0 and first[-1] <= len(sizes) + sum(sizes) // cells
