"""Large dense trace groups: the epilogue of a stacked GEMM tile packs the block and
the group of a column into one int (csrc/kernels/trace_tc.cu), so plan_trace_group
may stack operand indices only while both fit."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import PKG, REPO

WRAPPER = r"""
#include "schedule.hpp"
using namespace slaph;
// Values written per (entry, ia, ib), with block and group of a column taken from
// the packed word as the epilogue takes them; -1: outside the entry table.
extern "C" long cover(int n_e, const int *i, const int *j, int n_a, int n_b, int tr, int tc,
                      int *count, long *stacked) {
  TraceShape s;
  s.i.assign(i, i + n_e);
  s.j.assign(j, j + n_e);
  TraceGroupPlan const p = plan_trace_group(s, n_a, n_b, tr, tc);
  *stacked = 0;
  for (auto const &t : p.tiles) {
    auto const &x = p.a[t.a];
    auto const &y = p.b[t.b];
    long const off = p.off[t.a * p.b.size() + t.b];
    int const rows = static_cast<int>(x.size()) * n_a, cols = static_cast<int>(y.size()) * n_b;
    bool const table = x.size() > 1 || y.size() > 1;
    *stacked += table;
    for (int r = t.row; r < std::min(rows, t.row + tr); ++r)
      for (int c = t.col; c < std::min(cols, t.col + tc); ++c) {
        int v = 0, ib = c;
        if (table) {
          int const packed = static_cast<int>(static_cast<unsigned>(c / n_b) << 16) | (c % n_b);
          v = packed >> 16;
          ib = packed & 0xFFFF;
        }
        long const at = off + static_cast<long>(r / n_a) * y.size() + v;
        if (v < 0 || v >= static_cast<int>(y.size()) || ib >= n_b) return -1;
        int const e = p.entry[at];
        if (e >= 0) ++count[(static_cast<long>(e) * n_b + ib) * n_a + r % n_a];
      }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def cover(tmp_path_factory):
    d = tmp_path_factory.mktemp("packing")
    (d / "w.cpp").write_text(WRAPPER)
    so = d / "cover.so"
    host = PKG / "csrc" / "host"
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", f"-I{host}",
                    f"-I{REPO / 'include'}", str(d / "w.cpp"), str(host / "schedule.cpp"),
                    "-o", str(so)], check=True)
    fn = C.CDLL(str(so)).cover
    fn.restype = C.c_long
    return fn


@pytest.mark.parametrize("shape,n_a,n_b,stacks", [
    # two operands of A that meet one of B: stacked rows, plain columns
    ("rows", 16, 65535, True), ("rows", 16, 65536, True), ("rows", 16, 65537, False),
    ("rows", 16, 70000, False),
    # two of B that meet one of A: stacked columns
    ("columns", 16, 32745, True), ("columns", 16, 65537, False),
    # more operands than the block field counts
    ("many", 16, 16, None)])
def test_packed_columns(cover, shape, n_a, n_b, stacks):
    es = {"rows": [(0, 0), (1, 0)], "columns": [(0, 0), (0, 1)],
          "many": [(0, k) for k in range(40000)]}[shape]
    i, j = (np.array([e[k] for e in es], np.int32) for k in (0, 1))
    count = np.zeros(len(es) * n_a * n_b, np.int32)
    stacked = C.c_long()
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_int))  # noqa: E731
    assert cover(len(es), ptr(i), ptr(j), n_a, n_b, 64, 80, ptr(count), C.byref(stacked)) == 0
    assert np.all(count == 1)
    if stacks is not None:
        assert (stacked.value > 0) == stacks
