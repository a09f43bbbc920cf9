"""GEMM plan of the dense trace groups (plan_trace_group, csrc/host/schedule.hpp):
every value of every entry is computed once, by the tile that holds it."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import PKG, REPO

WRAPPER = r"""
#include "schedule.hpp"
using namespace slaph;
// Tiles as (entry, ia, ib) triples, in the arithmetic of the tile epilogue.
extern "C" long cover(int n_e, const int *i, const int *j, int n_a, int n_b, int tr, int tc,
                      int *count, long *tiles, long *plain) {
  TraceShape s;
  s.i.assign(i, i + n_e);
  s.j.assign(j, j + n_e);
  TraceGroupPlan const p = plan_trace_group(s, n_a, n_b, tr, tc);
  *tiles = static_cast<long>(p.tiles.size());
  *plain = 0;
  for (int e = 0; e < n_e; ++e) *plain += static_cast<long>((n_a + tr - 1) / tr) * ((n_b + tc - 1) / tc);
  for (auto const &t : p.tiles) {
    auto const &x = p.a[t.a];
    auto const &y = p.b[t.b];
    long const off = p.off[t.a * p.b.size() + t.b];
    if (off < 0) return -1;
    int const rows = static_cast<int>(x.size()) * n_a, cols = static_cast<int>(y.size()) * n_b;
    for (int r = t.row; r < std::min(rows, t.row + tr); ++r)
      for (int c = t.col; c < std::min(cols, t.col + tc); ++c) {
        int const u = r / n_a, v = c / n_b;
        int const e = p.entry[off + static_cast<long>(u) * y.size() + v];
        if (e < 0) continue;
        if (s.i[e] != x[u] || s.j[e] != y[v]) return -2;
        ++count[(static_cast<long>(e) * n_b + c % n_b) * n_a + r % n_a];
      }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def cover(tmp_path_factory):
    d = tmp_path_factory.mktemp("stacking")
    (d / "w.cpp").write_text(WRAPPER)
    so = d / "cover.so"
    host = PKG / "csrc" / "host"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{host}",
                    f"-I{REPO / 'include'}", str(d / "w.cpp"), str(host / "schedule.cpp"),
                    "-o", str(so)], check=True)
    fn = C.CDLL(str(so)).cover
    fn.restype = C.c_long
    return fn


def pairs(n_rnd, used_l, used_r):
    """Entries of tr(L R): L over (r1, r2[, used]), R over (r1, r2[, used])."""
    def lst(used):
        out = []
        for a in range(n_rnd):
            for b in range(n_rnd):
                if a == b:
                    continue
                out += ([(a, b, 1 << m) for m in range(n_rnd) if m not in (a, b)] if used
                        else [(a, b, 0)])
        return out
    left, right = lst(used_l), lst(used_r)
    return [(x, y) for x, a in enumerate(left) for y, b in enumerate(right)
            if a[1] == b[0] and a[0] == b[1] and not a[2] & b[2]]


@pytest.mark.parametrize("n_a,n_b", [(16, 16), (16, 72), (17, 81), (56, 56), (64, 80), (65, 79),
                                     (128, 144), (304, 33)])
@pytest.mark.parametrize("shape", ["plain", "one", "both", "dense", "ragged"])
def test_every_value_is_computed_once(cover, shape, n_a, n_b):
    rng = np.random.default_rng([n_a, n_b])
    es = {"plain": pairs(4, False, False), "one": pairs(5, True, False),
          "both": pairs(5, True, True), "dense": [(x, y) for x in range(5) for y in range(7)],
          "ragged": sorted({(int(x), int(y)) for x, y in rng.integers(0, 9, (20, 2))})}[shape]
    i, j = (np.array([e[k] for e in es], np.int32) for k in (0, 1))
    count = np.zeros(len(es) * n_a * n_b, np.int32)
    tiles, plain = C.c_long(), C.c_long()
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_int))  # noqa: E731
    assert cover(len(es), ptr(i), ptr(j), n_a, n_b, 64, 80, ptr(count), C.byref(tiles),
                 C.byref(plain)) == 0
    assert np.all(count == 1)
    assert tiles.value <= plain.value
