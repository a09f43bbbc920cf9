"""A schedule belongs to the contents of its plan, not to the plan's address: a
front end made where another was freed, or a caller that changes its tables in
place, gives other tables at the same address (plan_words, same_plan in
csrc/host/schedule.hpp)."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import PKG, REPO, workload_inputs

WRAPPER = r"""
#include "schedule.hpp"
static std::vector<int32_t> kept;
extern "C" long keep(slaph_plan const *p) {
  kept = slaph::plan_words(*p);
  return static_cast<long>(kept.size());
}
extern "C" int same(slaph_plan const *p) { return slaph::same_plan(kept, *p) ? 1 : 0; }
"""


@pytest.fixture(scope="module")
def words(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan_words")
    (d / "w.cpp").write_text(WRAPPER)
    so = d / "w.so"
    host = PKG / "csrc" / "host"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{host}",
                    f"-I{REPO / 'include'}", str(d / "w.cpp"), str(host / "schedule.cpp"),
                    "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.keep.restype = C.c_long
    return lib


def workload(tmp_path, name, momenta):
    from slaph_gb300 import GlobalData, synthetic
    w = synthetic.Workload(name, Lt=4, L=4, nev=8, n_rnd=3, dilT=2, dilE=2,
                           operators=[f"g5.d0.p{momenta}"],
                           correlators=[f"C2c:Q0:Op0:Q0:Op0:P{momenta}"])
    d = tmp_path / name
    d.mkdir()
    return w, GlobalData.from_infile(w.write_infile(str(d)))


def at_one_address(*plans):
    """A plan structure that holds each of the plans in turn."""
    from slaph_gb300 import _lib
    box = _lib.Plan()
    for p in plans:
        C.memmove(C.byref(box), p, C.sizeof(_lib.Plan))
        yield box


def test_equal_words_are_equal_plans(engine_lib, words, tmp_path):
    _, a = workload(tmp_path, "a", "0")
    _, b = workload(tmp_path, "b", "0,1")
    _, c = workload(tmp_path, "c", "0")
    for k, box in enumerate(at_one_address(a.plan_ptr, b.plan_ptr)):
        if k == 0:
            assert words.keep(C.byref(box)) > 0
            assert words.same(C.byref(box))
        else:
            assert not words.same(C.byref(box))
    assert words.same(a.plan_ptr) and words.same(c.plan_ptr)
    # every table and count, changed in place
    p = a.plan
    words.keep(a.plan_ptr)
    req = p.diagrams[0].requests[0]
    places = [(p, "n_vdv_ops"), (p.factors[0][0], "id_vdaggerv"),
              (p.factors[0][0], "need_vdaggerv_daggering"), (p.factors[2][0], "gamma"),
              (req, "n_traces"), (req.traces[0], "tr_id"), (req.traces[0], "kind")]
    for where, field in places:
        old = getattr(where, field)
        setattr(where, field, old ^ 1)
        assert not words.same(a.plan_ptr), field
        setattr(where, field, old)
    kind = req.traces[0].kind
    for array, k in ((p.factors[0][0].rnd_pairs, 1), (p.trace_ql_ids[kind], 0),
                     (req.traces[0].loc, 1)):
        old = array[k]
        array[k] = old ^ 1
        assert not words.same(a.plan_ptr)
        array[k] = old
    assert words.same(a.plan_ptr)


def test_tables_that_are_not_given_are_not_read(words):
    from slaph_gb300 import _lib
    p = _lib.Plan()
    p.n_factors[2], p.n_trace_ids[3] = 5, 4  # null tables
    words.keep(C.byref(p))
    assert words.same(C.byref(p))
    p.n_trace_ids[3] = 3
    assert not words.same(C.byref(p))


@pytest.mark.gpu
@pytest.mark.parametrize("per_block_pair", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_contract_follows_the_plan_at_one_address(engine_lib, tmp_path, precision,
                                                  per_block_pair):
    """The plan of one diagram, then that of two (more correlators), then as many
    correlators in another order, over one operator table."""
    from slaph_gb300 import GlobalData, _lib, synthetic
    from slaph_gb300.engine import Engine
    w = synthetic.Workload("one_address", Lt=4, L=4, nev=8, n_rnd=4, dilT=2, dilE=2,
                           operators=["g5.d0.p0,1"],
                           correlators=["C2c:Q0:Op0:Q0:Op0:P0,1", "C20:Q0:Op0:Q0:Op0:P0,1"])
    gd = GlobalData.from_infile(w.write_infile(str(tmp_path)))
    V, peram, noise = workload_inputs(w)

    def engine():
        eng = Engine(gd.dims)
        eng.set_factor_lifetime(per_block_pair)
        eng.set_operators(gd.plan)
        for t, v in enumerate(V):
            eng.set_eigenvectors(t, v)
        for r in range(w.n_rnd):
            eng.set_perambulator(r, peram[r])
            eng.set_random_vector(r, noise[r])
        eng.vdaggerv_build(precision)
        return eng

    first = _lib.Plan()
    C.memmove(C.byref(first), gd.plan_ptr, C.sizeof(_lib.Plan))
    one = (_lib.Diagram * 1)(gd.plan.diagrams[0])  # its first diagram only
    first.n_diagrams, first.diagrams = 1, one
    fresh = engine()
    want = fresh.contract(gd.plan_ptr, precision)
    fresh.close()
    eng = engine()
    last = _lib.Plan()
    C.memmove(C.byref(last), gd.plan_ptr, C.sizeof(_lib.Plan))
    turned = (_lib.Diagram * 2)(gd.plan.diagrams[1], gd.plan.diagrams[0])
    last.diagrams = turned
    n0 = gd.plan.diagrams[0].n_requests
    assert gd.plan.n_diagrams == 2 and not np.array_equal(want, np.roll(want, -n0, 0))
    for k, box in enumerate(at_one_address(C.byref(first), gd.plan_ptr, gd.plan_ptr,
                                           C.byref(last), gd.plan_ptr)):
        out = eng.contract(C.pointer(box), precision)
        ref = np.roll(want, -n0, 0) if k == 3 else want[:n0] if k == 0 else want
        assert np.array_equal(out, ref)
    eng.close()
