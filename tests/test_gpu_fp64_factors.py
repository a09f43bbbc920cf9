"""FP64 factors, traces and terms at matrix sizes below and between those of the
other tests (4 dilE = 4, 12, 16, 20, 24, 64): several trace entries per warp, row
tiles across Dirac blocks, shared Q1 products; against the oracle, with both
accumulators.  Seven random vectors make traces of 42 entries, more than the
terms keep inner sums for."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import corr_rel_err, og, workload_inputs


@pytest.mark.gpu
@pytest.mark.parametrize("dilE,nev,n_rnd", [(1, 7, 4), (3, 13, 4), (4, 17, 4), (5, 16, 4),
                                            (6, 33, 4), (16, 35, 4), (1, 7, 7)])
def test_pion_rho_set_matches_oracle(engine_lib, oracle_lib, tmp_path, dilE, nev, n_rnd):
    from slaph_gb300 import GlobalData, synthetic
    from slaph_gb300.engine import Engine
    ops = [o.replace("p0,1,2,3,4", "p0") for o in synthetic.PION_RHO_OPERATORS]
    corr = (["C2c:Q0:Op9:Q0:Op9:P0"]
            + [f"C3c:Q0:Op9:Q0:Op{k}:Q0:Op9:P0" for k in range(9)]
            + ["C4cD:Q0:Op9:Q0:Op9:Q0:Op9:Q0:Op9:P0", "C20:Q0:Op1:Q0:Op1:P0"])
    w = synthetic.Workload("fp64_factors", Lt=4, L=4, nev=nev, n_rnd=n_rnd, dilT=2, dilE=dilE,
                           operators=ops, correlators=corr, seed=70 + dilE)
    gd = GlobalData.from_infile(w.write_infile(str(tmp_path)))
    V, peram, noise = workload_inputs(w)
    eng = Engine(gd.dims)
    eng.set_operators(gd.plan)
    for t, v in enumerate(V):
        eng.set_eigenvectors(t, v)
    for r in range(w.n_rnd):
        eng.set_perambulator(r, peram[r])
        eng.set_random_vector(r, noise[r])
    eng.vdaggerv_build(0)
    vdv = oracle_lib.vdaggerv(og(gd).dims, og(gd).plan, V)
    for acc in (0, 1):
        ref = oracle_lib.contract(og(gd).dims, og(gd).plan_ptr, vdv, peram, noise, acc, -1,
                                  gd.output_doubles()).reshape(-1, gd.dims.Lt)
        assert np.max(np.abs(ref)) > 0
        # the bound of the FP64 path against the oracle
        assert corr_rel_err(eng.contract(gd.plan_ptr, 0, acc), ref) < 1e-12
    eng.close()
