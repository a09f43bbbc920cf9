"""Range of the Q2 factors in the split-precision path: with the perambulators of
one random vector scaled up and those of the other scaled down, every Q2 is what it
was, but its intermediate, the product of the first perambulator and VdaggerV, is
far outside the range of FP32."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import workload_inputs


@pytest.mark.gpu
@pytest.mark.parametrize("dilE", [1, 3, 8, 16])
@pytest.mark.parametrize("precision", [0, 1])
def test_scaled_perambulators_give_the_same_correlators(engine_lib, tmp_path, dilE, precision):
    from slaph_gb300 import GlobalData, synthetic
    from slaph_gb300.engine import Engine
    w = synthetic.Workload("factor_range", Lt=4, L=4, nev=19, n_rnd=2, dilT=2, dilE=dilE,
                           operators=["g5.d0.p0,1"], correlators=["C2c:Q0:Op0:Q0:Op0:P0,1"])
    gd = GlobalData.from_infile(w.write_infile(str(tmp_path)))
    assert gd.schedule_stats()["q1"] == 0 and gd.schedule_stats()["q2"] > 0
    V, peram, noise = workload_inputs(w)
    eng = Engine(gd.dims)
    eng.set_operators(gd.plan)
    for t, v in enumerate(V):
        eng.set_eigenvectors(t, v)
    for r in range(2):
        eng.set_random_vector(r, noise[r])
    eng.vdaggerv_build(precision)
    out = []
    for shift in (0, 90, 130, 400, -110, -400):
        eng.set_perambulator(0, peram[0] * 2.0 ** shift)
        eng.set_perambulator(1, peram[1] * 2.0 ** -shift)
        out.append(eng.contract(gd.plan_ptr, precision))
    eng.close()
    assert np.all(np.isfinite(out[0])) and np.max(np.abs(out[0])) > 0
    # powers of two throughout: the same digits and sums, bit for bit
    for o in out[1:]:
        assert np.array_equal(o, out[0])
