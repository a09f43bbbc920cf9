"""Every diagram of the reference's integration test with the tensor-core
products (4 dilE = 8 .. 32, padded to 16 or 32, and 64) and without them: factors
are written only in the layouts in which a trace or product reads them, so each
trace kind has to find its operands."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import GOLDEN, corr_rel_err


@pytest.mark.gpu
@pytest.mark.parametrize("dilE", [1, 2, 3, 4, 5, 6, 7, 8, 9, 16])
def test_all_diagrams_match_the_fp64_path(engine_lib, tmp_path, dilE):
    from slaph_gb300 import GlobalData
    from slaph_gb300.engine import Engine
    text = (GOLDEN / "l4" / "test_all.ini").read_text().replace("EI:2", f"EI:{dilE}")
    (tmp_path / "all.ini").write_text(text)
    gd = GlobalData.from_infile(tmp_path / "all.ini",
                                ["--start_config", "1000", "--end_config", "1000"])
    d = gd.dims
    assert d.dilE == dilE
    rng = np.random.default_rng(dilE)
    gauss = lambda *n: rng.standard_normal((*n, 2)).view(np.complex128)[..., 0]  # noqa: E731
    eng = Engine(d)
    eng.set_operators(gd.plan)
    for t in range(d.Lt):
        q, _ = np.linalg.qr(gauss(3 * d.Lx * d.Ly * d.Lz, d.nev))
        eng.set_eigenvectors(t, np.ascontiguousarray(q.T))
    for r in range(d.n_rnd):
        eng.set_perambulator(r, gauss(d.Lt // d.dilT * dilE * 4, 4 * d.nev * d.Lt))
        eng.set_random_vector(r, (np.sign(gauss(d.Lt * 4 * d.nev).view(float)) * np.sqrt(0.5)
                                  ).view(np.complex128))
    eng.vdaggerv_build(0)
    ref = eng.contract(gd.plan_ptr, 0, 0)
    eng.vdaggerv_build(1)
    out = eng.contract(gd.plan_ptr, 1, 0)
    # the documented bound of the split-precision path, per correlator
    assert corr_rel_err(out, ref) < 1e-10
    eng.close()
