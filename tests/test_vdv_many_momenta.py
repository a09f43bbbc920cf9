"""VdaggerV families of more operators than one holds, with more distinct |p_x| than
one pass of the Fourier sums over the planes keeps (kMaxK, csrc/kernels/vdv_tc.cu)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("L,nev", [((12, 12, 12), 19), ((5, 5, 5), 33), ((4, 6, 5), 7),
                                   ((16, 2, 2), 9)])
def test_build_matches_the_matrix_product(engine_lib, L, nev, precision):
    from slaph_gb300 import _lib
    from slaph_gb300.engine import Engine
    Lt, vol = 2, L[0] * L[1] * L[2]
    rng = np.random.default_rng([nev, *L])
    # 13 operators along x, 11 and 9 with a phase (both signs of it), in any order
    moms = ([(p, 0, 0) for p in range(-6, 7)] + [(p, 1, 0) for p in range(-5, 6, 2)]
            + [(p, -1, 0) for p in range(-4, 5, 2)] + [(p, 1, -2) for p in range(-4, 5)])
    moms = [moms[k] for k in rng.permutation(len(moms))]
    ops = (_lib.VdvOp * len(moms))()
    for i, p in enumerate(moms):
        ops[i].id, ops[i].momentum = i, (C.c_int32 * 3)(*p)
    eng = Engine(_lib.Dims(Lt, *L, nev, 1, 2, 2))
    _lib.check(_lib.lib().slaph_engine_set_operators(eng._h, ops, len(moms), -1))
    V = rng.standard_normal((Lt, nev, 3 * vol, 2)).view(np.complex128)[..., 0]
    V /= np.linalg.norm(V, axis=2, keepdims=True)
    for t in range(Lt):
        eng.set_eigenvectors(t, V[t])
    eng.vdaggerv_build(precision)
    x = np.indices(L).reshape(3, -1).repeat(3, axis=1)
    # Entries are sums of 3 vol products of norm at most one in all: FP64 rounds by
    # at most 3 vol units of 2^-53 of that on either side, the split by 2^-46 of
    # each row's scale per term (at most sqrt(3 vol) scales).
    tol = 3 * vol * 2.0 ** -52 if precision == 0 else 2 * np.sqrt(3 * vol) * 2.0 ** -44
    for i, p in enumerate(moms):
        ph = np.exp(-2j * np.pi * sum(p[a] * x[a] / L[a] for a in range(3)))
        for t in range(Lt):
            ref = V[t].conj() @ (ph * V[t]).T
            err = np.max(np.abs(eng.vdaggerv_fetch(i, t) - ref))
            assert err < tol, (p, t, err, tol)
    eng.close()
