"""SU(3) projection of the HYP smearing (proj_su3, csrc/kernels/gauge_smear.cu) of
matrices that are far from a multiple of a unitary one, or far from order one in
scale.  With alpha1 = alpha2 = 0 a smearing step is the projection of every link."""
from __future__ import annotations

import numpy as np
import pytest

from slaph_gb300 import _lib


def unitary(rng, n):
    u, _, vh = np.linalg.svd(rng.standard_normal((n, 3, 3)) + 1j * rng.standard_normal((n, 3, 3)))
    return u @ vh


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1.0, 1e-60, 1e-9, 1e60])
@pytest.mark.parametrize("sv", [
    (1, 1, 1), (1, 0.9, 0.6), (1, 0.5, 1e-3), (1, 0.36, 0.35), (1, 0.34, 0.33), (1, 0.41, 1e-4),
    (1, 0.39, 1e-4), (1, 0.1, 0.1), (1, 0.1, 1e-4), (1, 1.1e-2, 1e-2), (1, 1e-2, 1e-2),
    (1, 1e-3, 1e-3), (1, 2e-4, 1e-4), (1, 2e-5, 1e-5)])
def test_projection_of_any_matrix(engine_lib, sv, scale):
    from slaph_gb300.engine import Engine
    L, Lt = 2, 2
    rng = np.random.default_rng([int(1e6 * s) for s in sv])
    n = Lt * L ** 3 * 3
    m = (unitary(rng, n) * np.array(sv, float)) @ unitary(rng, n)
    u, _, vh = np.linalg.svd(m)
    want = u @ vh
    want *= np.exp(-1j * np.angle(np.linalg.det(want)) / 3)[:, None, None]
    # a power of two, so that the scaled matrices are the same ones
    m = m * 2.0 ** round(np.log2(scale))
    eng = Engine(_lib.Dims(Lt, L, L, L, 4, 1, 1, 1))
    links = np.ascontiguousarray(m.reshape(Lt, L ** 3, 3, 3, 3).swapaxes(-1, -2))
    for t in range(Lt):
        eng.set_gauge(t, links[t].reshape(L ** 3, 3, 9))
    eng.smear_gauge_hyp(0.0, 0.0, 1)
    got = np.array([eng.gauge_fetch(t).reshape(L ** 3, 3, 3, 3).swapaxes(-1, -2)
                    for t in range(Lt)]).reshape(n, 3, 3)
    eng.close()
    # The projection moves by 1 / (smallest singular value) per unit of M: some 64
    # roundings of it on both sides.  The phase comes from det M, whose terms of order one
    # round by about a unit, of a determinant of s2 s3.
    tol = 2.0 ** -53 * (64 / sv[2] + 1 / (sv[1] * sv[2]))
    # (beside the branch cut of the cube root either neighbour is right)
    beside = np.abs(np.abs(np.angle(np.linalg.det(m / np.abs(m).max()))) - np.pi) < 1e-3
    assert beside.sum() < n // 4
    assert np.max(np.abs(got - want)[~beside]) < tol
