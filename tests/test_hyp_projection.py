"""SU(3) projection of the HYP smearing (proj_su3, csrc/kernels/gauge_smear.cu)
away from thermalised links: the smearing of one site-uniform configuration is
the projection of a known matrix per link, checked against a projection by
singular value decomposition."""
from __future__ import annotations

import numpy as np
import pytest

from slaph_gb300 import _lib


def project(m):
    u, _, vh = np.linalg.svd(m)
    x = u @ vh
    d = np.linalg.det(x)
    return x * np.exp(-1j * np.angle(d) / 3)[..., None, None]


def su3(rng, n):
    q, _ = np.linalg.qr(rng.standard_normal((n, 3, 3)) + 1j * rng.standard_normal((n, 3, 3)))
    return project(q)


@pytest.mark.gpu
@pytest.mark.parametrize("alpha", [0.0, 0.3, 0.62, 0.9])
@pytest.mark.parametrize("kind", ["diagonal", "spread", "scaled"])
def test_uniform_links(engine_lib, kind, alpha):
    """Links U_d the same at every site: with commuting (diagonal) links the
    staples are U_d again, so every blend is a multiple of U_d (equal singular
    values); with general ones the blends have spread singular values; 'scaled'
    multiplies all links by 1e-9, which no projection may notice."""
    from slaph_gb300.engine import Engine
    rng = np.random.default_rng(int(100 * alpha) + len(kind))
    L, Lt = 2, 3
    if kind == "diagonal":
        ph = rng.uniform(-1, 1, (Lt, 3, 3))
        ph[..., 2] = -ph[..., 0] - ph[..., 1]
        U = np.zeros((Lt, 3, 3, 3), complex)
        U[..., range(3), range(3)] = np.exp(1j * ph)
    else:
        U = su3(rng, 3 * Lt).reshape(Lt, 3, 3, 3)
        # towards the unit matrix, as in a smooth configuration
        U = project(U + 2.0 * np.eye(3))
    dag = lambda x: x.conj().swapaxes(-1, -2)  # noqa: E731

    def staples(f, b):
        return f @ b @ dag(f) + dag(f) @ b @ f

    want = []
    for t in range(Lt):
        dec = {(d, p): project((1 - alpha) * U[t, d] + alpha / 2 * staples(U[t, p], U[t, d]))
               for d in range(3) for p in range(3) if p != d}
        want.append([project((1 - alpha) * U[t, d] + alpha / 4 * sum(
            staples(dec[n, 3 - d - n], dec[d, 3 - d - n]) for n in range(3) if n != d))
            for d in range(3)])
    want = np.array(want)
    eng = Engine(_lib.Dims(Lt, L, L, L, 4, 1, 1, 1))
    # 'scaled' needs alpha = 0: staples are cubic in the links
    f = 1e-9 if kind == "scaled" and alpha == 0.0 else 1.0
    for t in range(Lt):
        links = f * U[t].swapaxes(-1, -2).reshape(1, 3, 9)
        eng.set_gauge(t, np.ascontiguousarray(np.broadcast_to(links, (L ** 3, 3, 9))))
    eng.smear_gauge_hyp(alpha, alpha, 1)
    for t in range(Lt):
        got = eng.gauge_fetch(t).reshape(L ** 3, 3, 3, 3).swapaxes(-1, -2)
        # blends have singular values above 0.1 here: A^(-1/2) rounds by at
        # most about 100 units of 2^-53 times a few tens of operations
        assert np.max(np.abs(got - want[t])) < 1e-12
    eng.close()
