"""Momentum families of VdaggerV (csrc/kernels/vdv_families.hpp): on the CPU,
that every family reproduces the momenta it stands for; on the GPU, that the
builds agree with the plain matrix product for momenta, lattices and
eigenvector counts at the edges of the kernels' tiles and planes."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import PKG

WRAPPER = r"""
#include "vdv_families.hpp"
#include <cstring>
extern "C" int families(int n, const int *ids, const int *mom, int Lx, int Ly, int Lz,
                        int sheared, int max_ops, int *out, int cap) {
  std::vector<int32_t> i(ids, ids + n), m(mom, mom + 3 * n);
  auto f = slaph::dev::vdv_families(i, m, Lx, Ly, Lz, sheared != 0, max_ops);
  int const w = sizeof(slaph::dev::VdvFamily) / 4;
  if (static_cast<int>(f.size()) * w > cap) return -1;
  std::memcpy(out, f.data(), f.size() * sizeof(slaph::dev::VdvFamily));
  return static_cast<int>(f.size());
}
"""


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    d = tmp_path_factory.mktemp("families")
    (d / "w.cpp").write_text(WRAPPER)
    so = d / "families.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{PKG / 'csrc' / 'kernels'}",
                    str(d / "w.cpp"), str(PKG / "csrc" / "host" / "vdv_families.cpp"), "-o",
                    str(so)], check=True)
    return C.CDLL(str(so)).families


def momenta(p2):
    r = range(-3, 4)
    ps = [(x, y, z) for x in r for y in r for z in r if x * x + y * y + z * z <= p2]
    return sorted(ps, key=lambda p: (sum(k * k for k in p), p))


def unpack(row):
    f = dict(axis=row[0], n=row[1], sgn=row[2], sh=row[3:5], w=row[5:8], herm=row[8])
    f["ops"] = [(row[10 + i], row[18 + i], row[26 + i]) for i in range(row[9])]
    return f


def sites(f, h, L):
    """Sites of plane h, in the kernels' enumeration."""
    others = [a for a in range(3) if a != f["axis"]]
    if f["axis"] == 3:
        return [(x, y, z) for x in range(L[0]) for y in range(L[1]) for z in range(L[2])]
    out = []
    for u in range(L[others[0]]):
        for v in range(L[others[1]]):
            x = [0, 0, 0]
            x[others[0]], x[others[1]] = u, v
            x[f["axis"]] = int(f["sgn"] * (h - f["sh"][0] * u - f["sh"][1] * v)) % f["n"]
            out.append(tuple(x))
    return out


@pytest.mark.parametrize("sheared,max_ops", [(0, 8), (1, 3)])
@pytest.mark.parametrize("L", [(4, 4, 4), (5, 5, 5), (3, 3, 3), (8, 8, 8), (4, 6, 5), (8, 2, 2),
                               (1, 9, 7)])
@pytest.mark.parametrize("p2", [0, 1, 3, 5, 9])
def test_families_reproduce_their_momenta(planner, L, p2, sheared, max_ops):
    moms = momenta(p2)
    ids = list(range(3, 3 + len(moms)))
    out = (C.c_int * 20000)()
    n = planner(len(ids), (C.c_int * len(ids))(*ids),
                (C.c_int * (3 * len(ids)))(*[k for p in moms for k in p]), *L, sheared,
                max_ops, out, 20000)
    assert n > 0
    rows = np.array(out[:34 * n]).reshape(n, 34)
    seen = []
    if not sheared:  # one set of planes for all families
        assert len({(f["axis"], f["n"], f["sgn"], *f["sh"]) for f in map(unpack, rows)}) == 1
    for f in map(unpack, rows):
        assert 1 <= len(f["ops"]) <= max_ops
        if f["herm"]:
            assert not any(f["w"])
            assert all(dag == 0 for _, _, dag in f["ops"])
        visited = []
        for h in range(f["n"]):
            for x in sites(f, h, L):
                visited.append(x)
                inner = sum(w * c / l for w, c, l in zip(f["w"], x, L))
                for op, k, dag in f["ops"]:
                    p = moms[op - 3]
                    want = sum(q * c / l for q, c, l in zip(p, x, L))
                    have = inner + k * h / f["n"]
                    d = (want + have if dag else want - have)
                    assert abs(d - round(d)) < 1e-12
        assert sorted(visited) == [(x, y, z) for x in range(L[0]) for y in range(L[1])
                                   for z in range(L[2])]
        seen += [op for op, _, _ in f["ops"]]
    assert sorted(seen) == ids


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("L,nev,p2", [
    ((4, 4, 4), 1, 4), ((4, 4, 4), 33, 9), ((3, 3, 3), 16, 2), ((5, 5, 5), 31, 5),
    ((7, 7, 7), 65, 3), ((6, 6, 6), 80, 4), ((9, 9, 9), 2, 1), ((4, 6, 5), 34, 3),
    ((2, 8, 3), 20, 2), ((8, 2, 2), 11, 1), ((1, 9, 7), 17, 3), ((11, 11, 11), 97, 3),
    # a last tile of few rows and enough tiles that edge columns save a round
    ((40, 4, 4), 71, 4), ((60, 4, 5), 150, 3), ((48, 4, 4), 97, 1), ((33, 5, 4), 65, 9)])
def test_build_matches_the_matrix_product(engine_lib, L, nev, p2, precision):
    from slaph_gb300 import _lib
    from slaph_gb300.engine import Engine
    Lt, vol = 3, L[0] * L[1] * L[2]
    moms = momenta(p2)
    ops = (_lib.VdvOp * len(moms))()
    for i, p in enumerate(moms):
        ops[i].id, ops[i].momentum = i, (C.c_int32 * 3)(*p)
    eng = Engine(_lib.Dims(Lt, *L, nev, 1, 2, 2))
    _lib.check(_lib.lib().slaph_engine_set_operators(eng._h, ops, len(moms), -1))
    rng = np.random.default_rng([nev, p2, *L])
    V = rng.standard_normal((Lt, nev, 3 * vol, 2)).view(np.complex128)[..., 0]
    V /= np.linalg.norm(V, axis=2, keepdims=True)
    for t in range(Lt):
        eng.set_eigenvectors(t, V[t])
    eng.vdaggerv_build(precision)
    x = np.indices(L).reshape(3, -1).repeat(3, axis=1)
    # Entries of M are sums of 3 vol products of norm at most one in all: FP64
    # rounds by at most 3 vol units of 2^-53 of that on either side, the split
    # by 2^-46 of each row's scale per term (at most sqrt(3 vol) scales).
    tol = 3 * vol * 2.0 ** -52 if precision == 0 else 2 * np.sqrt(3 * vol) * 2.0 ** -44
    for i, p in enumerate(moms):
        ph = np.exp(-2j * np.pi * sum(p[a] * x[a] / L[a] for a in range(3)))
        for t in range(Lt):
            ref = V[t].conj() @ (ph * V[t]).T
            err = np.max(np.abs(eng.vdaggerv_fetch(i, t) - ref))
            assert err < tol, (p, t, err, tol)
    eng.close()


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [-300, -130, -60, -40, 0, 40, 60, 130, 300])
def test_split_precision_build_scales_exactly(engine_lib, shift):
    """Eigenvectors times 2^shift: the split works on scaled integers, so the
    blocks are those of the unscaled eigenvectors times 2^(2 shift), bit for
    bit, whichever way the columns' exponents are found.  Some columns have
    their largest entry on a power of two, where a bound of the norm does not
    settle the exponent."""
    from slaph_gb300 import _lib
    from slaph_gb300.engine import Engine
    L, nev = 4, 19
    rng = np.random.default_rng(3)
    V = rng.uniform(-0.4, 0.4, (nev, 3 * L ** 3, 2)).view(np.complex128)[..., 0]
    V[3, 7], V[5, 11], V[8, 100] = 1.0, 0.5j, -1.0 + 2.0 ** -40
    V[9] = 0.0
    ops = (_lib.VdvOp * 2)()
    for i, p in enumerate([(1, 0, 0), (1, -1, 2)]):
        ops[i].id, ops[i].momentum = i, (C.c_int32 * 3)(*p)
    x = np.indices((L, L, L)).reshape(3, -1).repeat(3, axis=1)
    blocks = []
    for s in (0, shift):
        eng = Engine(_lib.Dims(1, L, L, L, nev, 1, 2, 2))
        _lib.check(_lib.lib().slaph_engine_set_operators(eng._h, ops, 2, -1))
        eng.set_eigenvectors(0, V * 2.0 ** s)
        eng.vdaggerv_build(1)
        blocks.append([eng.vdaggerv_fetch(i, 0) for i in range(2)])
        eng.close()
    for i, p in enumerate([(1, 0, 0), (1, -1, 2)]):
        assert np.array_equal(blocks[0][i] * 2.0 ** (2 * shift), blocks[1][i])
        ref = V.conj() @ (np.exp(-2j * np.pi * (np.array(p) @ x) / L) * V).T
        # 47 bits of each row's scale per term, 192 terms
        assert np.max(np.abs(blocks[0][i] - ref)) < 2 * 192 * 2.0 ** -46


@pytest.mark.gpu
@pytest.mark.parametrize("nev", [64, 67, 195, 200])
def test_displaced_and_momentum_operators_share_tiles(engine_lib, nev):
    """Displaced operators need every row of the last tile, momentum operators
    take edge columns for it: both in one build, against the FP64 build."""
    from slaph_gb300 import _lib
    from slaph_gb300.engine import Engine
    L, Lt = 12, 2
    moms = momenta(2)
    disp = [b">x", b"<y>z"]
    ops = (_lib.VdvOp * (len(moms) + len(disp)))()
    for i, p in enumerate(moms):
        ops[i].id, ops[i].momentum = i, (C.c_int32 * 3)(*p)
    for d, s in enumerate(disp):
        ops[len(moms) + d].id, ops[len(moms) + d].n_disp = len(moms) + d, len(s) // 2
        ops[len(moms) + d].disp = s
    eng = Engine(_lib.Dims(Lt, L, L, L, nev, 1, 2, 2))
    _lib.check(_lib.lib().slaph_engine_set_operators(eng._h, ops, len(ops), -1))
    rng = np.random.default_rng(nev)
    V = rng.standard_normal((Lt, nev, 3 * L ** 3, 2)).view(np.complex128)[..., 0]
    V /= np.linalg.norm(V, axis=2, keepdims=True)
    for t in range(Lt):
        eng.set_eigenvectors(t, V[t])
        u, _ = np.linalg.qr(rng.standard_normal((L ** 3, 3, 3, 3, 2)).view(np.complex128)[..., 0])
        eng.set_gauge(t, np.ascontiguousarray(u).reshape(L ** 3, 3, 9))
    blocks = []
    for precision in (0, 1):
        eng.vdaggerv_build(precision)
        blocks.append([eng.vdaggerv_fetch(i, t) for i in range(len(ops)) for t in range(Lt)])
    # as above: 3 L^3 terms, the split 2^-46 of each row's scale per term; a
    # displaced vector of two steps has entries up to the norm of the
    # eigenvector times its longest run of links
    tol = 4 * np.sqrt(3 * L ** 3) * 2.0 ** -44
    for a, b in zip(*blocks):
        assert np.max(np.abs(a - b)) < tol * max(1.0, np.max(np.abs(a)))
    eng.close()
