"""The work that users of the engine have it do, as cases that can be timed.

A case is one pass through the package's public entry points: a gauge
configuration (VdaggerV build and contraction) from inputs that are already on
the device or from host buffers, the contraction of one block pair alone, or
VdaggerV of one operator and timeslice on the caller's device buffers.  Inputs
are synthetic, of the shapes and value distributions of production runs:
eigenvectors are normalised complex Gaussian columns, perambulators complex
Gaussian, noise Z2 x Z2, gauge links SU(3) matrices scattered about a pure gauge
(plaquette about 0.6, as thermalised links).

listed() and draw() give cases, prepare() what a program holds before the call,
run() one pass, work() the bytes and operations it cannot do without, and
exact() the result in plain 64-bit torch where that is quick: two-point
correlators and VdaggerV blocks.  The four-point diagrams have no such short
form: a plain evaluation of their factor products takes minutes.
"""
import ctypes
import math
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "slaph-contractions_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from slaph_gb300 import GlobalData, _lib, synthetic  # noqa: E402
from slaph_gb300.engine import (FP64, KAHAN, MIXED, NATIVE, Engine, OperatorFactory,  # noqa: E402
                                pinned_empty)

HYP = (0.62, 0.62, 3)  # alpha1, alpha2, iterations of the displaced runs
_DISPLACED_OPS = [">x", "<x", ">y", "<y", ">z", "<z"]


# ---------------------------------------------------------------- cases
def _config(name, diagrams, L, Lt, nev, n_rnd, dilT, dilE, p2, precision="mixed",
            accumulator="native", upload=False, slots=0, block_pair=-1):
    return {"name": name, "kind": "config", "diagrams": diagrams, "L": L, "Lt": Lt, "nev": nev,
            "n_rnd": n_rnd, "dilT": dilT, "dilE": dilE, "p2": p2, "precision": precision,
            "accumulator": accumulator, "upload": upload, "slots": slots,
            "block_pair": block_pair}


def listed():
    return [
        # The command line's work for one configuration of the smallest test
        # lattice: every input uploaded, build, contraction.  Launches and
        # synchronisations count here, not arithmetic.
        _config("twopoint_4x8", "twopoint", 4, 8, 16, 4, 2, 4, 1, upload=True),
        # The pipi set on the test lattice in the plain FP64 path with the
        # Kahan accumulator: what a validation run does.
        _config("pipi_4x8_fp64_kahan", "pipi", 4, 8, 16, 5, 4, 4, 1, precision="fp64",
                accumulator="kahan", upload=True),
        # An odd lattice, eigenvector count and interlace in FP64.
        _config("twopoint_14x24_fp64", "twopoint", 14, 24, 51, 3, 8, 3, 1, precision="fp64"),
        # Pion two-point run on the 24^3x48 ensemble, 27 momenta: the VdaggerV
        # build is nearly all of it.
        _config("twopoint_24x48", "twopoint", 24, 48, 120, 2, 16, 8, 3),
        # Few eigenvectors and three random vectors: two- and three-point
        # functions, fine time dilution (21 block pairs of little work each).
        _config("pipi_24x48_nev64", "pipi", 24, 48, 64, 3, 8, 8, 1),
        # The ordinary configuration of a scattering run on 24^3x48.
        _config("pipi_24x48_nev120", "pipi", 24, 48, 120, 5, 8, 8, 1),
        # The same on 32^3x64 with 220 eigenvectors: the largest.
        _config("pipi_32x64_nev220", "pipi", 32, 64, 220, 4, 16, 8, 1),
        # One block pair of a 32^3x64 contraction with moving frames, as a job
        # array splits a configuration (--single_time_slice_combination); the
        # VdaggerV blocks are there already.  The contraction does not see the
        # lattice volume, so they come from a small one.
        _config("blockpair_64_nev220", "pipi", 8, 64, 220, 5, 16, 8, 2, block_pair=1),
        # The plain FP64 path on a production lattice.
        _config("pipi_24x48_nev64_fp64", "pipi", 24, 48, 64, 3, 8, 8, 1, precision="fp64"),
        # One-derivative operators: gauge links uploaded and HYP-smeared, six
        # displaced operators beside the momenta.
        _config("displaced_24x48", "displaced", 24, 48, 96, 3, 16, 8, 1),
        # A lattice whose eigenvectors stay on the host: streamed through a
        # ring of device slots, factors per block pair; ragged sizes, Kahan.
        _config("streamed_18x48", "pipi", 18, 48, 81, 4, 12, 6, 1, accumulator="kahan",
                upload=True, slots=4),
        # VdaggerV of one operator and timeslice on the caller's own device
        # buffers, without allocation.
        {"name": "noalloc_24_nev120", "kind": "noalloc", "L": 24, "nev": 120, "px": 0, "py": 1,
         "pz": -1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["twopoint", "twopoint", "pipi", "pipi", "pipi", "blockpair", "fp64",
                       "displaced", "streamed", "noalloc"])
    if what == "noalloc":
        return {"kind": "noalloc", "L": _log_int(rng, 4, 32), "nev": rng.randint(8, 220),
                "px": rng.randint(-2, 2), "py": rng.randint(-2, 2), "pz": rng.randint(-2, 2)}
    dilT = rng.choice([4, 6, 8, 12, 16])
    nb = rng.randint(2, 6 if dilT < 12 else 4)
    c = {"diagrams": "pipi", "L": _log_int(rng, 4, 28), "Lt": dilT * nb,
         "nev": rng.randint(12, 180), "n_rnd": rng.randint(3, 5), "dilT": dilT,
         "dilE": rng.choice([2, 3, 4, 6, 8, 8, 8]), "p2": 1,
         "accumulator": rng.choice(["native", "native", "kahan"])}
    if what == "twopoint":
        c.update(diagrams="twopoint", n_rnd=rng.randint(2, 6), p2=rng.randint(1, 3),
                 upload=rng.random() < 0.3)
    elif what == "blockpair":
        c.update(L=8, block_pair=rng.randrange(nb * (nb + 1) // 2), p2=rng.randint(1, 2))
    elif what == "fp64":
        c.update(precision="fp64", L=_log_int(rng, 4, 20), nev=rng.randint(12, 64),
                 n_rnd=rng.randint(3, 4), diagrams=rng.choice(["twopoint", "pipi"]))
    elif what == "displaced":
        c.update(diagrams="displaced", L=rng.randint(6, 24), n_rnd=rng.randint(2, 4),
                 nev=rng.randint(12, 120))
    elif what == "streamed":
        c.update(L=rng.randint(6, 20), nev=rng.randint(12, 120), upload=True,
                 slots=rng.choice([2, 4, 6]))
    c["nev"] = min(c["nev"], 3 * c["L"] ** 3)
    full = _config("", **c)
    del full["name"]
    return full


def _workload(c):
    moms = ",".join(str(k) for k in range(c["p2"] + 1))
    if c["diagrams"] == "pipi":
        ops = [o.replace("p0,1,2,3,4", "p" + moms) for o in synthetic.PION_RHO_OPERATORS]
        corr = ([f"C2c:Q0:Op9:Q0:Op9:P{moms}"]
                + [f"C3c:Q0:Op9:Q0:Op{k}:Q0:Op9:P{moms}" for k in range(9)])
        if c["n_rnd"] >= 4:  # the four-point functions need four distinct random indices
            corr += [f"{d}:Q0:Op9:Q0:Op9:Q0:Op9:Q0:Op9:P{moms}" for d in ("C4cD", "C4cB", "C4cV")]
    else:
        ops = [f"g5.d0.p{moms}"]
        corr = [f"C2c:Q0:Op0:Q0:Op0:P{moms}"]
    extra = {}
    if c["diagrams"] == "displaced":
        ops.append("g5.d%s.p0" % ",".join(_DISPLACED_OPS))
        corr.append("C2c:Q0:Op1:Q0:Op1:P0")
        extra = {"alpha1": HYP[0], "alpha2": HYP[1], "iterations": HYP[2]}
    return synthetic.Workload("case", Lt=c["Lt"], L=c["L"], nev=c["nev"], n_rnd=c["n_rnd"],
                              dilT=c["dilT"], dilE=c["dilE"], operators=ops, correlators=corr,
                              orthonormal=False, extra=extra)


def _global_data(c):
    with tempfile.TemporaryDirectory() as d:
        return GlobalData.from_infile(_workload(c).write_infile(d))


# ---------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gauss(seed, what, k, shape):
    """Complex Gaussian of a fixed stream per (seed, array, index)."""
    g = torch.Generator(device=_device())
    g.manual_seed((int(seed) * 8 + what) * 4096 + k)
    x = torch.randn(*shape, 2, dtype=torch.float64, device=_device(), generator=g)
    return torch.view_as_complex(x)


def _eigenvectors(c, seed, t):
    """Timeslice t: (nev, 3 L^3), normalised rows."""
    v = _gauss(seed, 1, t, (c["nev"], 3 * c["L"] ** 3))
    return v / torch.linalg.vector_norm(v, dim=1, keepdim=True)


def _perambulator(c, seed, r):
    return _gauss(seed, 2, r, (c["Lt"] // c["dilT"] * c["dilE"] * 4, 4 * c["nev"] * c["Lt"]))


def _noise(c, seed, r):
    x = _gauss(seed, 3, r, (c["Lt"] * 4 * c["nev"],))
    return torch.complex(torch.sign(x.real), torch.sign(x.imag)) * math.sqrt(0.5)


def _su3(m):
    """Gram-Schmidt of the rows of (..., 3, 3), completed to determinant one."""
    u1 = m[..., 0, :] / torch.linalg.vector_norm(m[..., 0, :], dim=-1, keepdim=True)
    u2 = m[..., 1, :] - (u1.conj() * m[..., 1, :]).sum(-1, keepdim=True) * u1
    u2 = u2 / torch.linalg.vector_norm(u2, dim=-1, keepdim=True)
    return torch.stack([u1, u2, torch.linalg.cross(u1, u2, dim=-1).conj()], dim=-2)


def _links(c, seed, t):
    """Links of timeslice t, [x, y, z, dir, a, b]: near the unit matrix, then
    gauge-transformed with a random SU(3) matrix per site."""
    L = c["L"]
    u = _su3(torch.eye(3, dtype=torch.complex128, device=_device())
             + 0.23 * _gauss(seed, 4, t, (L, L, L, 3, 3, 3)))
    g = _su3(_gauss(seed, 5, t, (L, L, L, 3, 3)))
    return torch.stack([g @ u[..., d, :, :] @ torch.roll(g, -1, d).mH for d in range(3)], dim=3)


def _host(x, pinned=False):
    """x on the host, as the numpy array that the setters take."""
    out = pinned_empty(tuple(x.shape)) if pinned else np.empty(tuple(x.shape), np.complex128)
    torch.from_numpy(out).copy_(x)
    return out


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "noalloc":
        fn = _lib.lib().slaph_vdaggerv_noalloc
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.POINTER(_lib.Dims), ctypes.c_void_p,
                       ctypes.POINTER(ctypes.c_int32), ctypes.c_void_p, ctypes.c_void_p]
        v = _eigenvectors(c, seed, 0).contiguous()
        return {"case": c, "fn": fn, "V": v, "out": torch.empty(
                    c["nev"], c["nev"], dtype=torch.complex128, device=_device()),
                "dims": _lib.Dims(1, c["L"], c["L"], c["L"], c["nev"], 1, 1, 1),
                "mom": (ctypes.c_int32 * 3)(c["px"], c["py"], c["pz"])}
    gd = _global_data(c)
    eng = Engine(gd.dims)
    s = {"case": c, "gd": gd, "eng": eng, "fac": OperatorFactory(eng, gd),
         "precision": MIXED if c["precision"] == "mixed" else FP64,
         "accumulator": KAHAN if c["accumulator"] == "kahan" else NATIVE}
    if c["slots"] > 0:
        eng.set_eigenvector_slots(c["slots"])
        eng.set_factor_lifetime(True)
    if c["diagrams"] == "displaced":
        L = c["L"]  # links as the gauge reader gives them: [site][dir][a + 3 b]
        s["U"] = [_host(_links(c, seed, t).transpose(-1, -2).reshape(L ** 3, 3, 9))
                  for t in range(c["Lt"])]
    peram = [_host(_perambulator(c, seed, r)) for r in range(c["n_rnd"])]
    noise = [_host(_noise(c, seed, r)) for r in range(c["n_rnd"])]
    if c["upload"]:
        s["V"] = [_host(_eigenvectors(c, seed, t), pinned=True) for t in range(c["Lt"])]
        s["peram"], s["noise"] = peram, noise
    else:
        buf = pinned_empty((c["nev"], 3 * c["L"] ** 3))
        for t in range(c["Lt"]):
            torch.from_numpy(buf).copy_(_eigenvectors(c, seed, t))
            eng.set_eigenvectors(t, buf)
        for r in range(c["n_rnd"]):
            eng.set_perambulator(r, peram[r])
            eng.set_random_vector(r, noise[r])
        if c["block_pair"] >= 0:
            s["fac"].create_operators(s["precision"])
    if torch.cuda.is_available():
        torch.cuda.empty_cache()
    return s


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "noalloc":
        stream = torch.cuda.current_stream().cuda_stream
        _lib.check(s["fn"](ctypes.byref(s["dims"]), s["V"].data_ptr(), s["mom"],
                           s["out"].data_ptr(), stream))
        return s["out"]
    eng, gd = s["eng"], s["gd"]
    if c["upload"]:
        for r in range(c["n_rnd"]):
            eng.set_perambulator(r, s["peram"][r])
            eng.set_random_vector(r, s["noise"][r])
        for t in range(c["Lt"]):
            eng.set_eigenvectors(t, s["V"][t])
    if "U" in s:
        s["fac"].set_gauge_field(s["U"])  # uploads and smears
    if c["block_pair"] < 0:
        s["fac"].create_operators(s["precision"])
    return eng.contract(gd.plan_ptr, s["precision"], s["accumulator"], c["block_pair"])


# ---------------------------------------------------------------- work
def work(case):
    c = dict(case)
    K, nev = 3 * c["L"] ** 3, c["nev"]
    if c["kind"] == "noalloc":
        return {"bytes": 16 * (nev * K + nev * nev), "flops": 8 * nev * nev * K}
    gd = _global_data(c)
    st = gd.schedule_stats(c["block_pair"])
    eds = 4 * c["dilE"]
    n_ops = gd.plan.n_vdv_ops - (1 if gd.plan.index_of_unity >= 0 else 0)
    byts = 16 * st["requests"] * c["Lt"]
    byts += 16 * c["n_rnd"] * 4 * nev * c["Lt"] * (c["Lt"] // c["dilT"] * eds + 1)
    # factors (each built from one VdaggerV block), their products and traces
    flops = 8 * (st["q0"] * 4 * c["dilE"] * nev + (st["q1"] + 4 * st["q2"]) * eds * eds * nev
                 + st["products"] * eds ** 3 + st["distinct_entries"] * eds ** 2 + st["terms"])
    if c["block_pair"] < 0:
        byts += 16 * c["Lt"] * nev * K
        flops += 8 * nev * nev * K * n_ops * c["Lt"]
    else:
        byts += 16 * c["Lt"] * nev * nev * n_ops
    if c["diagrams"] == "displaced":
        sites = c["L"] ** 3 * c["Lt"]
        byts += 16 * 27 * sites
        # per site and iteration 9 projections (about 10 3x3 products) and 36 staple products
        flops += HYP[2] * sites * (9 * 10 + 36) * 216
    return {"bytes": byts, "flops": flops}


# ---------------------------------------------------------------- exact results
def _momenta(p2):
    """Momenta up to |p|^2 = p2 in the order of the correlators."""
    n = int(math.isqrt(p2))
    r = range(-n, n + 1)
    return sorted(((x, y, z) for x in r for y in r for z in r if x * x + y * y + z * z <= p2),
                  key=lambda p: (sum(k * k for k in p), p))


def _phase(L, p):
    """exp(-i 2 pi p.x / L) per (site, colour)."""
    x = torch.arange(L, dtype=torch.float64, device=_device()) * (2 * math.pi / L)
    a = (p[0] * x[:, None, None] + p[1] * x[None, :, None] + p[2] * x[None, None, :]).reshape(-1)
    return torch.polar(torch.ones_like(a), -a).repeat_interleave(3)


def _project(m):
    """The SU(3) matrix of proj_to_su3: unitary polar factor over the cube root
    of its determinant, by Newton's iteration on the polar decomposition."""
    for _ in range(14):
        m = 0.5 * (m + torch.linalg.inv(m).mH)
    d = torch.linalg.det(m)
    return m * torch.polar(d.abs() ** (-1.0 / 3.0), -torch.angle(d) / 3.0)[..., None, None]


def _smear(u):
    """HYP smearing of one timeslice's links u[x, y, z, dir, a, b]."""
    a1, a2, n = HYP

    def at(f, d, k):
        return torch.roll(f, -k, d)

    for _ in range(n):
        U = [u[..., d, :, :] for d in range(3)]

        def staples(f, b, nd, d):  # of b (direction d) with f (direction nd)
            up = f @ at(b, nd, 1) @ at(f, d, 1).mH
            dn = f.mH @ b @ at(f, d, 1)
            return up + at(dn, nd, -1)

        dec = {(d, p): _project((1 - a2) * U[d] + a2 / 2 * staples(U[p], U[d], p, d))
               for d in range(3) for p in range(3) if p != d}
        u = torch.stack([_project((1 - a1) * U[d] + a1 / 4 * sum(
            staples(dec[nd, 3 - d - nd], dec[d, 3 - d - nd], nd, d)
            for nd in range(3) if nd != d)) for d in range(3)], dim=3)
    return u


def _displace(v, u, step):
    """D(V) for v (nev, 3 L^3): the in-place sweep of the displacement, in which
    a site reads the already displaced value of a neighbour that precedes it."""
    L = u.shape[0]
    d = "xyz".index(step[1])
    w = v.reshape(v.shape[0], L, L, L, 3).movedim(1 + d, 0).clone()
    U = u[..., d, :, :].movedim(d, 0)
    for k in range(L):
        if step[0] == ">":
            w[k] = torch.einsum("xyab,nxyb->nxya", U[k], w[(k + 1) % L])
        else:
            w[k] = torch.einsum("xyba,nxyb->nxya", U[k - 1].conj(), w[k - 1])
    return w.movedim(0, 1 + d).reshape(v.shape[0], -1)


def _two_point(c, seed):
    """[correlator, t] of the pion two-point functions (gamma_5 at both ends)."""
    L, Lt, nev, dilT, dilE, R = (c[k] for k in ("L", "Lt", "nev", "dilT", "dilE", "n_rnd"))
    nb, eds = Lt // dilT, 4 * dilE
    moms = _momenta(c["p2"])
    # (source, sink) operator index of every correlator
    pairs = [(k, moms.index(tuple(-x for x in p))) for k, p in enumerate(moms)]
    n_ops = len(moms)
    if c["diagrams"] == "displaced":
        pairs += [(n_ops + i, n_ops + j) for i in range(6) for j in range(6)]
        n_ops += 6
    phases = {p: _phase(L, p) for p in moms}
    P = [_perambulator(c, seed, r).reshape(nb, eds, Lt, 4, nev) for r in range(R)]
    rho = [_noise(c, seed, r).reshape(Lt, nev, 4) for r in range(R)]
    rnd = [(a, b) for a in range(R) for b in range(R) if a != b]
    g5 = torch.tensor([1., 1., -1., -1.], dtype=torch.float64, device=_device())
    ev = torch.arange(nev, device=_device())
    cols = (ev[:, None] % dilE == torch.arange(dilE, device=_device())[None]).to(torch.complex128)
    # q0[op][pair]: [Lt, dirac, e1, e2]; q2[op][pair]: [Lt, block, dirac, e2, e1]
    q0 = torch.empty(n_ops, len(rnd), Lt, 4, dilE, dilE, dtype=torch.complex128, device=_device())
    q2 = torch.empty(n_ops, len(rnd), Lt, nb, 4, dilE, dilE, dtype=torch.complex128,
                     device=_device())
    for t in range(Lt):
        v = _eigenvectors(c, seed, t)
        m = [None] * n_ops
        for k, p in enumerate(moms):
            q = pairs[k][1]
            if p == (0, 0, 0):  # the identity, as the eigenvectors are taken to be orthonormal
                m[k] = torch.eye(nev, dtype=torch.complex128, device=_device())
            elif m[q] is not None:
                m[k] = m[q].mH
            else:
                m[k] = v.conj() @ (phases[p] * v).mT
        if c["diagrams"] == "displaced":
            u = _smear(_links(c, seed, t))
            for k, step in enumerate(_DISPLACED_OPS):
                m[len(moms) + k] = v.conj() @ _displace(v, u, step).mT
        for k in range(n_ops):
            x = [torch.einsum("vw,badw->badv", m[k], P[r][:, :, t]) for r in range(R)]
            for j, (r1, r2) in enumerate(rnd):
                a = rho[r1][t].mT.conj()[:, :, None] * cols  # [dirac, v, e]
                b = rho[r2][t].mT[:, :, None] * cols
                q0[k, j, t] = g5[:, None, None] * (a.mT @ m[k] @ b)
                # Q2 of the pair (r2, r1); only its Dirac-diagonal blocks meet Q0
                full = torch.einsum("badv,bcdv->bac", P[r2][:, :, t].conj(), x[r1])
                for d in range(4):
                    e = slice(d * dilE, (d + 1) * dilE)
                    q2[k, j, t, :, d] = g5[d] * full[:, e, e]
    blk = torch.arange(Lt, device=_device()) // dilT
    src = torch.arange(Lt, device=_device())
    out = torch.zeros(len(pairs), Lt, dtype=torch.complex128, device=_device())
    for n, (i, j) in enumerate(pairs):
        tr = torch.einsum("ksdef,ktbdfe->tbs", q0[j], q2[i]) / len(rnd)  # [source, block, sink]
        tr = tr[:, blk, src]  # the sink's own block
        for dt in range(Lt):
            out[n, dt] = tr[src, (src - dt) % Lt].sum() / Lt
    return out


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "noalloc":
        v = _eigenvectors(c, seed, 0)
        m = v.conj() @ (_phase(c["L"], (c["px"], c["py"], c["pz"])) * v).mT
        return m.mT.contiguous()  # the blocks are column-major
    if c["diagrams"] == "pipi":
        return None
    return _two_point(c, seed).cpu().numpy()
