"""The engine's workloads as measurable cases.

A case is one call (or a short sequence of calls) that a program using the
framework makes for one wavefunction: load the MOs with their integrals (or the
primitive list) into a context and solve, ask for a response property, or push
a batch of wavefunctions through the request server.  Each pass starts from
host arrays and ends with host arrays, as the engine's callers see it, so a
pass includes the upload and everything formed once per wavefunction (S^1/2).
The contexts and the server are opened once per process and serve every
wavefunction that comes, as in a running program.

Molecules are synthetic with a minimal basis: STO-3G clusters and chains of
C/N/O/H and graphene flakes with the valence part, MOs S^-1/2 Q with Q a Haar
random rotation, orbital energies spread evenly with a random shift of each
(occupied -0.8..-0.2 Eh, virtual 0..0.6 Eh).  The geometry belongs to the size; the MOs, the energies and, for
clusters, the atom positions follow the seed.

What the listed cases stand for:

* ``window_benzene``      the smallest call: every root below E_thr of benzene
                          (no root count given, the keyword default), FP64 form
* ``roots_cluster20``     the small end of a batch of molecules, where latency
                          and launches count: 20 roots
* ``roots_cluster61``     the median molecule of a request stream, 32 roots,
                          integrals formed on the device from the primitives
* ``roots_cluster141``    the large end of a batch of molecules, 20 roots
* ``alpha_cluster57``     alpha(w) at three frequencies of a stream request
                          (iterative solve)
* ``alpha_chain200``      alpha(w) of a 200-atom chain at five frequencies
* ``beta_cluster33``      hyperpolarizability at w = 0 and two wavelengths
                          (dense A+B, A-B)
* ``stddft_cluster26``    sTD-DFT roots (subspace solver of both A+B and A-B)
* ``uks_cluster37``       open-shell wavefunction, 20 roots
* ``flake8_mixed``        the large solve: C384H48, 50 roots, mixed form
* ``flake7_fp64``         a large solve in the FP64 form: C294H42, 50 roots
* ``served_batch``        16 molecules of 20 to 150 atoms through the request
                          server at once
"""
from __future__ import annotations

import math

import numpy as np
import torch

from stda_b200 import synth
from stda_b200.engine import (BoundaryInputs, Engine, Keywords, PrimInputs, Server, primitives)
from stda_b200.molden import BOHR_ANGSTROM, Molecule

EV = 27.211385050
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _case(name, kind, shape, natoms, e_thr, **kw):
    c = dict(name=name, kind=kind, shape=shape, natoms=natoms, e_thr=e_thr, ax=0.5, precision=1,
             nroots=0, solver=0, conv_tol=0.0, nomega=0, route="integrals", triplet=False,
             kshift=False, count=1)
    c.update(kw)
    return c


def listed():
    return [
        _case("window_benzene", "roots", "benzene", 12, 7.0, precision=0),
        _case("roots_cluster20", "roots", "cluster", 20, 6.5, nroots=20, conv_tol=1e-7),
        _case("roots_cluster61", "roots", "cluster", 61, 6.5, nroots=32, conv_tol=1e-7,
              route="primitives"),
        _case("roots_cluster141", "roots", "cluster", 141, 6.5, nroots=20, conv_tol=1e-7),
        _case("alpha_cluster57", "alpha", "cluster", 57, 6.5, solver=2, nomega=3),
        _case("alpha_chain200", "alpha", "chain", 200, 7.0, nomega=5),
        _case("beta_cluster33", "beta", "cluster", 33, 6.5, nomega=2),
        _case("stddft_cluster26", "stddft", "cluster", 26, 6.5, precision=0, nroots=10,
              conv_tol=1e-7),
        _case("uks_cluster37", "uks", "cluster", 37, 6.5, nroots=20, conv_tol=1e-7),
        _case("flake8_mixed", "roots", "flake", 8, 7.0, nroots=50),
        _case("flake7_fp64", "roots", "flake", 7, 7.0, precision=0, nroots=50),
        _case("served_batch", "served", "cluster", 20, 6.5, nroots=20, conv_tol=1e-7, count=16),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["window", "roots", "roots", "roots", "alpha", "alpha", "chain", "beta",
                       "stddft", "uks", "flake", "served"])
    ethr = round(rng.uniform(6.2, 7.2), 2)
    ax = rng.choice([0.25, 0.5, 0.5, 0.75])
    prec = rng.choice([0, 1])
    if kind == "window":
        n = size(12, 36)
        c = _case("", "roots", "cluster", n, round(ethr + 24.0 / n, 2), ax=ax, precision=prec,
                  kshift=rng.random() < 0.3)
    elif kind == "roots":
        c = _case("", "roots", "cluster", size(16, 141), ethr, ax=ax, precision=prec,
                  nroots=rng.choice([8, 20, 32, 45]), conv_tol=1e-7,
                  route=rng.choice(["integrals", "primitives"]), triplet=rng.random() < 0.2,
                  kshift=rng.random() < 0.2)
    elif kind == "alpha":
        c = _case("", "alpha", "cluster", size(16, 120), ethr, ax=rng.choice([0.25, 0.5]),
                  precision=prec, solver=2, nomega=rng.randint(1, 5))
    elif kind == "chain":
        c = _case("", "alpha", "chain", size(60, 200), ethr, nomega=rng.randint(1, 5))
    elif kind == "beta":
        c = _case("", "beta", "cluster", size(12, 36), ethr, ax=ax, precision=prec,
                  nomega=rng.randint(1, 3))
    elif kind == "stddft":
        c = _case("", "stddft", "cluster", size(12, 32), ethr, precision=prec,
                  nroots=rng.choice([5, 8, 10]), conv_tol=1e-7)
    elif kind == "uks":
        c = _case("", "uks", "cluster", size(12, 56), ethr, precision=prec,
                  nroots=rng.choice([8, 20, 32]), conv_tol=1e-7)
    elif kind == "flake":
        n = rng.randint(3, 8) if prec else rng.randint(3, 6)
        c = _case("", "roots", "flake", n, ethr, precision=prec, nroots=rng.choice([20, 35, 50]))
    else:
        c = _case("", "served", "cluster", 20, ethr, nroots=rng.choice([8, 20]), conv_tol=1e-7,
                  count=rng.randint(6, 18))
    del c["name"]
    return c


# ------------------------------------------------------------------ molecules
def _cluster(natoms, rng):
    """Compact C/N/O/H cluster: heavy atoms 1.45 A from an earlier one, H 1.09 A."""
    nheavy = max(1, (2 * natoms) // 3)
    pts = [np.zeros(3)]
    while len(pts) < nheavy:
        v = rng.standard_normal(3)
        c = pts[rng.integers(len(pts))] + 1.45 * v / np.linalg.norm(v)
        if np.min(np.linalg.norm(np.array(pts) - c, axis=1)) > 1.3:
            pts.append(c)
    heavy = np.array(pts)
    Z = [(6, 6, 6, 6, 6, 6, 6, 7, 7, 8)[k % 10] for k in range(nheavy)]
    hs = []
    tries = 0
    while len(hs) < natoms - nheavy and tries < 100000:
        tries += 1
        v = rng.standard_normal(3)
        c = heavy[rng.integers(nheavy)] + 1.09 * v / np.linalg.norm(v)
        if np.min(np.linalg.norm(heavy - c, axis=1)) > 1.0 and (
                not hs or np.min(np.linalg.norm(np.array(hs) - c, axis=1)) > 1.5):
            hs.append(c)
    xyz = np.vstack([heavy, np.array(hs)]) if hs else heavy
    return xyz, np.array(Z + [1] * len(hs), dtype=np.int32)


def _molecule(shape, natoms, rng):
    if shape == "benzene":
        t = math.pi / 3 * np.arange(6)
        ring = np.stack([np.cos(t), np.sin(t), 0 * t], axis=1)
        xyz, Z = np.vstack([1.39 * ring, 2.48 * ring]), np.array([6] * 6 + [1] * 6, np.int32)
    elif shape == "flake":
        C3, H3 = synth.flake_geometry(natoms)
        xyz, Z = np.vstack([C3, H3]), np.array([6] * len(C3) + [1] * len(H3), np.int32)
    elif shape == "chain":
        xyz, Z = synth.chain_geometry(natoms)
    else:
        xyz, Z = _cluster(natoms, rng)
    return Molecule(Z=Z, xyz=xyz / BOHR_ANGSTROM,
                    shells=synth.basis_shells(Z, valence_only=shape == "flake"), title=shape)


def _ao_integrals(mol):
    """S, -r, -d/dr (ket) and r x d/dr over the contracted s and p functions, FP64."""
    fn = mol.ao_functions()
    t = lambda v: torch.tensor(np.array(v), dtype=torch.float64, device=DEV)  # noqa: E731
    at = [f[0] for f in fn]
    R, lmn = t(mol.xyz[at]), t([f[1] for f in fn])
    ex, co = t([f[2] for f in fn]), t([f[3] for f in fn])
    n = len(fn)
    out = torch.zeros(10, n, n, dtype=torch.float64, device=DEV)
    A, B = R[:, None, :], R[None, :, :]
    AB2 = ((A - B) ** 2).sum(-1)
    la, lb = lmn[:, None, :] > 0.5, lmn[None, :, :] > 0.5
    for ka in range(ex.shape[1]):
        for kb in range(ex.shape[1]):
            a, b = ex[:, ka, None], ex[None, :, kb]
            p = a + b
            w = co[:, ka, None] * co[None, :, kb] * torch.exp(-a * b / p * AB2) * (math.pi / p) ** 1.5
            h = 0.5 / p
            S, Mo, De = [], [], []
            for d in range(3):
                P = (a * A[..., d] + b * B[..., d]) / p
                pa, pb = P - A[..., d], P - B[..., d]
                e02 = pb * pb + h
                one = torch.ones_like(p)
                e0 = torch.where(la[..., d], pa, one)                       # ket power 0
                e1 = torch.where(la[..., d], pa * pb + h, pb)               # ket power 1
                e2 = torch.where(la[..., d], pa * e02 + 2 * h * pb, e02)    # ket power 2
                s = torch.where(lb[..., d], e1, e0)
                up = torch.where(lb[..., d], e2, e1)
                S.append(s)
                Mo.append(up + B[..., d] * s)
                De.append(-2 * b * up + torch.where(lb[..., d], e0, 0 * e0))
            out[0] += w * S[0] * S[1] * S[2]
            for d in range(3):
                f, g = (d + 1) % 3, (d + 2) % 3
                out[1 + d] -= w * Mo[d] * S[f] * S[g]
                out[4 + d] -= w * De[d] * S[f] * S[g]
                out[7 + d] += w * S[d] * (Mo[f] * De[g] - Mo[g] * De[f])
    return out


def _haar(n, rng):
    q, r = torch.linalg.qr(torch.tensor(rng.standard_normal((n, n)), device=DEV))
    return q * torch.sign(torch.diagonal(r))


def _wavefunction(case, natoms, seed):
    """Molecule, its AO integrals (10 x nao x nao) and MOs, energies, occupations, spins."""
    rng = np.random.default_rng([int(seed), natoms])
    mol = _molecule(case["shape"], natoms, rng)
    ints = _ao_integrals(mol)
    n = ints.shape[1]
    nocc = (int(mol.Z.sum()) - (2 * int((mol.Z > 2).sum()) if case["shape"] == "flake" else 0)) // 2
    if case["shape"] == "flake" and natoms == 8:
        nocc = 780
    L = torch.linalg.cholesky(0.5 * (ints[0] + ints[0].T))
    nel = [nocc] if case["kind"] != "uks" else [nocc + 1, nocc]
    C, eps, occ, csp = [], [], [], []
    for sp, ne in enumerate(nel):
        C.append(torch.linalg.solve_triangular(L.T, _haar(n, rng), upper=True).cpu().numpy())
        level = lambda m: 0.6 * (np.arange(m) + rng.random(m)) / m  # noqa: E731
        eps += [level(ne) - 0.8, level(n - ne)]
        occ += [np.full(ne, 2.0 / len(nel)), np.zeros(n - ne)]
        csp += [np.full(n, sp + 1, dtype=np.int32)]
    return (mol, ints, np.asfortranarray(np.hstack(C)), np.concatenate(eps), np.concatenate(occ),
            np.concatenate(csp))


def _inputs(case, natoms, seed):
    mol, ints, C, eps, occ, csp = _wavefunction(case, natoms, seed)
    xyz4 = np.ascontiguousarray(np.hstack([mol.xyz, mol.Z[:, None].astype(np.float64)]))
    if case["route"] == "primitives":
        return PrimInputs(xyz4, C, eps, occ, primitives(mol)), csp
    i, j = np.tril_indices(ints.shape[1])
    pk = ints[:, torch.tensor(i, device=DEV), torch.tensor(j, device=DEV)].cpu().numpy()
    return BoundaryInputs(xyz4=xyz4, C=C, eps=eps, occ=occ,
                          iaoat1=np.ascontiguousarray(mol.iaoat() + 1, dtype=np.int32), S=pk[0].copy(),
                          muL=pk[1:4].copy(), muV=pk[4:7].copy(), muM=pk[7:10].copy()), csp


# -------------------------------------------------------------------- one pass
_open = {}


def _engine(precision):
    if precision not in _open:
        _open[precision] = Engine(0, precision)
    return _open[precision]


def _server():
    if "server" not in _open:
        _open["server"] = Server(0, 1, slots=8)
    return _open["server"]


def _keywords(case):
    return Keywords(ax=case["ax"], e_thr_ev=case["e_thr"], nroots=case["nroots"],
                    solver=case["solver"], conv_tol=case["conv_tol"], triplet=case["triplet"],
                    kshift=case["kshift"], rpa=case["kind"] == "stddft")


def _frequencies(case):
    """Evenly spaced from 0 to 0.06 Eh, below the first excitation."""
    return [0.06 * q / max(1, case["nomega"] - 1) for q in range(case["nomega"])]


def _sizes(case):
    """Atoms of every molecule of the case (a batch: 20 to 150, log-uniform)."""
    k = case["count"]
    if k == 1:
        return [case["natoms"]]
    return [int(round(case["natoms"] * (141.0 / case["natoms"]) ** (q / (k - 1)))) for q in range(k)]


def prepare(case, seed):
    state = dict(case=case, kw=_keywords(case), om=_frequencies(case),
                 inputs=[_inputs(case, n, seed + 1000 * q) for q, n in enumerate(_sizes(case))])
    state["handle"] = _server() if case["kind"] == "served" else _engine(case["precision"])
    return state


def _hash(sols):
    return np.array([[s.nci, s.csf_hash & 0xffffffff, s.csf_hash >> 32] for s in sols], np.int64)


def _pairs(occ):
    return int((occ > 1.0).sum() * (occ < 1.0).sum())


def _padded(x, room):
    """The rows of x, and zeros up to the number of occupied-virtual pairs."""
    out = np.zeros((room,) + x.shape[1:], x.dtype)
    out[:len(x)] = x
    return out


def _energies_only(case):
    # The mixed form's large solve stops at a residual of 1e-6, and its first
    # stage runs on rounded operands: the intensities of its closest roots
    # (1e-5 Eh apart) are defined to about residual / gap only, and a change of
    # 1e-16 in the inputs moves them by 1e-5.  Its energies, CSF space and
    # lowered diagonal do not depend on that.
    return case["precision"] == 1 and case["shape"] == "flake"


def run(state):
    case, kw, h = state["case"], state["kw"], state["handle"]
    if case["kind"] == "served":
        tickets = [h.submit(b, kw) for b, _ in state["inputs"]]
        sols = [h.wait(t)[0] for t in tickets]
        cat = lambda f: np.concatenate([getattr(s, f) for s in sols])  # noqa: E731
        return {"csf": _hash(sols), **{f: cat(f) for f in ("omega", "fL", "fV", "RL", "RV", "alpha0")}}
    b, csp = state["inputs"][0]
    if isinstance(b, PrimInputs):
        h.load_prims(b.xyz4, b.C, b.eps, b.occ, b.prims)
    else:
        h.load(b)
    if case["kind"] == "alpha":
        return {"alpha": h.polarizability(kw, state["om"])[0]}
    if case["kind"] == "beta":
        _, beta, hrs = h.hyperpolarizability(kw, [1064.0 + 200.0 * q for q in range(case["nomega"])])
        return {"beta": beta, "hrs": hrs}
    if case["kind"] == "uks":
        h.set_spins(csp)
    s = h.solve(kw)
    if _energies_only(case):
        iconf, ed = h.csf()
        room = _pairs(b.occ)
        return {"csf": _padded(iconf, room), "ed": _padded(ed, room), "omega": s.omega}
    out = {"omega": s.omega, "fL": s.fL, "fV": s.fV, "RL": s.RL, "RV": s.RV}
    if case["nroots"] == 0:      # a window: as many roots as there are
        out = {k: _padded(x, _pairs(b.occ)) for k, x in out.items()}
    return {"csf": _hash([s]), "alpha0": s.alpha0, **out}


# ------------------------------------------------------------- work and checks
def work(case):
    """Inputs and outputs once, and the contractions the path is made of: MO
    transforms, gamma products, the couplings of every candidate with every
    primary, and one product with the CI matrix per root (or right-hand side)."""
    nbytes = flops = 0.0
    for natoms in _sizes(case):
        if case["shape"] == "flake":
            N, nao = 6 * natoms ** 2 + 6 * natoms, 24 * natoms ** 2 + 6 * natoms
            occ, virt = 0.5 * nao, 0.5 * nao
        else:
            N = natoms
            h = natoms / 4 if case["shape"] == "chain" else natoms - (2 * natoms) // 3
            if case["shape"] == "benzene":
                h = 6
            nao = 5 * (N - h) + h
            occ = 0.5 * (6.5 * (N - h) + h) if case["shape"] != "benzene" else 21
            virt = nao - occ
        if case["kind"] == "uks":
            occ, virt = 2 * occ, 2 * virt
        thr = case["e_thr"] / EV
        frac = min(1.0, max(0.05, (2 * (1 + 0.8 * case["ax"]) * thr - 0.2) / 0.6))
        no, nv = frac * occ, frac * virt
        t = min(0.6, max(0.05, thr - 0.2 + 1.0 / math.sqrt(N)))
        nov = no * nv * (0.5 if case["kind"] == "uks" else 1.0)
        nex = max(1.0, 0.5 * (t / 0.6) ** 2 * occ * virt * (0.5 if case["kind"] == "uks" else 1.0))
        ints = 10 * nao * (nao + 1) / 2 if case["route"] == "integrals" else 15 * nao
        nbytes += 8 * (ints + nao * (occ + virt) + 6 * N)
        if case["kind"] == "alpha":
            nvec, nbytes = 3 * case["nomega"], nbytes + 72 * case["nomega"]
        elif case["kind"] == "beta":
            nvec, nbytes = 6 * (case["nomega"] + 1), nbytes + 224 * (case["nomega"] + 1)
        else:
            nvec = case["nroots"] or nex
            nbytes += 8 * 5 * nvec
        flops += 2 * 9 * nao * nv * (nao + no) + 2 * N * N * (nov + no * no / 2)
        flops += 2 * 2 * N * nex * nov
        flops += nvec * 2 * (2 * N * nov / 4 + nao * no * (2 * nv + no))
    return {"bytes": nbytes, "flops": flops}


_ETA = {1: 0.472592880, 6: 0.421954120, 7: 0.504381930, 8: 0.586918630}


def exact(case, seed):
    """The same quantities in FP64 from the definitions: dense A, A+B and A-B,
    complete eigen-decompositions and direct solves."""
    nao = 4 * max(_sizes(case))
    if case["shape"] == "flake" or case["kind"] == "served" or (nao > 440 and case["kind"] != "alpha"):
        return None
    mol, ints, C, eps, occ, csp = _wavefunction(case, case["natoms"], seed)
    uks, ax = case["kind"] == "uks", case["ax"]
    resp = case["kind"] in ("alpha", "beta")
    rpa = resp or case["kind"] == "stddft"
    ak = 1.0 if uks else (0.0 if case["triplet"] else 2.0)
    thr = case["e_thr"] / EV
    T = lambda v: torch.tensor(np.ascontiguousarray(v), device=DEV)  # noqa: E731
    # orbital window
    is_o, is_v = occ > (0.99 if uks else 1.99), occ < 0.01
    deps = 2 * (1 + 0.8 * ax) * thr
    sel = lambda m: np.concatenate([q[np.argsort(eps[q], kind="stable")] for q in  # noqa: E731
                                    (np.nonzero(m & (csp == s))[0] for s in (1, 2))])
    o = sel(is_o & (eps > eps[is_v].min() - deps))
    v = sel(is_v & (eps < eps[is_o].max() + deps))
    no, nv = len(o), len(v)
    sym = lambda q: torch.tril(q) + torch.tril(q, -1).T  # noqa: E731
    anti = lambda q: torch.tril(q, -1) - torch.tril(q, -1).T  # noqa: E731
    S = sym(ints[0])
    w, U = torch.linalg.eigh(S)
    Sh = (U * w.sqrt()) @ U.T
    Co, Cv = T(C[:, o]), T(C[:, v])
    Lo, Lv = Sh @ Co, Sh @ Cv
    ops = [sym(ints[1 + q]) if q < 3 else anti(ints[1 + q]) for q in range(9)]
    mu = torch.stack([Co.T @ q @ Cv for q in ops])
    # charges and damped Coulomb kernels
    atom = mol.iaoat()
    N = len(mol.Z)
    eta = T(np.array([_ETA[int(z)] for z in mol.Z]))
    R = torch.cdist(T(mol.xyz), T(mol.xyz), compute_mode="donot_use_mm_for_euclid_dist")
    eb = 0.5 * (eta[:, None] + eta[None, :])
    al, be = 1.420 + 0.480 * ax, 0.20 + 1.830 * ax
    gj = (R ** be + (ax * eb) ** (-be)) ** (-1 / be)
    gk = (R ** al + eb ** (-al)) ** (-1 / al)

    def charges(X, Y):
        q = torch.zeros(N, X.shape[1], Y.shape[1], dtype=torch.float64, device=DEV)
        for A in range(N):
            k = torch.tensor(np.nonzero(atom == A)[0], device=DEV)
            q[A] = X[k].T @ Y[k]
        return q

    qia, qij, qab = charges(Lo, Lv), charges(Lo, Lo), charges(Lv, Lv)
    so, sv = T(csp[o]), T(csp[v])
    same = so[:, None] == sv[None, :]
    qia, qij, qab = (qia * same, qij * (so[:, None] == so[None, :]),
                     qab * (sv[:, None] == sv[None, :]))
    pia = torch.einsum("AB,Bia->Aia", gk, qia)
    pij = torch.einsum("AB,Bij->Aij", gj, qij)
    jd = torch.einsum("Ai,Aa->ia", torch.diagonal(pij, dim1=1, dim2=2),
                      torch.diagonal(qab, dim1=1, dim2=2))
    ek = (pia * qia).sum(0)
    de = T(eps[v])[None, :] - T(eps[o])[:, None] - jd + ak * ek
    if case["kshift"]:
        au = 0.036749320
        de = de + 0.5 * au / (1.0 + (ek / (0.1 * au)) ** 4)
    # primaries, candidates and their PT sums
    prim = torch.nonzero((de <= thr) & same)
    ed = de[prim[:, 0], prim[:, 1]]
    ed, k = torch.sort(ed, stable=True)
    prim = prim[k]
    cand = torch.nonzero((de > thr) & same)
    dc = de[cand[:, 0], cand[:, 1]]
    P, Q = pia.reshape(N, -1), qia.reshape(N, -1)
    flat = lambda c: c[:, 0] * nv + c[:, 1]  # noqa: E731

    def coulomb(x, y):
        J = torch.zeros(len(x), len(y), dtype=torch.float64, device=DEV)
        for A in range(N):
            J += pij[A][x[:, 0]][:, y[:, 0]] * qab[A][x[:, 1]][:, y[:, 1]]
        return J

    a = ak * (P[:, flat(cand)].T @ Q[:, flat(prim)]) - coulomb(cand, prim)
    t = a * a / (dc[:, None] - ed[None, :] + 1e-10)
    keep = t.sum(1) > 1e-4
    csf = torch.cat([prim, cand[keep]])
    dia = torch.cat([ed - t[~keep].sum(0), dc[keep]])
    del a, t
    ekd = ek[csf[:, 0], csf[:, 1]]
    K, J = P[:, flat(csf)].T @ Q[:, flat(csf)], coulomb(csf, csf)
    Kx = torch.zeros_like(K)
    if rpa or case["kind"] != "alpha":
        for A in range(N):
            Kx += pia[A][csf[:, 0]][:, csf[:, 1]] * qia[A][csf[:, 0]][:, csf[:, 1]].T
    m = mu[:, csf[:, 0], csf[:, 1]].T.contiguous()        # nci x 9
    D = lambda q: torch.diag_embed(q - 0)  # noqa: E731
    off = lambda q: q - D(torch.diagonal(q))  # noqa: E731
    if rpa:
        apb = off(2 * ak * K - ax * Kx - J) + D(dia - ax * ekd + ak * ekd)
        amb = off(ax * Kx - J) + D(dia - ak * ekd + ax * ekd)
    if resp:
        nw = case["nomega"]
        oms = (_frequencies(case) if case["kind"] == "alpha" else
               sum([[x, -2 * x] for x in [0.0] + [45.56335 / (1064.0 + 200.0 * q) for q in range(nw)]], []))
        ainv = torch.cholesky_inverse(torch.linalg.cholesky(amb))
        Us = [torch.linalg.solve(apb - x * x * ainv, -2.0 * m[:, :3]) for x in oms]
        if case["kind"] == "alpha":
            return {"alpha": torch.stack([-2.0 * m[:, :3].T @ u for u in Us]).cpu()}
        moo, mvv = [Co.T @ q @ Co for q in ops[:3]], [Cv.T @ q @ Cv for q in ops[:3]]
        XY = [(0.5 * (u + x * (ainv @ u)), 0.5 * (u - x * (ainv @ u))) for u, x in zip(Us, oms)]

        def trip(x, y):          # G[a, c, b] = x_a . (M_c y_b)
            box = torch.zeros(3, no, nv, dtype=torch.float64, device=DEV)
            box[:, csf[:, 0], csf[:, 1]] = y.T
            my = torch.stack([box @ mvv[c] - moo[c] @ box for c in range(3)])
            return torch.einsum("ua,cbu->acb", x, my[:, :, csf[:, 0], csf[:, 1]]).cpu().numpy()

        beta = np.zeros((nw + 1, 3, 3, 3))
        for k in range(nw + 1):
            (X1, Y1), (X2, Y2) = XY[2 * k], XY[2 * k + 1]
            g21, g12, g11 = trip(X2, Y1), trip(X1, Y2), trip(X1, Y1)
            for x in range(3):
                for y in range(3):
                    for z in range(3):
                        beta[k, x, y, z] = (g21[x, y, z] + g21[x, z, y] + g12[y, z, x] + g11[y, x, z] +
                                            g11[z, x, y] + g12[z, y, x])
        return {"beta": beta, "hrs": None}
    if rpa:
        w, U = torch.linalg.eigh(amb)
        h = (U * w.sqrt()) @ U.T
        w2, Zv = torch.linalg.eigh(h @ apb @ h)
        om = w2.clamp(min=0).sqrt()
        k = case["nroots"]
        om, Zv = om[:k], Zv[:, :k]
        X = h @ Zv / om.sqrt()
        Y = apb @ X / om
        TL, TV = X.T @ m, Y.T @ m
    else:
        om, X = torch.linalg.eigh(off(ak * K - J) + D(dia))
        k = case["nroots"] or int(((om > 0) & (om <= thr)).sum())
        om, X = om[:k], X[:, :k]
        TL = TV = X.T @ m
        T2 = ((0.5 * ak * K - 0.5 * ax * Kx) @ X / (om + 1e-8)).T @ m
    l, ve, ma = TL[:, :3], TV[:, 3:6], TV[:, 6:]
    ef, rot = 1.0 / (om + 1e-8), -235.7220
    out = {"csf": None, "omega": om, "fL": 2.0 / 3.0 * om * ak * (l * l).sum(1),
           "fV": 2.0 / 3.0 * ef * ak * (ve * ve).sum(1), "RL": rot * ak * (l * ma).sum(1)}
    if rpa:
        out["RV"] = rot * ak * ef * (ve * ma).sum(1)
    else:
        em = 1.0 / (om ** (1.0 - torch.exp(-150.0 * om * om)) + 1e-8)
        out["RV"] = rot * ak * em * ((ve + T2[:, 3:6]) * ma + ve * T2[:, 6:]).sum(1)
    a0 = 2.0 * ak * (l.T * ef) @ l
    out["alpha0"] = torch.stack([a0[0, 0], a0[0, 1], a0[1, 1], a0[0, 2], a0[1, 2], a0[2, 2]])
    out = {q: (x.cpu().numpy() if x is not None else None) for q, x in out.items()}
    if not case["nroots"]:
        for q in ("omega", "fL", "fV", "RL", "RV"):
            out[q] = _padded(out[q], _pairs(occ))
    return out
