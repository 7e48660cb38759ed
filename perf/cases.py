"""The work a user of unomol_gb300 has it do, as measurable cases.

Every case goes through the public Python entry points (unomol_gb300.native, unomol_gb300.learned) on
synthetic molecules of the repository's own generators (unomol_gb300.molecules): rigid water clusters
and all-trans alkanes in STO-3G / 6-31G, the polarised basis being 6-31G with one d shell on every
heavy atom and one p shell on every hydrogen.

kind "fock"          one Fock build of one molecule (RHF, or UHF for an odd electron count)
kind "batch"         one Fock build of many molecules at once
kind "store"         one Fock build from the integrals kept in device memory
kind "scf"           a step of a geometry scan: recalculate, one-electron integrals, SCF to convergence
kind "one_electron"  overlap, kinetic and core Hamiltonian matrices of many geometries
kind "mlp"           forward and backward pass of the density network's MLP
"""
import math

import numpy as np
import torch

from unomol_gb300 import learned, molecules, native
from unomol_gb300.basis import Basis

# ---------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------


def _fock(name, system, n, basis="6-31G", charge=0, precision="fp64", density="full", entry="device", polar=False):
    c = {"kind": "fock", "system": system, "n": n, "basis": basis, "charge": charge, "precision": precision,
         "density": density, "entry": entry, "polar": polar}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one formGmatrix of a water molecule on host arrays, as the drop-in class makes
        # it once per SCF iteration of a small molecule; launches and copies are all of it
        _fock("water-sto3g-host", "water", 1, basis="STO-3G", entry="host"),
        # an open-shell molecule of ordinary size through the host entry point: the n-decane cation
        _fock("decane-uhf-host", "alkane", 10, charge=1, entry="host"),
        # the largest plain build: the 32-water cluster, FP64, device pointers
        _fock("water32-fp64", "water", 32),
        # the same cluster in the precision form: the full density of a rebuild, and the small density
        # difference of the incremental builds between rebuilds
        _fock("water32-mixed-full", "water", 32, precision="mixed"),
        _fock("water32-mixed-difference", "water", 32, precision="mixed", density="difference"),
        # a polarised basis: d shells on the oxygens, p shells on the hydrogens
        _fock("water4-polarised", "water", 4, polar=True),
        # many molecules of uneven size in one build, FP64 and in the precision form
        {"name": "batch256-fp64", "kind": "batch", "n": 256, "precision": "fp64"},
        {"name": "batch256-mixed", "kind": "batch", "n": 256, "precision": "mixed"},
        # the conventional build: integrals computed once and streamed from device memory
        {"name": "water16-stored", "kind": "store", "n": 16},
        # a whole step of a geometry scan
        {"name": "water8-scf-step", "kind": "scf", "n": 8},
        # one-electron integrals of the perturbed geometries that the density network is trained on
        {"name": "decane-one-electron-16", "kind": "one_electron", "n": 10, "geometries": 16},
        # one training pass of the density network: the rows of 16 n-decane molecules
        {"name": "mlp-13856-rows", "kind": "mlp", "rows": 13856},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["fock", "fock", "fock", "fock", "batch", "store", "scf", "one_electron", "mlp"])
    if kind == "fock":
        system = rng.choice(["water", "alkane"])
        polar = rng.random() < 0.2
        n = _log_int(rng, 1, 4 if system == "water" else 2) if polar else _log_int(rng, 1, 32 if system == "water" else 10)
        return _fock(None, system, n, basis="6-31G" if polar else rng.choice(["STO-3G", "6-31G"]), charge=rng.choice([0, 0, 1]),
                     precision=rng.choice(["fp64", "fp64", "mixed"]), density=rng.choice(["full", "difference"]),
                     entry=rng.choice(["host", "device"]), polar=polar)
    if kind == "batch":
        return {"kind": "batch", "n": _log_int(rng, 2, 256), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "store":
        return {"kind": "store", "n": _log_int(rng, 1, 16)}
    if kind == "scf":
        return {"kind": "scf", "n": _log_int(rng, 2, 8)}
    if kind == "one_electron":
        return {"kind": "one_electron", "n": rng.randint(1, 10), "geometries": _log_int(rng, 1, 64)}
    return {"kind": "mlp", "rows": _log_int(rng, 100, 30000)}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------

_MIXED = (1e-3, 1e-13)  # FP32 cutoff and density skip of the precision form, as bench.py runs it


def _atoms(system, n, seed):
    if system == "water":
        return molecules.water_cluster(n, seed)
    return molecules.perturb(molecules.alkane(n), 0.05, seed)


def _text(system, n, basis, seed, charge=0, polar=False):
    """patin text of one molecule; polar adds a d shell to every heavy atom and a p shell to every H."""
    atoms = _atoms(system, n, seed)
    text = molecules.patin_text(atoms, basis, charge=charge)
    if not polar:
        return text
    lines = text.rstrip("\n").split("\n")
    nshell, norb, ncen, _ = (int(v) for v in lines[0].split())
    for c, (e, _) in enumerate(atoms):
        l, a = (1, 1.1) if e == "H" else (2, 0.8)
        lines += [f"{1:4d}{l:4d}{c:6d}", f"{a:20.10f}{1.0:20.10f}"]
        norb += (l + 1) * (l + 2) // 2
    lines[0] = f"{nshell + len(atoms):7d}{norb:7d}{ncen:7d}{2:3d}"
    return "\n".join(lines) + "\n"


class _Mol:
    """patin text as plain arrays: shells (l, exponents, normalised coefficients, centre), centres."""

    def __init__(self, text):
        tok = text.split()
        nshell, self.norb, ncen, _, self.nelec = (int(t) for t in tok[:5])
        cen = np.array([float(t) for t in tok[15:15 + 4 * ncen]]).reshape(ncen, 4)
        self.charges, self.centers = cen[:, 0].copy(), cen[:, 1:].copy()
        p = 15 + 4 * ncen
        self.shells = []
        for _ in range(nshell):
            k, l, c = int(tok[p]), int(tok[p + 1]), int(tok[p + 2])
            v = np.array([float(t) for t in tok[p + 3:p + 3 + 2 * k]]).reshape(k, 2)
            p += 3 + 2 * k
            a, w = v[:, 0], v[:, 1]
            s = 2.0 ** 1.5 * np.sum(np.outer(w, w) * (np.sqrt(np.outer(a, a)) / (a[:, None] + a[None])) ** (1.5 + l))
            self.shells.append((l, a, w / math.sqrt(s) * (2 * a) ** ((1.5 + l) / 2) / math.pi ** 0.75, c))
        self.lmax = max(s[0] for s in self.shells)


def _carts(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _norm(c):
    d = (1.0, 1.0, 3.0)
    return 1.0 / math.sqrt(d[c[0]] * d[c[1]] * d[c[2]])


def _table1d(a, A, lmax):
    """1D overlaps s[i][j] of all primitive pairs, unit prefactors: a [n], A [n] -> arrays [n, n]."""
    p = a[:, None] + a[None, :]
    X = A[:, None] - A[None, :]
    s = [[None] * (lmax + 1) for _ in range(lmax + 1)]
    s[0][0] = np.sqrt(np.pi / p) * np.exp(-a[:, None] * a[None, :] / p * X * X)
    PA, PB, o = -a[None, :] / p * X, a[:, None] / p * X, 0.5 / p
    for i in range(lmax + 1):
        for j in range(lmax + 1):
            if i > 0:
                v = PA * s[i - 1][j]
                v = v + (i - 1) * o * s[i - 2][j] if i > 1 else v
                v = v + j * o * s[i - 1][j - 1] if j > 0 else v
            elif j > 0:
                v = PB * s[0][j - 1]
                v = v + (j - 1) * o * s[0][j - 2] if j > 1 else v
            else:
                continue
            s[i][j] = v
    return s


def _ao_maps(m):
    """Primitive shells and the map from basis functions to them: exponents, centres, per primitive
    function its primitive shell and powers, and the contraction matrix [primitive functions, functions]."""
    alpha, cen, ps, pw, rows = [], [], [], [], []
    f = 0
    for l, a, w, c in m.shells:
        for k in range(len(a)):
            alpha.append(a[k])
            cen.append(c)
            for q, xyz in enumerate(_carts(l)):
                ps.append(len(alpha) - 1)
                pw.append(xyz)
                rows.append((f + q, w[k] * _norm(xyz)))
        f += (l + 1) * (l + 2) // 2
    C = np.zeros((len(rows), m.norb))
    for r, (i, w) in enumerate(rows):
        C[r, i] = w
    return np.array(alpha), np.array(cen), np.array(ps), np.array(pw), C


def _overlap(m):
    alpha, cen, ps, pw, C = _ao_maps(m)
    S = np.ones((len(ps), len(ps)))
    for ax in range(3):
        t = np.array(_table1d(alpha, m.centers[cen, ax], m.lmax))
        S *= t[pw[:, ax][:, None], pw[:, ax][None, :], ps[:, None], ps[None, :]]
    return C.T @ S @ C


def _density(m, nocc, shift, seed):
    """Closed-shell density of an extended-Hueckel Hamiltonian (the size, decay and block structure of an
    SCF density without running one): P = C_occ C_occ^T, trace(P S) = nocc.  `shift` perturbs the
    orbital levels with the seed's random numbers."""
    S = _overlap(m)
    h = []
    for l, a, _, c in m.shells:
        z = m.charges[c]
        if z < 1.5:
            v = -0.5 if l == 0 else 0.8
        else:
            v = (-0.33 * z * z if a.max() > 40.0 * z / 6 and len(a) > 2 else -1.2) if l == 0 else -0.6 if l == 1 else 1.5
        if len(a) == 1 and l < 2:
            v *= 0.6
        h += [v] * ((l + 1) * (l + 2) // 2)
    h = np.array(h)
    if shift:
        h = h * (1.0 + shift * np.random.default_rng(seed + 77).standard_normal(len(h)))
    H = 0.875 * S * (h[:, None] + h[None, :])
    H[np.diag_indices(len(h))] = h
    s, U = np.linalg.eigh(S)
    X = U / np.sqrt(s)
    _, W = np.linalg.eigh(X.T @ H @ X)
    Cm = X @ W[:, :nocc]
    P = Cm @ Cm.T
    return np.ascontiguousarray(P[np.tril_indices(len(h))])


def _densities(case, text, seed):
    """The packed densities of one build: [P] (RHF) or [Pa, Pb] (UHF)."""
    m = _Mol(text)
    occ = [m.nelec // 2] if m.nelec % 2 == 0 else [(m.nelec + 1) // 2, m.nelec // 2]
    Ps = [_density(m, n, 0.02, seed) for n in occ]
    if case["density"] == "difference":  # two successive iterates of a converging SCF
        Ps = [P - _density(m, n, 0.02 + 1e-4, seed) for P, n in zip(Ps, occ)]
    return Ps


def _fock_text(case, seed):
    return _text(case["system"], case["n"], case["basis"], seed, case["charge"], case["polar"])


def _batch_texts(case, seed):
    """The batching workload's mix (half alkanes C1..C8, half clusters of 1..6 waters, STO-3G or 6-31G by
    a coin flip; the mix is fixed by the number of molecules) at the seed's geometries."""
    rng, n, out = np.random.default_rng(case["n"]), case["n"], []
    for i in range(n):
        basis = "STO-3G" if rng.integers(2) == 0 else "6-31G"
        system, k = ("alkane", int(rng.integers(1, 9))) if i < n // 2 else ("water", int(rng.integers(1, 7)))
        out.append(_text(system, k, basis, 1000 * seed + i))
    return out


def _random_projector(n, nocc, rng):
    q, _ = np.linalg.qr(rng.normal(size=(n, max(nocc, 1))))
    return np.ascontiguousarray((0.9 * q @ q.T)[np.tril_indices(n)])


def _batch_density(bases, seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([_random_projector(b.norb, b.nelec // 2, rng) for b in bases])


def _mlp_inputs(case, seed):
    """Rows as the density network sees them: one-hot elements and Gaussian radial features; dL/dy small."""
    rng = np.random.default_rng(seed)
    r = case["rows"]
    x = np.zeros((r, 20), np.float32)
    x[np.arange(r), rng.integers(0, 2, r)] = 1.0
    x[np.arange(r), 2 + rng.integers(0, 2, r)] = 1.0
    d = rng.uniform(0.0, 15.0, r)
    x[:, 4:] = np.exp(-(d[:, None] - np.arange(16)[None]) ** 2)
    return x, (rng.standard_normal((r, 48)) * 1e-3).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "stream": torch.cuda.Stream()}
    if kind == "fock":
        text = _fock_text(case, seed)
        b = Basis(text=text)
        t = native.TwoElectronInts(b)
        if case["precision"] == "mixed":
            t.set_precision(native.PREC_MIXED, _MIXED[0])
            t.set_density_screening(_MIXED[1])
        st.update(t=t, entry=case["entry"], P=_densities(case, text, seed))
        if case["entry"] == "device":
            st["P"] = [torch.from_numpy(p).cuda() for p in st["P"]]
            st["G"] = [torch.empty_like(p) for p in st["P"]]
    elif kind == "store":
        c = {"density": "full"}
        text = _text("water", case["n"], "6-31G", seed)
        t = native.TwoElectronInts(Basis(text=text))
        t.store_integrals(native.STORE_RHF)
        P = [torch.from_numpy(p).cuda() for p in _densities(c, text, seed)]
        st.update(kind="fock", entry="device", t=t, P=P, G=[torch.empty_like(P[0])])
    elif kind == "batch":
        bases = [Basis(text=t) for t in _batch_texts(case, seed)]
        bat = native.Batch(bases)
        if case["precision"] == "mixed":
            bat.set_precision(native.PREC_MIXED, *_MIXED)
        P = torch.from_numpy(_batch_density(bases, seed)).cuda()
        st.update(bat=bat, P=P, G=torch.empty_like(P))
    elif kind == "scf":
        text = _text("water", case["n"], "6-31G", seed)
        b = Basis(text=text)
        st.update(b=b, t=native.TwoElectronInts(b), P0=_densities({"density": "full"}, text, seed)[0])
    elif kind == "one_electron":
        b = Basis(text=_text("alkane", case["n"], "6-31G", seed))
        rng = np.random.default_rng(seed)
        st.update(b=b, centers=b.centers[None] + rng.normal(scale=0.05, size=(case["geometries"],) + b.centers.shape))
    else:
        x, dy = _mlp_inputs(case, seed)
        st.update(m=learned.Mlp(20, 256, 3, 48, seed=seed % 1000), x=torch.from_numpy(x).cuda(), dy=torch.from_numpy(dy).cuda(),
                  y=torch.empty(case["rows"], 48, device="cuda"))
    return st


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------


def run(st):
    kind = st["kind"]
    if kind == "fock":
        t = st["t"]
        if st["entry"] == "host":
            return {"G": list(t.form_g_uhf(*st["P"])) if len(st["P"]) == 2 else [t.form_g(st["P"][0])]}
        s = st["stream"]
        with torch.cuda.stream(s):
            for g in st["G"]:
                g.zero_()
        ptr = [x.data_ptr() for x in st["P"] + st["G"]]
        (t.fock_device_uhf if len(ptr) == 4 else t.fock_device)(*ptr, s.cuda_stream)
        return {"G": st["G"]}
    if kind == "batch":
        st["bat"].fock_device(st["P"].data_ptr(), st["G"].data_ptr(), native.BATCH_GRAPH, st["stream"].cuda_stream)
        return {"G": st["G"]}
    if kind == "scf":
        b, t = st["b"], st["t"]
        t.recalculate(b)
        S, H = native.one_electron_gpu(b)
        r = native.scf(t, b, S=S, H=H, accel=native.SCF_DIIS, conv_type=0, eps=1e-10, diis_tol=1e-8, maxits=100,
                       guess_P=st["P0"], density=native.DENSITY_PSEUDO)
        return {"S": S, "H": H, "energy": r["energy"], "P": r["P"], "levels": r["orbital_energies"]}
    if kind == "one_electron":
        S, T, H = native.one_electron_gpu(st["b"], st["centers"], with_t=True)
        return {"S": S, "T": T, "H": H}
    m = st["m"]
    m.forward(st["x"], st["y"])
    m.backward(st["dy"])
    return {"y": st["y"], "grads": m.grads()}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------


def _build_flops(t, Ps):
    """Operations of one build, counted by the context's own work counters."""
    t.set_counting(True)
    (t.form_g_uhf if len(Ps) == 2 else t.form_g)(*Ps)
    t.set_counting(False)
    return t.stats()["eri_flops"]


def work(case):
    kind = case["kind"]
    if kind == "fock":
        st = prepare(dict(case, entry="host"), 1)
        fl = _build_flops(st["t"], st["P"])
        st["t"].close()
        return {"bytes": 2.0 * sum(p.nbytes for p in st["P"]), "flops": fl}
    if kind == "store":
        t = native.TwoElectronInts(Basis(text=_text("water", case["n"], "6-31G", 1)))
        t.store_integrals(native.STORE_RHF)
        i, no2 = t.store_info(), t.basis.no2
        t.close()
        return {"bytes": float(i["bytes"] + 16 * no2), "flops": 2.0 * i["nonzeros"]}
    if kind == "batch":
        bases = [Basis(text=t) for t in _batch_texts(case, 1)]
        P, off, fl = _batch_density(bases, 1), 0, 0.0
        for b in bases:
            t = native.TwoElectronInts(b)
            if case["precision"] == "mixed":
                t.set_precision(native.PREC_MIXED, _MIXED[0])
                t.set_density_screening(_MIXED[1])
            fl += _build_flops(t, [np.ascontiguousarray(P[off:off + b.no2])])
            off += b.no2
            t.close()
        return {"bytes": 16.0 * off, "flops": fl}
    if kind == "scf":
        st = prepare(case, 1)
        fl, b = _build_flops(st["t"], [st["P0"]]), st["b"]
        st["t"].close()
        its = 12  # builds of a typical convergence; about 12 N^3 of matrix products and one eigen-solve each
        return {"bytes": 8.0 * 6 * b.no2, "flops": its * (fl + 24.0 * b.norb ** 3)}
    if kind == "one_electron":
        m = _Mol(_text("alkane", case["n"], "6-31G", 1))
        k = sum(len(a) * (2 * l + 1) for l, a, _, _ in m.shells)
        no2, g = m.norb * (m.norb + 1) // 2, case["geometries"]
        return {"bytes": 8.0 * g * (3 * no2 + m.centers.size), "flops": g * 0.5 * k * k * (60.0 + 60.0 * len(m.charges))}
    r, w = case["rows"], 20 * 256 + 2 * 256 * 256 + 256 * 48
    # rows in, rows out and their gradient, parameters in, gradients out; one product forward, two backward
    return {"bytes": 4.0 * (r * (20 + 48 + 48) + 2 * (w + 3 * 256 + 48)), "flops": 6.0 * r * w}


# ---------------------------------------------------------------------------------------------
# the same results in 64 bits, without the package
# ---------------------------------------------------------------------------------------------


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _boys(mmax, T):
    """F_0 .. F_mmax (T): series for the highest order below T = 40 and downward recursion; above, the
    asymptotic F_0 (exact to 1e-18 there) and upward recursion."""
    e = torch.exp(-T)
    Ts = torch.clamp(T, max=40.0)
    term = torch.full_like(T, 1.0 / (2 * mmax + 1))
    acc = term.clone()
    for k in range(1, 150):
        term = term * (2.0 * Ts / (2 * mmax + 2 * k + 1))
        acc += term
    lo = [None] * (mmax + 1)
    lo[mmax] = acc * torch.exp(-Ts)
    for m in range(mmax - 1, -1, -1):
        lo[m] = (2.0 * Ts * lo[m + 1] + torch.exp(-Ts)) / (2 * m + 1)
    big = T > 40.0
    Tb = torch.clamp(T, min=40.0)
    hi = 0.5 * torch.sqrt(math.pi / Tb)
    out = []
    for m in range(mmax + 1):
        out.append(torch.where(big, hi, lo[m]))
        hi = ((2 * m + 1) * hi - e) / (2.0 * Tb)
    return out


def _boys_quartet(L, T):
    """The moments a quartet of total angular momentum L is built from.  A two-root quartet (L = 2, 3) with
    15 < T <= 40 is evaluated by default with unomol's own large-T nodes and weights (its Rys::root2),
    whose moments sum_i w_i x_i^m stand in the place of F_m."""
    F = _boys(L, T)
    if L not in (2, 3):
        return F
    on = (T > 15.0) & (T <= 40.0)
    Tc = torch.clamp(T, 15.0, 40.0)
    r1, r2, w2 = 0.275255128608411, 2.72474487139158, 0.0917517095361369
    g, w0 = torch.exp(-Tc), torch.sqrt(0.785398163397448 / Tc)
    u = [(-0.87894730749888 * Tc + 10.9243702330261) * g + r1 / (Tc - r1),
         (-9.28903924275977 * Tc + 81.0642367843811) * g + r2 / (Tc - r2)]
    wb = (4.468573893084 * Tc - 77.9250653461045) * g + w2 * w0
    x = [v / (1.0 + v) for v in u]
    return [torch.where(on, (w0 - wb) * x[0] ** m + wb * x[1] ** m, F[m]) for m in range(L + 1)]


def _herm(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _hermite_coefs(la, lb, PA, PB, o):
    """E[i][j][t] of one axis for all primitive pairs (unit prefactor)."""
    E = [[[None] * (la + lb + 2) for _ in range(lb + 1)] for _ in range(la + 1)]
    one, zero = torch.ones_like(PA), torch.zeros_like(PA)

    def get(i, j, t):
        return zero if t < 0 or t > i + j else E[i][j][t]

    E[0][0][0] = one
    for i in range(la + 1):
        for j in range(lb + 1):
            for t in range(i + j + 1):
                if i > 0:
                    E[i][j][t] = PA * get(i - 1, j, t) + o * get(i - 1, j, t - 1) + (t + 1) * get(i - 1, j, t + 1)
                elif j > 0:
                    E[i][j][t] = PB * get(i, j - 1, t) + o * get(i, j - 1, t - 1) + (t + 1) * get(i, j - 1, t + 1)
    return E


def _r_tuv(L, F, a, PC):
    """Hermite Coulomb integrals R_tuv, t + u + v <= L, from the moments F and exponent a."""
    R = {}
    m2 = -2.0 * a
    pw = torch.ones_like(a)
    base = []
    for n in range(L + 1):
        base.append(pw * F[n])
        pw = pw * m2
    for n in range(L, -1, -1):
        new = {}
        for t, u, v in _herm(L - n):
            if t + u + v == 0:
                new[t, u, v] = base[n]
            else:
                ax = 0 if t else 1 if u else 2
                k = [t, u, v]
                k[ax] -= 1
                r = PC[ax] * R[tuple(k)]
                if k[ax] > 0:
                    c = k[ax]
                    k[ax] -= 1
                    r = r + c * R[tuple(k)]
                new[t, u, v] = r
        R = new
    return R


def _pair_classes(m):
    """Per class (la >= lb) of unique shell pairs: primitive exponents p, centres P, Hermite coefficients
    [primitive pairs, components, Hermites] with contraction and norms, and packed indices of the functions."""
    dev = _dev()
    off, f = [], 0
    for s in m.shells:
        off.append(f)
        f += (s[0] + 1) * (s[0] + 2) // 2
    cls = {}
    for i, A in enumerate(m.shells):
        for j, B in enumerate(m.shells[:i + 1]):
            k, l = (i, j) if A[0] >= B[0] else (j, i)
            cls.setdefault((m.shells[k][0], m.shells[l][0]), []).append((k, l))
    out = []
    for (la, lb), pairs in sorted(cls.items()):
        rows, seg = [], []
        for q, (k, l) in enumerate(pairs):
            _, a, wa, ca = m.shells[k]
            _, b, wb, cb = m.shells[l]
            aa, bb = np.repeat(a, len(b)), np.tile(b, len(a))
            ww = np.repeat(wa, len(b)) * np.tile(wb, len(a))
            A, B = m.centers[ca], m.centers[cb]
            rows.append(np.column_stack([aa, bb, ww, np.broadcast_to(A, (len(aa), 3)), np.broadcast_to(B, (len(aa), 3))]))
            seg += [q] * len(aa)
        r = torch.from_numpy(np.concatenate(rows)).to(dev)
        a, b, w, A, B = r[:, 0], r[:, 1], r[:, 2], r[:, 3:6], r[:, 6:9]
        p = a + b
        P = (a[:, None] * A + b[:, None] * B) / p[:, None]
        K = w * torch.exp(-a * b / p * ((A - B) ** 2).sum(1))
        E = [_hermite_coefs(la, lb, P[:, x] - A[:, x], P[:, x] - B[:, x], 0.5 / p) for x in range(3)]
        hs = _herm(la + lb)
        comps = [(x, y) for x in _carts(la) for y in _carts(lb)]
        M = torch.zeros(len(p), len(comps), len(hs), dtype=torch.float64, device=dev)
        for c, (x, y) in enumerate(comps):
            n = _norm(x) * _norm(y)
            for h, tuv in enumerate(hs):
                if all(tuv[d] <= x[d] + y[d] for d in range(3)):
                    M[:, c, h] = K * n * E[0][x[0]][y[0]][tuv[0]] * E[1][x[1]][y[1]][tuv[1]] * E[2][x[2]][y[2]][tuv[2]]
        idx = np.array([[(lambda i, j: max(i, j) * (max(i, j) + 1) // 2 + min(i, j))(off[k] + x, off[l] + y)
                         for x in range((la + 1) * (la + 2) // 2) for y in range((lb + 1) * (lb + 2) // 2)] for k, l in pairs])
        out.append({"L": la + lb, "p": p, "P": P, "M": M, "hs": hs, "seg": torch.tensor(seg, device=dev),
                    "idx": torch.from_numpy(idx).to(dev)})
    return out


def _eri(m):
    """All integrals (ij|kl) as a symmetric matrix over packed pairs."""
    dev = _dev()
    cls = _pair_classes(m)
    no2 = m.norb * (m.norb + 1) // 2
    V = torch.zeros(no2, no2, dtype=torch.float64, device=dev)
    for x, a in enumerate(cls):
        for b in cls[:x + 1]:
            L = a["L"] + b["L"]
            nb = len(b["p"])
            step = max(1, int(2.0e8 / (nb * (8 + len(_herm(L)) + len(a["hs"]) * len(b["hs"]) / 2))))
            npb = b["idx"].shape[0]
            col = torch.zeros(a["idx"].shape[0], a["M"].shape[1], npb, b["M"].shape[1], dtype=torch.float64, device=dev)
            for i in range(0, len(a["p"]), step):
                p, P, M, seg = (a[k][i:i + step] for k in ("p", "P", "M", "seg"))
                q, Q = b["p"], b["P"]
                s = p[:, None] + q[None]
                rho = p[:, None] * q[None] / s
                D = [P[:, None, d] - Q[None, :, d] for d in range(3)]
                F = _boys_quartet(L, rho * (D[0] ** 2 + D[1] ** 2 + D[2] ** 2))
                pre = 2.0 * math.pi ** 2.5 / (p[:, None] * q[None] * torch.sqrt(s))
                R = _r_tuv(L, [f * pre for f in F], rho, D)
                for h, t in enumerate(a["hs"]):
                    # ket contraction per bra Hermite, primitives of a ket pair summed, then the bra
                    k = torch.stack([R[t[0] + u[0], t[1] + u[1], t[2] + u[2]] * (-1.0) ** sum(u) for u in b["hs"]], 2)
                    ket = torch.einsum("pqh,qch->pqc", k, b["M"])
                    kc = torch.zeros(len(p), npb, ket.shape[2], dtype=torch.float64, device=dev).index_add_(1, b["seg"], ket)
                    add = M[:, :, h][:, :, None, None] * kc[:, None]
                    col.index_add_(0, seg, add)
            r, c = a["idx"].reshape(-1), b["idx"].reshape(-1)
            blk = col.reshape(len(r), len(c))
            V[r[:, None], c[None]] = blk
            V[c[:, None], r[None]] = blk.T
    return V


def _square(P, n):
    M = torch.zeros(n, n, dtype=torch.float64, device=P.device)
    i, j = torch.tril_indices(n, n, device=P.device)
    M[i, j] = P
    M[j, i] = P
    return M


def _form_g(m, Ps):
    n, V = m.norb, _eri(m)
    dev = V.device
    i, j = torch.tril_indices(n, n, device=dev)
    full = torch.empty(n, n, dtype=torch.int64, device=dev)
    full[i, j] = torch.arange(len(i), device=dev)
    full[j, i] = full[i, j].clone()
    D = [_square(torch.from_numpy(np.asarray(p, np.float64)).to(dev), n) for p in Ps]
    w = torch.where(i == j, 1.0, 2.0).to(torch.float64)
    Dj = 2.0 * D[0] if len(D) == 1 else D[0] + D[1]
    J = V @ (w * Dj[i, j])
    out = []
    for d in D:
        K = torch.zeros(n, n, dtype=torch.float64, device=dev)
        for k in range(n):  # K_kl = sum_bd (kb|ld) D_bd
            K[k] = torch.einsum("bld,bd->l", V[full[k]][:, full], d)
        out.append((J - K[i, j]).cpu().numpy())
    return out


def _one_electron(m, centers):
    """S, T, H packed for one geometry."""
    dev = _dev()
    m.centers = centers
    alpha, cen, ps, pw, C = _ao_maps(m)
    t = [np.array(_table1d(alpha, centers[cen, ax], m.lmax + 1)) for ax in range(3)]
    a, b = alpha[ps][:, None], alpha[ps][None, :]

    def s1(ax, di, dj):
        i, j = pw[:, ax] + di, pw[:, ax] + dj
        v = t[ax][np.maximum(i, 0)[:, None], np.maximum(j, 0)[None, :], ps[:, None], ps[None, :]]
        return v * ((i >= 0)[:, None] & (j >= 0)[None, :])

    s0 = [s1(ax, 0, 0) for ax in range(3)]
    k0 = []
    for ax in range(3):
        i, j = pw[:, ax][:, None], pw[:, ax][None, :]
        k0.append(0.5 * (4 * a * b * s1(ax, 1, 1) + i * j * s1(ax, -1, -1) - 2 * a * j * s1(ax, 1, -1) - 2 * b * i * s1(ax, -1, 1)))
    S = C.T @ (s0[0] * s0[1] * s0[2]) @ C
    T = C.T @ (k0[0] * s0[1] * s0[2] + s0[0] * k0[1] * s0[2] + s0[0] * s0[1] * k0[2]) @ C
    V = torch.zeros(m.norb * (m.norb + 1) // 2, dtype=torch.float64, device=dev)
    X, Z = torch.from_numpy(np.ascontiguousarray(centers)).to(dev), torch.from_numpy(m.charges).to(dev)
    for c in _pair_classes(m):
        PC = [c["P"][:, None, d] - X[None, :, d] for d in range(3)]
        p = c["p"][:, None].expand(-1, len(Z)).contiguous()
        F = _boys(c["L"], p * (PC[0] ** 2 + PC[1] ** 2 + PC[2] ** 2))
        R = _r_tuv(c["L"], [f * (-2.0 * math.pi / p * Z[None]) for f in F], p, PC)
        v = torch.einsum("pch,ph->pc", c["M"], torch.stack([R[h].sum(1) for h in c["hs"]], 1))
        blk = torch.zeros(c["idx"].shape, dtype=torch.float64, device=dev).index_add_(0, c["seg"], v)
        V[c["idx"].reshape(-1)] = blk.reshape(-1)
    i, j = np.tril_indices(m.norb)
    return S[i, j], T[i, j], T[i, j] + V.cpu().numpy()


def _mlp_exact(case, seed):
    m = learned.Mlp(20, 256, 3, 48, seed=seed % 1000)  # the initial weights are inputs
    p = m.params()
    m.close()
    x, dy = (torch.from_numpy(v).double().to(_dev()) for v in _mlp_inputs(case, seed))
    dims, W, k = [20, 256, 256, 256, 48], [], 0
    for di, do in zip(dims[:-1], dims[1:]):
        W.append([torch.from_numpy(p[k:k + di * do].reshape(do, di)).double().to(x.device).requires_grad_(),
                  torch.from_numpy(p[k + di * do:k + di * do + do]).double().to(x.device).requires_grad_()])
        k += di * do + do
    h = x
    for n, (w, b) in enumerate(W):
        h = h @ w.T + b
        if n < 3:
            h = torch.nn.functional.silu(h)
    g = torch.autograd.grad(h, [v for wb in W for v in wb], dy)
    return {"y": h.detach(), "grads": torch.cat([v.reshape(-1) for v in g])}


def exact(case, seed):
    kind = case["kind"]
    if kind == "fock":
        text = _fock_text(case, seed)
        m = _Mol(text)
        return {"G": _form_g(m, _densities(case, text, seed))} if m.norb <= 140 else None
    if kind == "store":
        text = _text("water", case["n"], "6-31G", seed)
        m = _Mol(text)
        return {"G": _form_g(m, _densities({"density": "full"}, text, seed))} if m.norb <= 140 else None
    if kind == "scf":
        m = _Mol(_text("water", case["n"], "6-31G", seed))
        S, _, H = _one_electron(m, m.centers)
        return {"S": S, "H": H, "energy": None, "P": None, "levels": None}
    if kind == "one_electron":
        m = _Mol(_text("alkane", case["n"], "6-31G", seed))
        rng = np.random.default_rng(seed)
        cen = m.centers[None] + rng.normal(scale=0.05, size=(case["geometries"],) + m.centers.shape)
        r = [_one_electron(m, c) for c in cen]
        return {k: np.array([v[i] for v in r]) for i, k in enumerate("STH")}
    if kind == "batch":
        texts = _batch_texts(case, seed)
        if sum(_Mol(t).norb for t in texts) > 200:
            return None
        bases = [Basis(text=t) for t in texts]
        P, off, G = _batch_density(bases, seed), 0, []
        for b, t in zip(bases, texts):
            G += _form_g(_Mol(t), [P[off:off + b.no2]])
            off += b.no2
        return {"G": np.concatenate(G)}
    return _mlp_exact(case, seed)
