"""Timed workloads of the engine, each ONE call a user's program makes through hfgpu.engine.

The path is the two-electron part of a Hartree-Fock calculation on water clusters (5.5 bohr lattices and
chains of randomly rotated monomers): direct Fock builds (RHF and UHF, FP64 and mixed precision, host
arrays and device pointers, full densities and the small increments of late SCF iterations), batches of
uneven molecules, the nuclear gradient, Fock builds from stored integrals, and a whole small SCF.

Densities come from a generalized Wolfsberg-Helmholz guess (the overlap matrix and one orbital energy per
kind of shell), which has the magnitudes and the decay with distance of a converged density and is made
here in plain torch, so the inputs depend on the seed alone.
"""
import itertools
import json
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "hartree-fock_gb300")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

MONOMER = np.array([[1.4327076887, -0.9610871670, 0.0], [-1.4327076887, -0.9610871670, 0.0], [0.0, 0.2403536480, 0.0]])
MONOMER_Z = (1, 1, 8)
SPACING = 5.5
AO_PER_WATER = {"sto-3g": 7, "6-31g": 13, "6-31g**": 25, "6-311g*": 25, "6-311g**": 31, "cc-pvdz": 18}


# ------------------------------------------------------------------------------------------------- cases

def fock(name, basis, waters, precision, uhf=False, density="full", where="device"):
    return dict(name=name, kind="fock", basis=basis, waters=waters, precision=precision, uhf=uhf, density=density,
                where=where)


def listed():
    return [
        # The smallest call: one water, the input of the reference's README; launches and latency.
        fock("fock_h2o_631g_fp64", "6-31g", 1, "fp64", where="host"),
        # A small open-shell cation with d functions, as in a geometry scan: still latency.
        fock("fock_w2_ccpvdz_uhf_fp64", "cc-pvdz", 2, "fp64", uhf=True, where="host"),
        # An odd, ragged size in a triple-zeta basis, open shell, mixed precision.
        fock("fock_w7_6311gss_uhf_mixed", "6-311g**", 7, "mixed", uhf=True, where="host"),
        # The ordinary medium build in plain FP64 (every class, FP64 pipe).
        fock("fock_w16_631gss_fp64", "6-31g**", 16, "fp64"),
        # The increment of a late SCF iteration in mixed precision: mostly FP32 quartets.
        fock("fock_w27_631gss_mixed_step", "6-31g**", 27, "mixed", density="step"),
        # The largest: the first full build of the (H2O)_64 benchmark in mixed precision.
        fock("fock_w64_631gss_mixed", "6-31g**", 64, "mixed"),
        # 256 independent chains of 1 to 12 waters in one engine (one Fock build of every molecule).
        dict(name="batch256_631g_mixed", kind="batch", basis="6-31g", molecules=256, kmax=12, precision="mixed"),
        # Nuclear gradients: a small FP64 one of an optimisation, and a larger mixed one.
        dict(name="grad_w8_ccpvdz_fp64", kind="gradient", basis="cc-pvdz", waters=8, precision="fp64"),
        dict(name="grad_w16_631gss_mixed", kind="gradient", basis="6-31g**", waters=16, precision="mixed"),
        # DIRECT FALSE: one Fock build from the integrals kept on the device.
        dict(name="stored_w6_631gss", kind="stored", basis="6-31g**", waters=6, uhf=False),
        # A whole SCF of a small cluster, input to converged energy and density.
        dict(name="scf_w2_631gss_fp64", kind="scf", basis="6-31g**", waters=2),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))

    kind = rng.choice(["fock"] * 6 + ["batch", "gradient", "gradient", "stored", "scf"])
    if kind == "fock":
        basis, precision = rng.choice(sorted(AO_PER_WATER)), rng.choice(["fp64", "mixed"])
        most = (420 if precision == "fp64" else 1000) // AO_PER_WATER[basis]
        return dict(kind="fock", basis=basis, waters=spread(1, most), precision=precision, uhf=rng.random() < 0.3,
                    density=rng.choice(["full", "step"]), where=rng.choice(["host", "device"]))
    if kind == "batch":
        return dict(kind="batch", basis="6-31g", molecules=spread(16, 256), kmax=rng.randint(3, 12),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "gradient":
        precision = rng.choice(["fp64", "mixed"])
        return dict(kind="gradient", basis=rng.choice(["6-31g", "6-31g**", "cc-pvdz"]),
                    waters=spread(1, 8 if precision == "fp64" else 16), precision=precision)
    if kind == "stored":
        return dict(kind="stored", basis=rng.choice(["6-31g", "6-31g**", "cc-pvdz"]), waters=spread(1, 8),
                    uhf=rng.random() < 0.3)
    return dict(kind="scf", basis=rng.choice(["sto-3g", "6-31g", "6-31g**"]), waters=spread(1, 4))


# -------------------------------------------------------------------------------------------- molecules

def rotated(rng):
    """The monomer about its centroid, turned by a uniform random rotation."""
    w, x, y, z = (lambda q: q / np.linalg.norm(q))(rng.standard_normal(4))
    turn = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                     [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                     [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])
    return (MONOMER - MONOMER.mean(axis=0)) @ turn.T


def cluster(waters, rng):
    """The first `waters` points of a cubic lattice, each with a turned and jittered monomer."""
    side = math.ceil(waters ** (1 / 3) - 1e-9)
    points = list(itertools.product(range(side), repeat=3))[:waters]
    xyz = [rotated(rng) + np.array(p, float) * SPACING + rng.uniform(-0.2, 0.2, 3) for p in points]
    return list(MONOMER_Z) * waters, np.concatenate(xyz)


def chain(waters, rng):
    xyz = [rotated(rng) + np.array([i * SPACING, 0.0, 0.0]) for i in range(waters)]
    return list(MONOMER_Z) * waters, np.concatenate(xyz)


def molecules_of(case, seed):
    """[(Z, xyz)] of the case: one molecule, or a batch's chains (whose lengths the case fixes)."""
    rng = np.random.default_rng([seed, 77])
    if case["kind"] != "batch":
        return [cluster(case["waters"], rng)]
    lengths = np.random.default_rng(case["molecules"]).integers(1, case["kmax"] + 1, case["molecules"])
    return [chain(int(k), rng) for k in lengths]


def cartesians(l):
    return [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]


_basis_files = {}


def element_shells(basis, z):
    """[(l, exponents, coefficients)] of an element from the basis file (first contraction of each l)."""
    if basis not in _basis_files:
        with open(os.path.join(PACKAGE, "basis_sets", basis.replace("*", "_st_") + ".json")) as f:
            _basis_files[basis] = json.load(f)["elements"]
    out = []
    for sh in _basis_files[basis][str(z)]["electron_shells"]:
        ex = [float(e) for e in sh["exponents"]]
        for row, l in enumerate(sh["angular_momentum"]):
            out.append((int(l), ex, [float(c) for c in sh["coefficients"][row]][:len(ex)]))
    return out


def dfact(n):
    return math.prod(range(n, 1, -2))


def primitive_shells(basis, Z, xyz):
    """One row per primitive shell: (l, exponent, coefficient with the l-part of the norm, atom, first AO)."""
    rows, ao = [], 0
    for atom, z in enumerate(Z):
        for l, ex, co in element_shells(basis, int(z)):
            rows += [(l, a, c * (2 * a / math.pi) ** 0.75 * (4 * a) ** (l / 2), atom, ao) for a, c in zip(ex, co)]
            ao += (l + 1) * (l + 2) // 2
    return rows, ao


def component_norms(l):
    return [1 / math.sqrt(dfact(2 * i - 1) * dfact(2 * j - 1) * dfact(2 * k - 1)) for i, j, k in cartesians(l)]


# ---------------------------------------------------------------------- overlap, kinetic energy, densities

def one_centre_tables(basis, Z, xyz, dev):
    """Every primitive Cartesian function: exponent, factor, centre, powers, AO; and the AO count."""
    rows, n = primitive_shells(basis, Z, xyz)
    flat = [(a, c * nrm, *xyz[atom], *pw, ao + k) for l, a, c, atom, ao in rows
            for k, (pw, nrm) in enumerate(zip(cartesians(l), component_norms(l)))]
    t = torch.tensor(flat, dtype=torch.float64, device=dev)
    return t[:, 0], t[:, 1], t[:, 2:5], t[:, 5:8].long(), t[:, 8].long(), n


def overlap(basis, Z, xyz, dev, kinetic=False):
    """S, or (S, T), over the contracted functions (Obara-Saika recursion, one axis at a time)."""
    a, c, R, pw, ao, n = one_centre_tables(basis, Z, xyz, dev)
    p = a[:, None] + a[None, :]
    axes, kin = [], []
    for k in range(3):
        x = R[:, k]
        d = x[:, None] - x[None, :]
        PA, PB, h = -a[None, :] / p * d, a[:, None] / p * d, 0.5 / p
        s = {(0, 0): torch.sqrt(math.pi / p) * torch.exp(-a[:, None] * a[None, :] / p * d * d)}
        top = 4 if kinetic else 2
        for i in range(3):
            for j in range(top + 1):
                if j:
                    s[i, j] = PB * s[i, j - 1] + h * ((j - 1) * s[i, j - 2] if j > 1 else 0) + (
                        h * i * s[i - 1, j - 1] if i else 0)
                elif i:
                    s[i, 0] = PA * s[i - 1, 0] + (h * (i - 1) * s[i - 2, 0] if i > 1 else 0)
        S, T = torch.zeros_like(p), torch.zeros_like(p)
        for i in range(3):
            for j in range(3):
                m = (pw[:, k] == i)[:, None] & (pw[:, k] == j)[None, :]
                S = torch.where(m, s[i, j], S)
                if kinetic:
                    b = a[None, :]
                    t = -2 * b * b * s[i, j + 2] + b * (2 * j + 1) * s[i, j] - (
                        j * (j - 1) / 2 * s[i, j - 2] if j > 1 else 0)
                    T = torch.where(m, t, T)
        axes.append(S)
        kin.append(T)
    C = torch.zeros(len(a), n, dtype=torch.float64, device=dev)
    C[torch.arange(len(a), device=dev), ao] = c
    S = C.T @ (axes[0] * axes[1] * axes[2]) @ C
    if not kinetic:
        return S
    T = kin[0] * axes[1] * axes[2] + axes[0] * kin[1] * axes[2] + axes[0] * axes[1] * kin[2]
    return S, C.T @ T @ C


def shell_energies(basis, Z):
    """A rough orbital energy per AO: deep for the oxygen core, valence by l, positive for outer shells."""
    out = []
    for z in Z:
        seen = {}
        for l, ex, _ in element_shells(basis, int(z)):
            k = seen[l] = seen.get(l, -1) + 1
            if z == 1:
                e = -0.5 if l == 0 and k == 0 else 0.3 if l == 0 else 1.5
            else:
                e = [-20.5, -1.3, 0.2, 0.9][min(k, 3)] if l == 0 else [-0.6, 0.4, 1.0][min(k, 2)] if l == 1 else 2.0
            out += [e] * ((l + 1) * (l + 2) // 2)
    return torch.tensor(out, dtype=torch.float64)


def guess(basis, Z, xyz, na, nb, rng, step):
    """(D_alpha, D_beta, W) of the Wolfsberg-Helmholz guess, or with `step` the change of the densities when
    the orbital energies move by some mEh (an increment between two late SCF iterations)."""
    dev = "cuda" if torch.cuda.is_available() and len(Z) > 36 else "cpu"
    S = overlap(basis, Z, xyz, dev)
    e = shell_energies(basis, Z).to(dev)
    L = torch.linalg.cholesky(S)

    def densities(e):
        H = 0.875 * (e[:, None] + e[None, :]) * S
        H.diagonal().copy_(e * S.diagonal())
        X = torch.linalg.solve_triangular(L, H, upper=False)
        X = torch.linalg.solve_triangular(L, X.T.contiguous(), upper=False)
        w, V = torch.linalg.eigh((X + X.T) / 2)
        C = torch.linalg.solve_triangular(L.T, V, upper=True)
        Da, Db = C[:, :na] @ C[:, :na].T, C[:, :nb] @ C[:, :nb].T
        W = (C[:, :na] * w[:na]) @ C[:, :na].T + (C[:, :nb] * w[:nb]) @ C[:, :nb].T
        return [(M + M.T) / 2 for M in (Da, Db, W)]

    D = densities(e)
    if step:
        moved = e + torch.tensor(rng.standard_normal(len(e)) * 0.01, dtype=torch.float64, device=dev)
        D = [x - y for x, y in zip(densities(moved), D)]
    return [M.cpu().numpy() for M in D]


def electrons(case, Z):
    total = sum(Z) - (1 if case.get("uhf") else 0)
    return (total + 1) // 2, total // 2


def densities_of(case, seed):
    """Per molecule (Z, xyz, D_alpha, D_beta, W)."""
    rng = np.random.default_rng([seed, 78])
    out = []
    for Z, xyz in molecules_of(case, seed):
        na, nb = electrons(case, Z)
        out.append((Z, xyz, *guess(case["basis"], Z, xyz, na, nb, rng, case.get("density") == "step")))
    return out


# --------------------------------------------------------------------------------------- prepare and run

def prepare(case, seed):
    from hfgpu import basis as hb, engine as he

    s = dict(case)
    s["precision"] = he.MIXED if case.get("precision") == "mixed" else he.FP64
    if case["kind"] == "scf":
        (Z, xyz), = molecules_of(case, seed)
        s.update(Z=Z, xyz=xyz, engine=he.Engine(hb.pack(case["basis"], Z, xyz)))
        s["engine"].schwartz()
        return s
    mols = densities_of(case, seed)
    packed = [hb.pack(case["basis"], Z, xyz) for Z, xyz, *_ in mols]
    s["engine"] = he.Engine(packed if case["kind"] == "batch" else packed[0])
    s["engine"].schwartz()
    if case["kind"] == "gradient":
        s["Z"], s["xyz"], s["Da"], s["Db"], s["W"] = mols[0]
        return s
    if case["kind"] == "stored":
        s["engine"].store_integrals()
    uhf = bool(case.get("uhf"))
    mats = [[Da + Db, Da] + ([Db] if uhf else []) for _, _, Da, Db, _ in mols]
    if case["kind"] == "stored" or case.get("where") == "host":
        s["D"] = [np.asfortranarray(m) for m in mats[0]]
        return s
    # Device pointers: the molecules' blocks one after another, inputs and outputs on the GPU.
    D = [torch.from_numpy(np.concatenate([m[k].ravel() for m in mats])).cuda() for k in range(len(mats[0]))]
    s["D"], s["out"] = D, [torch.empty_like(d) for d in D]
    names = ["dD_tot", "dD_alpha", "dD_beta"], ["J", "K_alpha", "K_beta"]
    s["pointers"] = {k: t.data_ptr() for ks, ts in zip(names, (D, s["out"])) for k, t in zip(ks, ts)}
    torch.cuda.synchronize()
    return s


def run(s):
    e = s["engine"]
    if s["kind"] == "scf":
        r, Da, _ = e.scf(s["Z"], s["xyz"], opts=dict(max_iter=100, energy_tol=1e-8, density_tol=1e-7, diis_tol=1e-7))
        return {"e_total": r["e_total"], "D_alpha": Da}
    if s["kind"] == "gradient":
        return e.gradient(s["Z"], s["xyz"], s["Da"], s["Db"], s["W"], precision=s["precision"])[0]
    if s["kind"] == "stored":
        return [m for m in e.fock_conventional(*s["D"])[:3] if m is not None]
    if "pointers" in s:
        e.fock_device(s["pointers"], unrestricted=len(s["D"]) == 3, precision=s["precision"])
        return s["out"]
    return [m for m in e.fock(*s["D"], precision=s["precision"])[:3] if m is not None]


# --------------------------------------------------------------------------------------------------- work

def pair_classes(basis, Z, xyz):
    """Per shell-pair class (l1, l2): sorted Schwarz bounds of the significant pairs (their s-type primitive
    self-repulsions added up) and their mean count of significant primitive pairs."""
    shells = [(l, np.array(ex), np.abs(co), xyz[atom]) for atom, z in enumerate(Z)
              for l, ex, co in element_shells(basis, int(z))]
    kinds = {}
    for i, (l, ex, co, r) in enumerate(shells):
        kinds.setdefault((l, len(ex), ex[0]), []).append(i)
    found = {}
    for ka, kb in itertools.combinations_with_replacement(sorted(kinds), 2):
        (la, ea, ca, _), (lb, eb, cb, _) = shells[kinds[ka][0]], shells[kinds[kb][0]]
        ra, rb = (np.array([shells[i][3] for i in kinds[k]]) for k in (ka, kb))
        r2 = ((ra[:, None] - rb[None]) ** 2).sum(-1)
        r2 = r2[np.triu_indices(len(ra))] if ka == kb else r2.ravel()
        q, npp = np.zeros(len(r2)), np.zeros(len(r2))
        for (a, x), (b, y) in itertools.product(zip(ea, ca), zip(eb, cb)):
            p = a + b
            norm = x * y * (4 * a * b / math.pi ** 2) ** 0.75 * math.sqrt(2 * math.pi ** 2.5 / (p * p * math.sqrt(2 * p)))
            t = norm * np.exp(-a * b / p * r2)
            q += t
            npp += t > 1e-15
        keep = q > 1e-11
        old = found.setdefault((max(la, lb), min(la, lb)), ([], []))
        old[0].append(q[keep])
        old[1].append(npp[keep])
    return {k: (np.sort(np.concatenate(q)), float(np.concatenate(n).mean()))
            for k, (q, n) in found.items() if sum(map(len, q))}


def hermites(L):
    return (L + 1) * (L + 2) * (L + 3) // 6


def quartet_work(basis, Z, xyz, scale, gradient):
    """(surviving quartets' integrals, flops) of the McMurchie-Davidson evaluation and digestion."""
    cls = pair_classes(basis, Z, xyz)
    keys = sorted(cls, reverse=True)
    integrals = flops = 0.0
    for x, (a, b) in enumerate(keys):
        for c, d in keys[x:]:
            (q1, n1), (q2, n2) = cls[a, b], cls[c, d]
            count = float((len(q2) - np.searchsorted(q2, 1e-10 / (scale * q1))).sum()) * (0.5 if (a, b) == (c, d) else 1)
            L, nab, ncd = a + b + c + d, len(cartesians(a)) * len(cartesians(b)), len(cartesians(c)) * len(cartesians(d))
            per = 2 * math.comb(L + 4 + gradient, 4) + 2 * hermites(a + b) * ncd * hermites(c + d) + 2 * (L + 1) + 10
            per += 2 * nab * ncd * hermites(a + b)
            integrals += count * nab * ncd
            flops += count * (n1 * n2 * per * (3 if gradient else 1) + 12 * nab * ncd)
    return integrals, flops


def work(case):
    mols = molecules_of(case, 0)
    kind, spins = case["kind"], 3 if case.get("uhf") else 2
    scale = 0.02 if case.get("density") == "step" else 1.0
    sizes, nbytes, flops, seen = [], 0.0, 0.0, {}
    for Z, xyz in mols:
        if len(Z) not in seen:  # the molecules of one size differ by rotations only
            seen[len(Z)] = quartet_work(case["basis"], Z, xyz, scale, kind == "gradient")
        integrals, f = seen[len(Z)]
        n = AO_PER_WATER[case["basis"]] * len(Z) // 3
        if kind == "stored":
            nbytes, f = nbytes + 8 * integrals, 12 * integrals
        if kind == "scf":
            f *= 12  # about a dozen iterations
        nbytes += 8 * n * n * ({"gradient": 3, "scf": 2}.get(kind) or 2 * spins)
        flops += f
    return {"bytes": nbytes, "flops": flops}


# -------------------------------------------------------------------------------------- 64-bit references

def boys(m_max, T):
    """[F_0 .. F_m_max](T): the series for the top order and downward recursion, or for large T the error
    function and upward recursion."""
    small = T < 36.0
    t = torch.where(small, T, torch.ones_like(T))
    e = torch.exp(-t)
    term = torch.full_like(t, 1.0 / (2 * m_max + 1))
    total = term.clone()
    for i in range(1, 170):
        term = term * t / (m_max + i + 0.5)
        total += term
    low = {m_max: e * total}
    for m in range(m_max, 0, -1):
        low[m - 1] = (2 * t * low[m] + e) / (2 * m - 1)
    b = torch.where(small, torch.full_like(T, 40.0), T)
    e, high = torch.exp(-b), [0.5 * torch.sqrt(math.pi / b) * torch.erf(torch.sqrt(b))]
    for m in range(m_max):
        high.append(((2 * m + 1) * high[m] - e) / (2 * b))
    return [torch.where(small, low[m], high[m]) for m in range(m_max + 1)]


def hermite_integrals(L, alpha, X):
    """R_{tuv}, t+u+v <= L, for exponent alpha and distance X (3 arrays), as a dict of arrays."""
    F = boys(L, alpha * (X[0] ** 2 + X[1] ** 2 + X[2] ** 2))
    cur = {(0, 0, 0): (-2 * alpha) ** L * F[L]}
    for n in range(L - 1, -1, -1):
        new = {(0, 0, 0): (-2 * alpha) ** n * F[n]}
        for tuv in itertools.product(range(L - n + 1), repeat=3):
            if 0 < sum(tuv) <= L - n:
                k = next(i for i in range(3) if tuv[i])
                one = tuple(v - (i == k) for i, v in enumerate(tuv))
                new[tuv] = X[k] * cur[one]
                if one[k]:
                    two = tuple(v - 2 * (i == k) for i, v in enumerate(tuv))
                    new[tuv] = new[tuv] + one[k] * cur[two]
        cur = new
    return cur


def tuvs(L):
    return [t for t in itertools.product(range(L + 1), repeat=3) if sum(t) <= L]


def charge_groups(basis, Z, xyz, dev):
    """The products of contracted functions as sums of Hermite Gaussians: per total degree L (p, P, M) with
    M[AO pair i >= j, primitive pair, tuv]; and the AO pairs (i, j)."""
    rows, n = primitive_shells(basis, Z, xyz)
    ij = torch.full((n, n), -1, dtype=torch.long)
    lo = torch.tril_indices(n, n)
    ij[lo[0], lo[1]] = torch.arange(lo.shape[1])
    groups = {}
    by_l = {l: [r for r in rows if r[0] == l] for l in range(3)}
    for l1, l2 in ((0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2)):
        pairs = [(x, y) for x in by_l[l1] for y in by_l[l2] if l1 != l2 or x[4] >= y[4]]
        if not pairs:
            continue
        t = lambda f: torch.tensor([f(x, y) for x, y in pairs], dtype=torch.float64)  # noqa: E731
        a, b = t(lambda x, y: x[1]), t(lambda x, y: y[1])
        A, B = t(lambda x, y: list(xyz[x[3]])), t(lambda x, y: list(xyz[y[3]]))
        p = a + b
        P = (a[:, None] * A + b[:, None] * B) / p[:, None]
        E = []
        for k in range(3):
            e = {(0, 0, 0): torch.exp(-a * b / p * (A[:, k] - B[:, k]) ** 2)}
            get = lambda i, j, u: e.get((i, j, u), torch.zeros_like(p))  # noqa: E731
            for i in range(l1 + 1):
                for j in range(l2 + 1):
                    for u in range(i + j + 1):
                        if i:
                            e[i, j, u] = get(i - 1, j, u - 1) / (2 * p) + (P - A)[:, k] * get(i - 1, j, u) + (u + 1) * get(i - 1, j, u + 1)
                        elif j:
                            e[i, j, u] = get(i, j - 1, u - 1) / (2 * p) + (P - B)[:, k] * get(i, j - 1, u) + (u + 1) * get(i, j - 1, u + 1)
            E.append(e)
        c = t(lambda x, y: x[2] * y[2])
        hs = tuvs(l1 + l2)
        M = torch.zeros(lo.shape[1], len(pairs), len(hs), dtype=torch.float64)
        here = torch.arange(len(pairs))
        ao1, ao2 = (torch.tensor([q[s][4] for q in pairs]) for s in (0, 1))
        for i, (pi, ni) in enumerate(zip(cartesians(l1), component_norms(l1))):
            for j, (pj, nj) in enumerate(zip(cartesians(l2), component_norms(l2))):
                r, s = ao1 + i, ao2 + j
                # A shell with itself lists each AO pair twice: keep the half with r >= s.
                at = ij[torch.maximum(r, s), torch.minimum(r, s)]
                w = torch.where((ao1 == ao2) & (r < s), 0.0, 1.0) * c * ni * nj
                for h, (x, y, z) in enumerate(hs):
                    if (pi[0], pj[0], x) in E[0] and (pi[1], pj[1], y) in E[1] and (pi[2], pj[2], z) in E[2]:
                        M[at, here, h] += w * E[0][pi[0], pj[0], x] * E[1][pi[1], pj[1], y] * E[2][pi[2], pj[2], z]
        groups.setdefault(l1 + l2, []).append((p, P, M))
    out = {L: (torch.cat([g[0] for g in v]).to(dev), torch.cat([g[1] for g in v]).to(dev),
               torch.cat([g[2] for g in v], 1).to(dev)) for L, v in groups.items()}
    return out, lo.to(dev), n


def repulsion_tensor(basis, Z, xyz, dev):
    """(ij|kl) over all AOs, n x n x n x n."""
    groups, lo, n = charge_groups(basis, Z, xyz, dev)
    npair = lo.shape[1]
    V = torch.zeros(npair, npair, dtype=torch.float64, device=dev)
    for L1, (p, P, M1) in groups.items():
        for L2, (q, Q, M2) in groups.items():
            h1, h2 = tuvs(L1), tuvs(L2)
            sign = torch.tensor([(-1.0) ** sum(t) for t in h2], dtype=torch.float64, device=dev)
            step = max(1, int(4e7 / (len(q) * (len(h1) * len(h2) + 2 * hermites(L1 + L2)))))
            for b in range(0, len(p), step):
                pp, X = p[b:b + step, None], P[b:b + step, None] - Q[None]
                R = hermite_integrals(L1 + L2, pp * q / (pp + q), [X[..., k] for k in range(3)])
                pref = 2 * math.pi ** 2.5 / (pp * q * torch.sqrt(pp + q))
                block = torch.stack([torch.stack([R[tuple(x + y for x, y in zip(t, u))] for u in h2], -1) for t in h1], 1)
                block = block * pref[:, None, :, None] * sign
                half = M1[:, b:b + step].reshape(npair, -1) @ block.reshape(-1, len(q) * len(h2))
                V += half @ M2.reshape(npair, -1).T
    full = torch.zeros(n, n, npair, dtype=torch.float64, device=dev)
    full[lo[0], lo[1]] = V
    full[lo[1], lo[0]] = V
    out = torch.zeros(n, n, n, n, dtype=torch.float64, device=dev)
    out[:, :, lo[0], lo[1]] = full
    out[:, :, lo[1], lo[0]] = full
    return out


def attraction(basis, Z, xyz, dev):
    groups, lo, n = charge_groups(basis, Z, xyz, dev)
    V = torch.zeros(n, n, dtype=torch.float64, device=dev)
    C = torch.tensor(np.asarray(xyz), dtype=torch.float64, device=dev)
    charge = torch.tensor([float(z) for z in Z], dtype=torch.float64, device=dev)
    for L, (p, P, M) in groups.items():
        X = P[:, None] - C[None]
        R = hermite_integrals(L, p[:, None].expand(-1, len(Z)), [X[..., k] for k in range(3)])
        v = torch.stack([-(2 * math.pi / p) * (R[t] @ charge) for t in tuvs(L)], 1)
        half = M.reshape(M.shape[0], -1) @ v.reshape(-1)
        V[lo[0], lo[1]] += half
        V[lo[1], lo[0]] += half * (lo[0] != lo[1])
    return V


def closed_shell(basis, Z, xyz, dev):
    """Converged RHF energy and alpha density, with DIIS."""
    S, T = overlap(basis, Z, xyz, dev, kinetic=True)
    h, g = T + attraction(basis, Z, xyz, dev), repulsion_tensor(basis, Z, xyz, dev)
    s, U = torch.linalg.eigh(S)
    X, occ = U / torch.sqrt(s), sum(Z) // 2
    F, Fs, errs = h, [], []
    for _ in range(200):
        _, C = torch.linalg.eigh(X.T @ F @ X)
        C = (X @ C)[:, :occ]
        D = C @ C.T
        F = h + 2 * torch.einsum("ijkl,kl->ij", g, D) - torch.einsum("ikjl,kl->ij", g, D)
        energy = ((h + F) * D).sum()
        err = X.T @ (F @ D @ S - S @ D @ F) @ X
        if err.abs().max() < 1e-12:
            break
        Fs, errs = (Fs + [F])[-8:], (errs + [err])[-8:]
        k = len(Fs)
        B = torch.ones(k + 1, k + 1, dtype=torch.float64)
        B[:k, :k] = torch.tensor([[float((x * y).sum()) for x in errs] for y in errs])
        B[:k, :k] /= B[:k, :k].abs().max()
        B[k, k] = 0.0
        c = torch.linalg.lstsq(B, torch.tensor([[0.0]] * k + [[1.0]], dtype=torch.float64), driver="gelsd").solution
        F = sum(float(c[i]) * Fs[i] for i in range(k))
    nuclear = sum(Z[i] * Z[j] / np.linalg.norm(xyz[i] - xyz[j]) for i in range(len(Z)) for j in range(i))
    return float(energy) + float(nuclear), D.cpu().numpy()


def exact(case, seed):
    """J and K (or the converged SCF) from the whole integral tensor in 64 bits, without screening; None for
    gradients and for molecules whose tensor takes over about 20 s."""
    if case["kind"] not in ("fock", "stored", "scf") or AO_PER_WATER[case["basis"]] * case["waters"] > 60:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "scf":
        (Z, xyz), = molecules_of(case, seed)
        e, D = closed_shell(case["basis"], Z, xyz, dev)
        return {"e_total": e, "D_alpha": D}
    (Z, xyz, Da, Db, _), = densities_of(case, seed)
    g = repulsion_tensor(case["basis"], Z, xyz, dev)
    D = [torch.from_numpy(d).to(dev) for d in ([Da + Db, Da] + ([Db] if case["uhf"] else []))]
    out = [torch.einsum("ijkl,kl->ij", g, D[0])] + [torch.einsum("ikjl,kl->ij", g, d) for d in D[1:]]
    if case.get("where") == "device":
        return [m.reshape(-1) for m in out]
    return [m.cpu().numpy() for m in out]
