"""The calls whose speed matters to a user of the engine, with their inputs.

listed() names them, draw() gives more of the same ranges, prepare() makes what
a program holds before the call, run() is the call, work() what it cannot do
without, exact() its results from plain numpy / torch in 64 bits.

Molecules are those of the engine's own configurations: linear alkanes CnH2n+2
(n = 1 .. 40) and clusters of 1 .. 32 waters in cc-pVDZ / cc-pVDZ-RI. The seed
turns and shakes an alkane (0.03 Angstrom, as in a geometry scan or the guess
network's training set) or places the waters, so another seed is another
geometry with other screened pairs.

Calls:
  fock     set_density + build_FockMat: one FP64 J, K, F and energy, the step
           of a host program that runs its own SCF loop
  density  set_fock + build_DenMat: eigensolve of F' and the density
  solve    reset_scf + do_SCF: one SCF solve on a prepared molecule, plain
           (SAD guess, FP64, an eigensolve every iteration) or accelerated
           (learned guess, tensor-core K, refinement, CUDA graph)
  batch    one batched SCF over several water clusters, accelerated
  job      files to converged energy: init, integrals, DF tensor, SCF, free
  train    the guess network's training on the GPU
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "yatscf-df_b200"))
import geometry  # noqa: E402
import tinyscf  # noqa: E402

DATA = os.path.join(ROOT, "tests", "golden", "data")
BAS = os.path.join(DATA, "cc-pvdz", "cc-pvdz.gbs")
DFBAS = os.path.join(DATA, "cc-pVDZ-RI", "cc-pVDZ-RI.gbs")
MAX_ITER = 100
ENE_TOL = 1e-8
NBF = {"H": 5, "C": 15, "O": 15}          # functions an element has in cc-pVDZ (Cartesian)
NAUX = {"H": 15, "C": 66, "O": 66}        # and in cc-pVDZ-RI
CHARGE = {"H": 1, "C": 6, "O": 8}


def listed():
    return [
        # the smallest call: latency and the number of launches
        {"name": "fock_water", "call": "fock", "mol": "water", "n": 1},
        # a compact, odd-sized molecule: every pair of functions survives the screening
        {"name": "fock_waters13", "call": "fock", "mol": "water", "n": 13},
        # an ordinary chain: half of the pairs are screened away
        {"name": "fock_c20h42", "call": "fock", "mol": "alkane", "n": 20},
        # the largest molecule of the configurations
        {"name": "fock_c40h82", "call": "fock", "mol": "alkane", "n": 40},
        # eigensolve and density of an ordinary and of the largest basis
        {"name": "density_c10h22", "call": "density", "mol": "alkane", "n": 10},
        {"name": "density_c40h82", "call": "density", "mol": "alkane", "n": 40},
        # the reference's algorithm from guess to convergence
        {"name": "solve_plain_c10h22", "call": "solve", "mol": "alkane", "n": 10, "accelerated": False},
        # the accelerated form at the headline size
        {"name": "solve_c40h82", "call": "solve", "mol": "alkane", "n": 40, "accelerated": True},
        # many molecules of uneven size at once
        {"name": "batch_waters", "call": "batch", "count": 8, "n_min": 2, "n_max": 12},
        # whole jobs: the smallest, and the headline molecule
        {"name": "job_water", "call": "job", "mol": "water", "n": 1, "accelerated": False},
        {"name": "job_c40h82", "call": "job", "mol": "alkane", "n": 40, "accelerated": True},
        # training of the guess network: forward, backward and Adam
        {"name": "train_guess", "call": "train", "rows": 4096, "epochs": 2},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng):
    call = rng.choice(["fock", "fock", "fock", "density", "density", "solve", "solve", "batch", "job", "train"])
    if call == "batch":
        lo = rng.randint(2, 6)
        return {"call": call, "count": rng.randint(2, 8), "n_min": lo, "n_max": rng.randint(lo + 1, 12)}
    if call == "train":
        return {"call": call, "rows": _log_int(rng, 300, 6000), "epochs": rng.randint(1, 2)}
    mol = rng.choice(["alkane", "water"])
    case = {"call": call, "mol": mol, "n": _log_int(rng, 1, 39) if mol == "alkane" else _log_int(rng, 1, 24)}
    if call in ("solve", "job"):
        # SAD + DIIS may end in other solutions on random clusters: those start from the network
        case["accelerated"] = True if mol == "water" and case["n"] > 1 else rng.random() < 0.5
    return case


# ------------------------------------------------------------------ inputs
def _atoms(case, seed):
    if case["mol"] == "water":
        return geometry.water_cluster(seed, case["n"], case["n"])
    rng = np.random.default_rng(seed)
    atoms = geometry.alkane(case["n"])
    q = rng.normal(size=4)
    w, x, y, z = q / np.linalg.norm(q)
    rot = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                    [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                    [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])
    xyz = np.array([a[1:] for a in atoms]) @ rot.T + rng.normal(0.0, 0.03, size=(len(atoms), 3))
    return [(a[0], *map(float, p)) for a, p in zip(atoms, xyz)]


def _size(atoms):
    """(basis functions, aux functions, occupied orbitals)"""
    return (sum(NBF[a[0]] for a in atoms), sum(NAUX[a[0]] for a in atoms), sum(CHARGE[a[0]] for a in atoms) // 2)


class Files:
    """An .xyz file that lives as long as its owner."""

    def __init__(self, atoms):
        self.dir = tempfile.TemporaryDirectory()
        self.xyz = os.path.join(self.dir.name, "molecule.xyz")
        geometry.write_xyz(self.xyz, atoms)


def _engine(atoms):
    files = Files(atoms)
    e = tinyscf.TinySCF(BAS, DFBAS, files.xyz, MAX_ITER)
    e.s.ene_tol = ENE_TOL
    return e


def _accelerate(e):
    e.set_k_precision(tinyscf.K_MIXED)
    e.set_density_solver(tinyscf.DENSITY_REFINE)
    e.set_graph(True)


def _density(case, seed):
    """A density of orthonormal occupied orbitals (D, Cocc)."""
    n, _, o = _size(_atoms(case, seed))
    q, _ = np.linalg.qr(np.random.default_rng(seed + 1).normal(size=(n, o)))
    return np.ascontiguousarray(q @ q.T), np.ascontiguousarray(q)


def _fock_orthogonal(case, seed):
    """F' with a Fock operator's spectrum: cores, valence and virtual levels."""
    atoms = _atoms(case, seed)
    n, _, o = _size(atoms)
    rng = np.random.default_rng(seed + 2)
    core = [-20.5 if a[0] == "O" else -11.2 for a in atoms if a[0] != "H"]
    w = np.concatenate([np.array(core) + rng.normal(0, 0.02, len(core)),
                        rng.uniform(-1.3, -0.4, o - len(core)), rng.uniform(0.15, 4.5, n - o)])
    q, _ = np.linalg.qr(rng.normal(size=(n, n)))
    f = (q * w) @ q.T
    return 0.5 * (f + f.T)


def prepare(case, seed):
    call = case["call"]
    if call == "train":
        rng = np.random.default_rng(seed)
        n = case["rows"]
        feat = np.zeros((n, tinyscf.GUESS_DIN), dtype=np.float32)
        feat[:, :24] = rng.random((n, 24), dtype=np.float32)          # element one-hots, distance Gaussians
        feat[:, 24:] = rng.normal(0.0, 0.5, (n, tinyscf.GUESS_DIN - 24))
        target = rng.normal(0.0, 0.1, (n, tinyscf.GUESS_MAXF ** 2)).astype(np.float32)
        types = rng.integers(0, 5, n).astype(np.int32)
        d = tempfile.TemporaryDirectory()
        return {"case": case, "feat": feat, "target": target, "types": types, "dir": d}
    if call == "batch":
        engines = []
        for k in range(case["count"]):
            n = case["n_min"] + k * (case["n_max"] - case["n_min"]) // (case["count"] - 1)
            e = _engine(geometry.water_cluster(1000 * seed + k, n, n))
            e.setup(guess=tinyscf.GUESS_LEARNED)
            e.set_k_precision(tinyscf.K_MIXED)
            e.set_density_solver(tinyscf.DENSITY_REFINE)
            engines.append(e)
        return {"case": case, "engines": engines, "batch": tinyscf.TinySCFBatch(engines)}
    atoms = _atoms(case, seed)
    if call == "job":
        return {"case": case, "files": Files(atoms)}
    e = _engine(atoms)
    s = {"case": case, "engine": e}
    if call == "density":
        e.compute_Hcore_Ovlp_mat()
        s["fock"] = _fock_orthogonal(case, seed)
    elif call == "fock":
        e.setup()
        s["D"], s["Cocc"] = _density(case, seed)
    else:
        e.setup(guess=tinyscf.GUESS_LEARNED if case["accelerated"] else None)
        if case["accelerated"]:
            _accelerate(e)
    return s


# ------------------------------------------------------------------ the calls
class Mirror(np.ndarray):
    """A matrix of a handle's struct, where it lies; it keeps the handle."""


def _mirror(e, name):
    n = e.s.nbasfuncs
    shape = (n,) if name == "eigval" else (n, n)
    a = np.ctypeslib.as_array(getattr(e.s, name), shape=shape).view(Mirror)
    a.owner = e
    return a


def run(s):
    case = s["case"]
    call = case["call"]
    if call == "train":
        path = os.path.join(s["dir"].name, "weights.bin")
        loss = tinyscf.guess_train(s["feat"], s["target"], s["types"], path, epochs=case["epochs"], seed=1)
        with open(path, "rb") as f:
            head = 8 + 4 * 3 + 4 * 5      # magic, sizes, the five block types' widths
            return {"loss": loss, "weights": np.frombuffer(f.read()[head:], dtype=np.float32)}
    if call == "batch":
        for e in s["engines"]:
            e.reset_scf()
        s["batch"].do_SCF()
        return {"energy": np.array([e.energy for e in s["engines"]]), "D": [_mirror(e, "D_mat") for e in s["engines"]]}
    if call == "job":
        e = tinyscf.TinySCF(BAS, DFBAS, s["files"].xyz, MAX_ITER)
        e.s.ene_tol = ENE_TOL
        e.setup(guess=tinyscf.GUESS_LEARNED if case["accelerated"] else None)
        if case["accelerated"]:
            _accelerate(e)
        e.do_SCF()
        out = {"energy": e.energy, "D": e.mat("D_mat"), "J": e.mat("J_mat"), "K": e.mat("K_mat")}
        e.free()
        return out
    e = s["engine"]
    if call == "fock":
        e.set_density(s["D"], s["Cocc"])
        e.build_FockMat()
        return {"J": _mirror(e, "J_mat"), "K": _mirror(e, "K_mat"), "F": _mirror(e, "F_mat"), "energy": e.energy}
    if call == "density":
        e.set_fock(s["fock"], orthogonal=True)
        e.build_DenMat()
        return {"D": _mirror(e, "D_mat"), "eigval": _mirror(e, "eigval")}
    e.reset_scf()
    e.do_SCF()
    return {"energy": e.energy, "D": _mirror(e, "D_mat"), "J": _mirror(e, "J_mat"), "K": _mirror(e, "K_mat")}


# ------------------------------------------------------------------ what a pass cannot do without
def _molecule_sizes(mol, n):
    """(basis functions, aux functions, occupied orbitals, surviving ordered pairs)"""
    h = 2 * n + 2 if mol == "alkane" else 2 * n
    nbf, naux, o = 15 * n + 5 * h, 66 * n + 15 * h, (6 * n + h) // 2 if mol == "alkane" else 5 * n
    # along a chain a function keeps about 240 partners; a cluster's volume grows slowly enough to keep nearly all
    return nbf, naux, o, nbf * min(nbf, 240) if mol == "alkane" else nbf * nbf


def _fock_work(mol, n):
    nbf, naux, o, nnz = _molecule_sizes(mol, n)
    return {"bytes": 8.0 * (nnz / 2 * naux + 5 * nbf * nbf),
            "flops": 2.0 * o * naux * nnz + 1.0 * nbf * nbf * o * naux + 2.0 * nnz * naux}


def _solve_work(mol, n, iterations, eigensolves):
    f = _fock_work(mol, n)
    nbf, _, o, _ = _molecule_sizes(mol, n)
    return {"bytes": iterations * f["bytes"],
            "flops": iterations * (f["flops"] + 8.0 * nbf ** 3) + eigensolves * 9.0 * nbf ** 3}


def work(case):
    call = case["call"]
    if call == "train":
        per_row = 2.0 * (tinyscf.GUESS_DIN * 192 + 192 * 192 + 192 * 120)
        return {"bytes": 4.0 * case["rows"] * (128 + 225) * case["epochs"], "flops": 3.0 * per_row * case["rows"] * case["epochs"]}
    if call == "batch":
        mean = (case["n_min"] + case["n_max"]) / 2
        w = _solve_work("water", mean, 9, 1)
        return {k: case["count"] * v for k, v in w.items()}
    mol, n = case["mol"], case["n"]
    nbf, naux, o, nnz = _molecule_sizes(mol, n)
    if call == "fock":
        return _fock_work(mol, n)
    if call == "density":
        return {"bytes": 8.0 * 4 * nbf * nbf, "flops": 9.0 * nbf ** 3 + 4.0 * nbf * nbf * o}
    w = _solve_work(mol, n, 9, 1) if case["accelerated"] else _solve_work(mol, n, 11, 11)
    if call == "job":
        w["bytes"] += 8.0 * (nnz / 2 * naux + naux * naux)
        w["flops"] += 1.0 * nnz * naux * naux + 9.0 * naux ** 3
    return w


# ------------------------------------------------------------------ exact values: Gaussian integrals in 64 bits
# McMurchie-Davidson with Hermite expansions, over whole groups of equal shells
# at once. Cartesian components run xx, xy, xz, yy, yz, zz; a contracted
# shell's x^l component has unit norm; Angstrom to Bohr as the engine has it.
BOHR = 0.52917720859
FP = torch.float64


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _parse_basis(path):
    shells, element, todo = {}, None, iter(open(path).read().splitlines()[1:])
    for line in todo:
        f = line.split()
        if not f or f[0].startswith("*"):
            continue
        if f[0].isalpha() and len(f) >= 3 and f[1].isdigit():
            prims = [next(todo).replace("D", "E").split() for _ in range(int(f[1]))]
            shells[element].append(("SPDFG".index(f[0].upper()), [float(p[0]) for p in prims], [float(p[1]) for p in prims]))
        elif f[0].isalpha():
            element = f[0]
            shells[element] = []
    return shells


def _dfact(n):
    return 1.0 if n <= 1 else n * _dfact(n - 2)


def _groups(atoms, path):
    """[{l, cen [s,3], a [s,p], c [s,p], first [s]}] for shells of equal momentum and length, and the number of functions."""
    basis, groups, at = _parse_basis(path), {}, 0
    for el, *xyz in atoms:
        for l, ex, cc in basis[el]:
            a, c = np.array(ex), np.array(cc)
            c = c * (2 * a / math.pi) ** 0.75 * (4 * a) ** (0.5 * l) / math.sqrt(_dfact(2 * l - 1))
            p = a[:, None] + a[None, :]
            c = c / math.sqrt(float((c[:, None] * c[None, :] * (math.pi / p) ** 1.5 * _dfact(2 * l - 1) / (2 * p) ** l).sum()))
            g = groups.setdefault((l, len(a)), {"l": l, "cen": [], "a": [], "c": [], "first": []})
            g["cen"].append(np.array(xyz) * (1.0 / BOHR))
            g["a"].append(a)
            g["c"].append(c)
            g["first"].append(at)
            at += (l + 1) * (l + 2) // 2
    dev = _device()
    for g in groups.values():
        for k in ("cen", "a", "c"):
            g[k] = torch.tensor(np.array(g[k]), dtype=FP, device=dev)
        g["first"] = torch.tensor(g["first"], device=dev)
    return list(groups.values()), at


def _cart(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _hermites(l):
    return [(t, u, v) for t in range(l + 1) for u in range(l + 1 - t) for v in range(l + 1 - t - u)]


def _hermite_1d(la, lb, p, pa, pb, k):
    """E[i][j][t] of one direction; k is the t = 0 coefficient of two s functions."""
    E = {(0, 0, 0): k}

    def get(i, j, t):
        return E.get((i, j, t)) if 0 <= t <= i + j else None

    def total(parts):
        out = None
        for f, x in parts:
            if x is not None:
                out = f * x if out is None else out + f * x
        return out

    h = 0.5 / p
    for i in range(la + 1):
        for j in range(lb + 1):
            if i == j == 0:
                continue
            for t in range(i + j + 1):
                a, b, r = (i - 1, j, pa) if i else (i, j - 1, pb)
                E[i, j, t] = total([(h, get(a, b, t - 1)), (r, get(a, b, t)), (float(t + 1), get(a, b, t + 1))])
    return E


def _pairs(ga, gb, ia, ib, extra=0):
    """Hermite data of the shell pairs (ia[k], ib[k]): exponents p, centres P [s,q,3], E per direction, coefficients."""
    a, b = ga["a"][ia][:, :, None], gb["a"][ib][:, None, :]
    A, B = ga["cen"][ia], gb["cen"][ib]
    s = len(ia)
    p = (a + b).reshape(s, -1)
    mu = (a * b).reshape(s, -1) / p
    wa = (a / (a + b)).reshape(s, -1)
    P = B[:, None, :] + wa[..., None] * (A - B)[:, None, :]
    cc = (ga["c"][ia][:, :, None] * gb["c"][ib][:, None, :]).reshape(s, -1)
    E = []
    for d in range(3):
        x = (A - B)[:, d][:, None]
        E.append(_hermite_1d(ga["l"], gb["l"] + extra, p, P[..., d] - A[:, d][:, None], P[..., d] - B[:, d][:, None], torch.exp(-mu * x * x)))
    return p, P, E, cc


def _expand(la, lb, E, cc):
    """[s, q, components of a x components of b, hermites]"""
    rows, zero = [], torch.zeros_like(cc)
    for ca in _cart(la):
        for cb in _cart(lb):
            row = []
            for h in _hermites(la + lb):
                ok = all(h[d] <= ca[d] + cb[d] for d in range(3))
                row.append(cc * E[0][ca[0], cb[0], h[0]] * E[1][ca[1], cb[1], h[1]] * E[2][ca[2], cb[2], h[2]] if ok else zero)
            rows.append(torch.stack(row, -1))
    return torch.stack(rows, -2)


def _boys(m, T):
    """F_0 .. F_m."""
    x = T.clamp(min=1e-2)
    top = torch.special.gammainc(torch.full_like(x, m + 0.5), x) * (0.5 * math.gamma(m + 0.5)) / x ** (m + 0.5)
    series = sum((-T) ** k / (math.factorial(k) * (2 * m + 2 * k + 1)) for k in range(8))
    F = [torch.where(T < 1e-2, series, top)]
    e = torch.exp(-T)
    for k in range(m, 0, -1):
        F.append((2 * T * F[-1] + e) / (2 * k - 1))
    return F[::-1]


def _coulomb(l, alpha, R):
    """Hermite Coulomb integrals {(t,u,v): ...} up to t + u + v = l for distances R [..., 3]."""
    F = _boys(l, alpha * (R * R).sum(-1))
    cur = {(0, 0, 0): [(-2 * alpha) ** n * F[n] for n in range(l + 1)]}
    for t, u, v in sorted(_hermites(l), key=sum):
        if (t, u, v) == (0, 0, 0):
            continue
        d = 0 if t else 1 if u else 2
        low = [t, u, v]
        low[d] -= 1
        k, one = low[d], tuple(low)
        low[d] -= 1
        two = cur.get(tuple(low))
        vals = []
        for n in range(l - (t + u + v) + 1):
            x = R[..., d] * cur[one][n + 1]
            vals.append(x + k * two[n + 1] if k else x)
        cur[t, u, v] = vals
    return {h: x[0] for h, x in cur.items()}


def _place(out, ga, gb, ia, ib, vals):
    """vals [s, comps a, comps b, ...] into out[a, b, ...] and out[b, a, ...]"""
    na, nb = vals.shape[1], vals.shape[2]
    r = ga["first"][ia][:, None, None] + torch.arange(na, device=vals.device)[None, :, None]
    c = gb["first"][ib][:, None, None] + torch.arange(nb, device=vals.device)[None, None, :]
    out[r, c] = vals
    out[c.expand(-1, na, -1), r.expand(-1, -1, nb)] = vals


def _all_pairs(groups):
    for x, ga in enumerate(groups):
        for gb in groups[: x + 1]:
            if ga["l"] < gb["l"]:
                ga_, gb_ = gb, ga
            else:
                ga_, gb_ = ga, gb
            na, nb = len(ga_["first"]), len(gb_["first"])
            k = torch.arange(na * nb, device=ga["a"].device)
            yield ga_, gb_, k // nb, k % nb


def _overlap(atoms, kinetic=False):
    groups, n = _groups(atoms, BAS)
    S = torch.zeros(n, n, dtype=FP, device=_device())
    T = torch.zeros_like(S)
    for ga, gb, ia, ib in _all_pairs(groups):
        p, _, E, cc = _pairs(ga, gb, ia, ib, 2)
        r = torch.sqrt(math.pi / p)
        beta = gb["a"][ib][:, None, :].expand(-1, ga["a"].shape[1], -1).reshape(len(ia), -1)

        def s1(d, i, j):
            return E[d][i, j, 0] * r

        def t1(d, i, j):
            x = beta * (2 * j + 1) * s1(d, i, j) - 2 * beta ** 2 * s1(d, i, j + 2)
            return x - 0.5 * j * (j - 1) * s1(d, i, j - 2) if j > 1 else x

        sv, tv = [], []
        for a in _cart(ga["l"]):
            for b in _cart(gb["l"]):
                s = [s1(d, a[d], b[d]) for d in range(3)]
                sv.append((cc * s[0] * s[1] * s[2]).sum(-1))
                if kinetic:
                    t = [t1(d, a[d], b[d]) for d in range(3)]
                    tv.append((cc * (t[0] * s[1] * s[2] + s[0] * t[1] * s[2] + s[0] * s[1] * t[2])).sum(-1))
        shape = (len(ia), len(_cart(ga["l"])), len(_cart(gb["l"])))
        _place(S, ga, gb, ia, ib, torch.stack(sv, -1).reshape(shape))
        if kinetic:
            _place(T, ga, gb, ia, ib, torch.stack(tv, -1).reshape(shape))
    return S, T


def _attraction(atoms):
    groups, n = _groups(atoms, BAS)
    dev = _device()
    V = torch.zeros(n, n, dtype=FP, device=dev)
    C = torch.tensor([a[1:] for a in atoms], dtype=FP, device=dev) * (1.0 / BOHR)
    Z = torch.tensor([float(CHARGE[a[0]]) for a in atoms], dtype=FP, device=dev)
    for ga, gb, ia, ib in _all_pairs(groups):
        l, q = ga["l"] + gb["l"], ga["a"].shape[1] * gb["a"].shape[1]
        step = max(1, int(4e6 / (q * len(atoms) * len(_hermites(l)))))
        for k in range(0, len(ia), step):
            a, b = ia[k:k + step], ib[k:k + step]
            p, P, E, cc = _pairs(ga, gb, a, b)
            R = _coulomb(l, p[:, :, None].expand(-1, -1, len(atoms)), P[:, :, None, :] - C)
            H = torch.stack([-(R[h] * Z).sum(-1) for h in _hermites(l)], -1) * (2 * math.pi / p)[..., None]
            vals = (_expand(ga["l"], gb["l"], E, cc) * H[:, :, None, :]).sum((1, 3))
            _place(V, ga, gb, a, b, vals.reshape(len(a), len(_cart(ga["l"])), -1))
    return V


def _three_centre(bra, n, aux, naux):
    """(ab|P) [n, n, naux] of shell groups."""
    dev = _device()
    out = torch.zeros(n, n, naux, dtype=FP, device=dev)
    for gc in aux:
        lc, nc = gc["l"], len(_cart(gc["l"]))
        g, w = gc["a"][:, 0], gc["c"][:, 0]
        if gc["a"].shape[1] != 1:
            raise ValueError("contracted auxiliary shell")
        zero = torch.zeros_like(g)
        Ec = _hermite_1d(lc, 0, g, zero, zero, torch.ones_like(g))
        Xc = _expand(lc, 0, [Ec, Ec, Ec], w)                                  # [c, comps, hermites]
        Xc = Xc * torch.tensor([(-1.0) ** sum(h) for h in _hermites(lc)], dtype=FP, device=dev)
        cols = (gc["first"][:, None] + torch.arange(nc, device=dev)).reshape(-1)
        for ga, gb, ia, ib in _all_pairs(bra):
            lab = ga["l"] + gb["l"]
            q, hab = ga["a"].shape[1] * gb["a"].shape[1], _hermites(lab)
            step = max(1, int(3e7 / (q * len(g) * max(len(hab) * nc, len(_hermites(lab + lc)) * 3))))
            for k in range(0, len(ia), step):
                a, b = ia[k:k + step], ib[k:k + step]
                p, P, E, cc = _pairs(ga, gb, a, b)
                p, s = p[:, :, None], len(a)
                R = _coulomb(lab + lc, p * g / (p + g), P[:, :, None, :] - gc["cen"])
                pre = 2 * math.pi ** 2.5 / (p * g * torch.sqrt(p + g))
                G = torch.stack([torch.einsum("sqch,cdh->sqcd", torch.stack([R[t + x, u + y, v + z] for x, y, z in _hermites(lc)], -1), Xc) * pre[..., None]
                                 for t, u, v in hab], 2)                      # [s, q, hab, c, comps]
                X = _expand(ga["l"], gb["l"], E, cc)                          # [s, q, ab, hab]
                vals = torch.matmul(X.permute(0, 2, 1, 3).reshape(s, X.shape[2], -1), G.reshape(s, q * len(hab), -1))
                na = len(_cart(ga["l"]))
                vals = vals.reshape(s, na, -1, len(cols))
                block = torch.zeros(vals.shape[:3] + (naux,), dtype=FP, device=dev) if len(cols) == naux else None
                if block is not None:
                    block[..., cols] = vals
                    _place(out, ga, gb, a, b, block)
                else:
                    nb = vals.shape[2]
                    r = (ga["first"][a][:, None, None] + torch.arange(na, device=dev)[None, :, None]).expand(-1, -1, nb)
                    c = (gb["first"][b][:, None, None] + torch.arange(nb, device=dev)[None, None, :]).expand(-1, na, -1)
                    out[r[..., None], c[..., None], cols] = vals
                    out[c[..., None], r[..., None], cols] = vals
    return out


def exact(case, seed):
    call = case["call"]
    if call == "density":
        S, _ = _overlap(_atoms(case, seed))
        S = S.cpu().numpy()
        w, U = np.linalg.eigh(S)
        X = (U / np.sqrt(w)) @ U.T
        _, _, o = _size(_atoms(case, seed))
        w, V = np.linalg.eigh(_fock_orthogonal(case, seed))
        C = X @ V[:, :o]
        return {"D": C @ C.T, "eigval": w}
    if call != "fock":
        return None       # a converged solve, or a training run, is where its own iterations end
    atoms = _atoms(case, seed)
    n, naux, _ = _size(atoms)
    if n > 520:
        return None       # over 20 seconds
    dev = _device()
    D, Cocc = (torch.tensor(x, device=dev) for x in _density(case, seed))
    aux, _ = _groups(atoms, DFBAS)
    bra, _ = _groups(atoms, BAS)
    one = {"l": 0, "cen": torch.zeros(1, 3, dtype=FP, device=dev), "a": torch.zeros(1, 1, dtype=FP, device=dev),
           "c": torch.ones(1, 1, dtype=FP, device=dev), "first": torch.tensor([0], device=dev)}
    metric = torch.zeros(naux, naux, dtype=FP, device=dev)
    for g in aux:                                     # (P|Q) = (P 1|Q) with a function 1 that is constant
        three = _pair_with_one(g, one, aux, naux)
        metric[(g["first"][:, None] + torch.arange(three.shape[1], device=dev)).reshape(-1)] = three.reshape(-1, naux)
    L = torch.linalg.cholesky(0.5 * (metric + metric.T))
    B = _three_centre(bra, n, aux, naux).reshape(n * n, naux)
    B = torch.linalg.solve_triangular(L, B.T, upper=False).reshape(naux, n, n)
    J = torch.einsum("p,pij->ij", torch.einsum("pij,ij->p", B, D), B)
    half = torch.einsum("pij,js->ips", B, Cocc).reshape(n, -1)
    K = half @ half.T
    S, T = _overlap(atoms, kinetic=True)
    H = T + _attraction(atoms)
    F = H + 2 * J - K
    xyz = np.array([a[1:] for a in atoms]) * (1.0 / BOHR)
    z = np.array([CHARGE[a[0]] for a in atoms], dtype=float)
    i, j = np.triu_indices(len(z), 1)
    nuc = float((z[i] * z[j] / np.linalg.norm(xyz[i] - xyz[j], axis=1)).sum()) if len(z) > 1 else 0.0
    out = {k: v.cpu().numpy() for k, v in (("J", J), ("K", K), ("F", F))}
    out["energy"] = float((D * (F + H)).sum()) + nuc
    return out


def _pair_with_one(g, one, aux, naux):
    """(P 1|Q) [shells of g, comps, naux]"""
    ia = torch.arange(len(g["first"]), device=g["a"].device)
    here = {**g, "first": ia * len(_cart(g["l"]))}
    n = len(ia) * len(_cart(g["l"]))
    out = torch.zeros(len(ia), len(_cart(g["l"])), naux, dtype=FP, device=g["a"].device)
    for gc in aux:
        p, P, E, cc = _pairs(here, {**one, "cen": one["cen"]}, ia, torch.zeros_like(ia))
        # with an exponent of zero the pair is the shell itself, at its own centre
        lc = gc["l"]
        q = gc["a"][:, 0]
        zero = torch.zeros_like(q)
        Ec = _hermite_1d(lc, 0, q, zero, zero, torch.ones_like(q))
        Xc = _expand(lc, 0, [Ec, Ec, Ec], gc["c"][:, 0]) * torch.tensor([(-1.0) ** sum(h) for h in _hermites(lc)], dtype=FP, device=q.device)
        R = _coulomb(g["l"] + lc, p * q / (p + q), P - gc["cen"])
        pre = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        X = _expand(g["l"], 0, E, cc)[:, 0]                     # [s, comps, hermites]
        ha = _hermites(g["l"])
        G = torch.stack([torch.einsum("sch,cdh->scd", torch.stack([R[t + x, u + y, v + z] for x, y, z in _hermites(lc)], -1), Xc) * pre[..., None]
                         for t, u, v in ha], 1)                # [s, ha, c, comps]
        vals = torch.einsum("sah,shcd->sacd", X, G)
        cols = (gc["first"][:, None] + torch.arange(len(_cart(lc)), device=q.device)).reshape(-1)
        out[:, :, cols] = vals.reshape(len(ia), -1, len(cols))
    return out
