"""Cases that a user of the engine has it do, for timing and for comparing outputs.

Every case is a plain dict; ``kind`` names the entry point, the rest are sizes and options:

* ``quartet``     ``ElectronRepulsionIntegral.construct_array_contraction`` of four shells;
* ``tensor``      ``electron_repulsion_integral``, host shells in, host array out;
* ``resident``    ``DeviceBasis.full_device``: the basis stays on the GPU, so does the tensor;
* ``batch``       ``EriBatch.run``: many molecules packed once, run many times;
* ``batch_call``  ``electron_repulsion_integral_batch``: many molecules in one call;
* ``coulomb``     ``coulomb_matrix``: direct J with screening, host in, host out;
* ``jk``          ``coulomb_exchange``: J and K of a density without symmetry;
* ``lincomb``     ``electron_repulsion_integral`` with a transform;
* ``attenuated``  ``electron_repulsion_integral_improved`` with a screening threshold and the
                  erf / erfc operators;
* ``nuclear``     ``nuclear_electron_attraction_integral``.

The shells of an atom are a text such as ``"s6 s3 p3 d1"`` (letter and number of primitives);
the patterns are those of the synthetic workloads in ``gbasis_b200/synthetic.py``, whose
distributions of exponents, coefficients and positions the inputs follow too.  What a case
costs is fixed by the case (numbers of atoms, shells and primitives); the seed draws positions,
exponents, coefficients and densities.

``exact`` evaluates the same integrals by the McMurchie-Davidson scheme in plain torch (FP64).
"""
from __future__ import annotations

import ctypes
import itertools
import math

import numpy as np
import torch

from gbasis_b200 import _engine
from gbasis_b200.batch import EriBatch, electron_repulsion_integral_batch
from gbasis_b200.contractions import GeneralizedContractionShell
from gbasis_b200.coulomb import coulomb_exchange, coulomb_matrix
from gbasis_b200.electron_repulsion import (ElectronRepulsionIntegral, electron_repulsion_integral,
                                            electron_repulsion_integral_improved)
from gbasis_b200.flops import basis_flops, hrr_flops, prim_flops
from gbasis_b200.point_charge import nuclear_electron_attraction_integral

LETTERS = "spdf"
TINY = "s3 s1 p3"
MEDIUM = "s6 s3 s1 p3 p1 d1"
CHAIN = "s5 s5 s5 p3 p3 d2 f1"
LARGE = "s8 s4 s2 s1 p3 p3 p3 d2 d2 f1"
SMALL_SPD = "s3 s2 p2 d1"
# most primitives of a shell where the shells are drawn: contractions get shorter with l, as in
# contracted basis sets (a six-fold d shell spanning exponents 0.1 to 260 costs the contracted
# recursions seven digits, so that no two evaluation orders agree on it)
MOST_PRIMS = (6, 4, 3, 2)


def listed():
    return [
        # one shell quartet for host code that drives the engine quartet by quartet: the smallest
        # call there is, all latency
        {"name": "quartet d p p s", "kind": "quartet", "shells": "d3 p3 p2 s4"},
        # the four-atom basis of the tests and tutorials, default arguments, host array out
        {"name": "tensor 4 atoms", "kind": "tensor", "shells": TINY, "atoms": 4, "volume": 54.0,
         "coord": "cartesian", "notation": "physicist"},
        # a small molecule with d shells, spherical functions, an odd number of atoms
        {"name": "tensor 5 atoms spd", "kind": "tensor", "shells": SMALL_SPD, "atoms": 5,
         "volume": 54.0, "coord": "spherical", "notation": "chemist"},
        # the 120-function tensor kept on the GPU: the headline configuration of the benchmark
        {"name": "resident 8 atoms spd", "kind": "resident", "shells": MEDIUM, "atoms": 8,
         "volume": 125.0, "coord": "cartesian"},
        # f shells, spherical, as in the chain configuration
        {"name": "resident 7 atoms spdf", "kind": "resident", "shells": CHAIN, "atoms": 7,
         "volume": 0.0, "coord": "spherical"},
        # many uneven molecules packed once, then run at every geometry or step: the batch
        # configuration
        {"name": "batch 60 molecules", "kind": "batch", "molecules": 60, "most_atoms": 14,
         "mix": 11, "precision": "fp64"},
        # a few small molecules in one call, mixed precision
        {"name": "batch call 12 mixed", "kind": "batch_call", "molecules": 12, "most_atoms": 7,
         "mix": 5, "precision": "mixed"},
        # direct J of a part of the 64-atom box: contracted s shells up to f, screened
        {"name": "coulomb 9 atoms spdf", "kind": "coulomb", "shells": LARGE, "atoms": 9,
         "volume": 125.0, "coord": "spherical", "precision": "fp64"},
        # J and K of a density without symmetry
        {"name": "jk 7 atoms spd", "kind": "jk", "shells": MEDIUM, "atoms": 7, "volume": 125.0,
         "coord": "cartesian"},
        # integrals over molecular orbitals
        {"name": "lincomb 4 atoms spd", "kind": "lincomb", "shells": SMALL_SPD, "atoms": 4,
         "volume": 54.0, "coord": "cartesian", "orbitals": 21},
        # long-range part of a range-separated functional, screened
        {"name": "erf 5 atoms spd", "kind": "attenuated", "shells": SMALL_SPD, "atoms": 5,
         "volume": 125.0, "coord": "spherical", "potential": "erf", "omega": 0.4,
         "threshold": 1e-12},
        # the one-electron companion of a calculation
        {"name": "nuclear 11 atoms", "kind": "nuclear", "shells": CHAIN, "atoms": 11,
         "volume": 0.0, "coord": "spherical"},
    ]


def draw(rng):
    def between(lo, hi):  # a whole number, spread over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    coord = rng.choice(["cartesian", "spherical"])
    volume = rng.choice([0.0, 54.0, 125.0])
    kind = rng.choice(["quartet", "tensor", "resident", "resident", "batch", "batch", "batch_call",
                       "coulomb", "coulomb", "jk", "lincomb", "attenuated", "nuclear"])
    if kind == "quartet":
        ls = [rng.randrange(4) for _ in range(4)]
        return {"kind": kind,
                "shells": " ".join(LETTERS[l] + str(rng.randint(1, MOST_PRIMS[l])) for l in ls)}
    if kind in ("batch", "batch_call"):
        most, atoms = (60, 14) if kind == "batch" else (14, 7)
        return {"kind": kind, "molecules": between(3, most), "most_atoms": rng.randint(4, atoms),
                "mix": rng.randrange(1, 10 ** 6), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "resident":
        shells = rng.choice([TINY, MEDIUM, SMALL_SPD, CHAIN])
        atoms = between(2, 7 if shells == CHAIN else 9)
        return {"kind": kind, "shells": shells, "atoms": atoms, "volume": volume, "coord": coord}
    if kind == "tensor":
        shells = rng.choice([TINY, SMALL_SPD, CHAIN])
        atoms = between(1, 3 if shells == CHAIN else 5)
        return {"kind": kind, "shells": shells, "atoms": atoms, "volume": volume, "coord": coord,
                "notation": rng.choice(["physicist", "chemist"])}
    if kind == "coulomb":
        return {"kind": kind, "shells": rng.choice([MEDIUM, CHAIN, LARGE]), "atoms": between(2, 8),
                "volume": 125.0, "coord": coord, "precision": rng.choice(["fp64", "mixed"])}
    if kind == "jk":
        shells = rng.choice([MEDIUM, SMALL_SPD, CHAIN])
        return {"kind": kind, "shells": shells, "atoms": between(2, 5 if shells == CHAIN else 8),
                "volume": volume, "coord": coord}
    if kind == "lincomb":
        return {"kind": kind, "shells": rng.choice([TINY, SMALL_SPD]), "atoms": between(2, 5),
                "volume": volume, "coord": coord, "orbitals": rng.randint(3, 30)}
    if kind == "attenuated":
        return {"kind": kind, "shells": rng.choice([TINY, SMALL_SPD]), "atoms": between(2, 6),
                "volume": volume, "coord": coord, "potential": rng.choice(["erf", "erfc"]),
                "omega": round(rng.uniform(0.2, 1.5), 2), "threshold": rng.choice([0.0, 1e-12])}
    return {"kind": kind, "shells": rng.choice([TINY, MEDIUM, CHAIN]), "atoms": between(2, 20),
            "volume": volume, "coord": coord}


# ------------------------------------------------------------------------------- inputs
def _shell(rng, l, k, center):
    """(l, center, exponents, coefficients): exponents a0 * beta^i, coefficients in (0.1, 1)."""
    a0 = math.exp(rng.uniform(math.log(0.1), math.log(0.5)))
    exps = a0 * rng.uniform(2.5, 3.5) ** np.arange(k, dtype=float)
    return l, np.asarray(center, dtype=float), exps, rng.uniform(0.1, 1.0, size=k)


def _atoms(rng, n, volume):
    """Positions: in a box of ``volume`` bohr^3 per atom (at least 1.2 bohr apart), or, with
    volume 0, a random walk of steps of 1.4 to 2 bohr."""
    pts = [] if volume else [np.zeros(3)]
    while len(pts) < n:
        if volume:
            p = rng.uniform(0.0, (volume * n) ** (1.0 / 3.0), size=3)
            if any(np.linalg.norm(p - q) < 1.2 for q in pts):
                continue
        else:
            v = rng.normal(size=3)
            p = pts[-1] + v / np.linalg.norm(v) * rng.uniform(1.4, 2.0)
        pts.append(p)
    return pts


def _pattern(text):
    return [(LETTERS.index(w[0]), int(w[1:])) for w in text.split()]


def _structure(case):
    """Per molecule, per atom, the (l, primitives) of its shells: fixed by the case alone."""
    if case["kind"] in ("batch", "batch_call"):
        rng = np.random.default_rng(case["mix"])

        def shell():
            l = int(rng.integers(0, 3))
            return l, int(rng.integers(1, MOST_PRIMS[l] + 1))
        return [[[shell() for _ in range(int(rng.integers(1, 4)))]
                 for _ in range(int(rng.integers(2, case["most_atoms"] + 1)))]
                for _ in range(case["molecules"])]
    if case["kind"] == "quartet":
        return [[[s] for s in _pattern(case["shells"])]]
    return [[_pattern(case["shells"])] * case["atoms"]]


def _molecules(case, seed):
    """The molecules of a case as plain data: lists of (l, center, exponents, coefficients)."""
    rng = np.random.default_rng([seed, 77])
    out = []
    for mol in _structure(case):
        pts = _atoms(rng, len(mol), case.get("volume", 54.0))
        out.append([_shell(rng, l, k, p) for p, shells in zip(pts, mol) for l, k in shells])
    return out


def _n_functions(case, mol):
    sph = case.get("coord", "cartesian") == "spherical"
    return sum(2 * l + 1 if sph else _ncart(l) for shells in mol for l, _ in shells)


def _density(case, n, seed):
    rng = np.random.default_rng([seed, 78])
    x = rng.normal(size=(n, max(1, n // 4)))
    d = x @ x.T
    if case["kind"] == "jk":
        d = d + 0.3 * rng.normal(size=(n, n))
    return d / np.linalg.norm(d)


def _transform(case, n, seed):
    return np.random.default_rng([seed, 79]).normal(size=(case["orbitals"], n)) / math.sqrt(n)


def _points(case, seed):
    """The nuclei: the atoms of the molecule with their charges."""
    mol, pts = _molecules(case, seed)[0], []
    for _, center, _, _ in mol:
        if not any(np.array_equal(center, p) for p in pts):
            pts.append(center)
    charges = np.random.default_rng([seed, 80]).integers(1, 9, size=len(pts)).astype(float)
    return np.array(pts), charges


def prepare(case, seed):
    kind, coord = case["kind"], case.get("coord", "cartesian")
    mols = [[GeneralizedContractionShell(l, p, c, e, coord) for l, p, e, c in m]
            for m in _molecules(case, seed)]
    state = {"case": case, "basis": mols[0]}
    if kind == "resident":
        state["db"] = _engine.DeviceBasis(mols[0])
        state["out"] = torch.empty((state["db"].nbf,) * 4, dtype=torch.float64, device="cuda")
    elif kind == "batch":
        state["batch"] = EriBatch(mols)
        state["outs"] = [torch.empty((n,) * 4, dtype=torch.float64, device="cuda")
                         for n in state["batch"].nbf]
    elif kind == "batch_call":
        state["molecules"] = mols
    elif kind in ("coulomb", "jk"):
        state["density"] = _density(case, _n_functions(case, _structure(case)[0]), seed)
    elif kind == "lincomb":
        state["transform"] = _transform(case, _n_functions(case, _structure(case)[0]), seed)
    elif kind == "nuclear":
        state["points"] = _points(case, seed)
    return state


def run(state):
    case, basis = state["case"], state["basis"]
    kind = case["kind"]
    if kind == "quartet":
        return ElectronRepulsionIntegral.construct_array_contraction(*basis)
    if kind == "tensor":
        return electron_repulsion_integral(basis, notation=case["notation"])
    if kind == "resident":
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        state["db"].full_device(state["out"].data_ptr(), "chemist", 0.0, stream=stream)
        return state["out"]
    if kind == "batch":
        mixed = (1e-11, 1e-8) if case["precision"] == "mixed" else None
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        state["batch"].run(state["outs"], stream=stream, mixed=mixed)
        return state["outs"]
    if kind == "batch_call":
        return electron_repulsion_integral_batch(state["molecules"], notation="chemist",
                                                 precision=case["precision"])
    if kind == "coulomb":
        return coulomb_matrix(basis, state["density"], precision=case["precision"])
    if kind == "jk":
        return coulomb_exchange(basis, state["density"])
    if kind == "lincomb":
        return electron_repulsion_integral(basis, transform=state["transform"], notation="chemist")
    if kind == "attenuated":
        return electron_repulsion_integral_improved(
            basis, notation="chemist", schwarz_threshold=case["threshold"],
            potential=case["potential"], omega=case["omega"])
    return nuclear_electron_attraction_integral(basis, *state["points"])


# --------------------------------------------------------------------------------- work
class _Counted:
    """A shell as the FLOP model reads it: angular momentum, primitives, one contraction."""

    def __init__(self, l, k):
        self.angmom, self.exps, self.coeffs = l, [0.0] * k, np.zeros((k, 1))


def work(case):
    """Inputs read once and outputs written once; the operations of the recursions over the unique
    shell quartets (for a screened call: over all of them, an upper bound)."""
    mols = _structure(case)
    flat = [[s for shells in m for s in shells] for m in mols]
    nbf = [_n_functions(case, m) for m in mols]
    read = sum(8 * (3 + 2 * k) for m in flat for _, k in m)
    kind = case["kind"]
    if kind == "quartet":
        (a, ka), (b, kb), (c, kc), (d, kd) = flat[0]
        x, y = sorted(((max(a, b), min(a, b)), (max(c, d), min(c, d))), reverse=True)
        flops = ka * kb * kc * kd * prim_flops(*x, *y) + hrr_flops(*x, *y)
        return {"bytes": read + 8 * _ncart(a) * _ncart(b) * _ncart(c) * _ncart(d), "flops": flops}
    if kind == "nuclear":
        n, atoms = nbf[0], case["atoms"]
        flops = sum(k1 * k2 * atoms * (30 + 8 * _ncart(l1 + l2) * (l1 + l2 + 1))
                    for (l1, k1), (l2, k2) in itertools.combinations_with_replacement(flat[0], 2))
        return {"bytes": read + 8 * (n * n + 4 * atoms), "flops": flops}
    flops = sum(basis_flops([_Counted(l, k) for l, k in m]) for m in flat)
    out = {"coulomb": 2 * nbf[0] ** 2, "jk": 3 * nbf[0] ** 2}.get(kind, sum(n ** 4 for n in nbf))
    if kind == "lincomb":
        k, n = case["orbitals"], nbf[0]
        out = k ** 4 + k * n
        flops += 2 * (k * n ** 4 + k ** 2 * n ** 3 + k ** 3 * n ** 2 + k ** 4 * n)
    return {"bytes": read + 8 * out, "flops": flops}


# -------------------------------------------------------------------------------- exact
# McMurchie-Davidson: a product of two Cartesian Gaussians is a sum of Hermite Gaussians with
# separable coefficients E; the Coulomb integral of two Hermite Gaussians is a derivative of the
# Boys function of their distance.
def _ncart(l):
    return (l + 1) * (l + 2) // 2


def _comps(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _hermites(l):
    return [c for k in range(l + 1) for c in _comps(k)]


def _odd(n):  # n!! for odd n, 1 for n < 1
    return math.prod(range(n, 0, -2))


def _spherical(l):
    """Real solid harmonics over the monomials of degree l, unit-normalised with a Gaussian, as
    (2l+1, ncart): labels s_l..s_1, c_0..c_l; for l = 1 x, y, z."""
    if l < 2:
        return np.eye(_ncart(l))
    comps = _comps(l)
    index = {c: i for i, c in enumerate(comps)}
    rows = []
    for m in [-k for k in range(l, 0, -1)] + list(range(l + 1)):
        row, am = np.zeros(len(comps)), abs(m)
        # S = sum_t c_t r^(2t) z^(l - am - 2t) * Re or Im (x + iy)^am
        for t in range((l - am) // 2 + 1):
            ct = (-0.25) ** t * math.comb(l, t) * math.comb(l - t, am + t)
            for u in range(t + 1):
                for v in range(am + 1):
                    if (v % 2 == 1) != (m < 0):
                        continue
                    x, y = 2 * (t - u) + am - v, 2 * u + v
                    row[index[(x, y, l - am - 2 * t)]] += (ct * math.comb(t, u) * math.comb(am, v)
                                                           * (-1) ** (v // 2))
        # unit norm: <x^a x^b> over the Gaussian is prod (a_i + b_i - 1)!! for even sums
        s = sum(p * q * math.prod(_odd(i + j - 1) if (i + j) % 2 == 0 else 0
                                  for i, j in zip(a, b))
                for p, a in zip(row, comps) for q, b in zip(row, comps))
        rows.append(row / math.sqrt(s))
    return np.array(rows)


def _functions(l, coord):
    """(functions, ncart): the shell's functions over monomials times (2a/pi)^(3/4) (4a)^(l/2)."""
    if coord == "spherical":
        return _spherical(l)
    return np.diag([1.0 / math.sqrt(math.prod(_odd(2 * i - 1) for i in c)) for c in _comps(l)])


def _boys(top, t):
    """F_0..F_top(t): the ascending series at the top and downward recursion, or the asymptotic
    form upward above t = 36 (where erfc(sqrt(t)) is below 1e-17)."""
    small = t < 36.0
    ts = torch.where(small, t, torch.zeros_like(t))
    term = torch.full_like(ts, 1.0 / (2 * top + 1))
    total = term.clone()
    for k in range(1, 160):
        term = term * (2.0 * ts / (2 * top + 2 * k + 1))
        total += term
    e = torch.exp(-ts)
    down = [total * e]
    for m in range(top - 1, -1, -1):
        down.insert(0, (2.0 * ts * down[0] + e) / (2 * m + 1))
    tl = torch.where(small, torch.full_like(t, 36.0), t)
    el = torch.exp(-tl)
    up = [0.5 * torch.sqrt(math.pi / tl)]
    for m in range(top):
        up.append(((2 * m + 1) * up[-1] - el) / (2.0 * tl))
    return [torch.where(small, a, b) for a, b in zip(down, up)]


def _hermite_integrals(order, alpha, x, f):
    """R_tuv for t + u + v <= order, from the separations x = (X, Y, Z) and f[n] = F_n."""
    r = {(0, 0, 0, n): (-2.0 * alpha) ** n * f[n] for n in range(order + 1)}
    for total in range(1, order + 1):
        for c in _comps(total):
            i = max(range(3), key=lambda k: c[k])
            lower = tuple(v - (k == i) for k, v in enumerate(c))
            lowest = tuple(v - 2 * (k == i) for k, v in enumerate(c))
            for n in range(order - total + 1):
                v = x[i] * r[(*lower, n + 1)]
                if lowest[i] >= 0:
                    v = v + lower[i] * r[(*lowest, n + 1)]
                r[(*c, n)] = v
        for key in [k for k in r if sum(k[:3]) < total - 1 and k[3] > 0]:
            del r[key]  # only the n = 0 values of the lower totals are needed from here on
    return r


class _Pairs:
    """The shell pairs of one (la, lb) of a basis: a row per primitive pair."""

    def __init__(self, la, lb, pairs, shells, coord, raw, device):
        rows = {"p": [], "P": [], "PA": [], "PB": [], "c": [], "ab": [], "owner": []}
        for owner, (i, j) in enumerate(pairs):
            (_, A, ea, ca), (_, B, eb, cb) = shells[i], shells[j]
            na, nb = (_contraction(shells[k], raw) for k in (i, j))
            for a, b in itertools.product(range(len(ea)), range(len(eb))):
                p = ea[a] + eb[b]
                P = (ea[a] * A + eb[b] * B) / p
                rows["p"].append(p)
                rows["P"].append(P)
                rows["PA"].append(P - A)
                rows["PB"].append(P - B)
                rows["c"].append(na[a] * nb[b])
                rows["ab"].append(-ea[a] * eb[b] / p * (A - B) ** 2)
                rows["owner"].append(owner)
        t = {k: torch.tensor(np.array(v), device=device) for k, v in rows.items()}
        self.p, self.P, self.owner, self.order = t["p"], t["P"], t["owner"], la + lb
        self.n_pairs, self.pairs = len(pairs), pairs
        # E[d][i][j][t] along each axis
        E = [[[None] * (lb + 1) for _ in range(la + 1)] for _ in range(3)]
        for d in range(3):
            zero = torch.zeros_like(self.p)

            def get(row, t_, zero=zero):
                return row[t_] if 0 <= t_ < len(row) else zero

            def raised(row, x, p=self.p):
                return [get(row, t_ - 1) / (2 * p) + x * get(row, t_) + (t_ + 1) * get(row, t_ + 1)
                        for t_ in range(len(row) + 1)]
            E[d][0][0] = [torch.exp(t["ab"][:, d])]
            for i in range(la + 1):
                if i:
                    E[d][i][0] = raised(E[d][i - 1][0], t["PA"][:, d])
                for j in range(1, lb + 1):
                    E[d][i][j] = raised(E[d][i][j - 1], t["PB"][:, d])
        herm = _hermites(la + lb)
        e = torch.zeros((len(self.p), _ncart(la), _ncart(lb), len(herm)), dtype=torch.float64,
                        device=device)
        for (x, a), (y, b), (h, c) in itertools.product(enumerate(_comps(la)), enumerate(_comps(lb)),
                                                        enumerate(herm)):
            if all(c[d] <= a[d] + b[d] for d in range(3)):
                e[:, x, y, h] = t["c"] * math.prod((E[d][a[d]][b[d]][c[d]] for d in range(3)),
                                                   start=torch.ones_like(self.p))
        fa, fb = (torch.tensor(_functions(l, coord), device=device) for l in (la, lb))
        e = torch.einsum("rabh,xa,yb->rxyh", e, fa, fb)
        self.nfun = (e.shape[1], e.shape[2])
        self.E = e.reshape(len(self.p), -1, len(herm))


def _contraction(shell, raw):
    """Contraction coefficients with the primitives' norm (2a/pi)^(3/4) (4a)^(l/2), scaled so that
    the contracted function has unit norm (unless ``raw``)."""
    l, _, e, c = shell
    c = c * (2 * e / math.pi) ** 0.75 * (4 * e) ** (l / 2.0)
    s = e[:, None] + e[None, :]
    return c if raw else c / math.sqrt(c @ ((math.pi / s) ** 1.5 / (2 * s) ** l) @ c)


def _groups(shells, coord, raw, device, pairs=None):
    by = {}
    for i, j in pairs or itertools.combinations_with_replacement(range(len(shells)), 2):
        by.setdefault((shells[i][0], shells[j][0]), []).append((i, j))
    return [_Pairs(la, lb, v, shells, coord, raw, device) for (la, lb), v in sorted(by.items())]


def _repulsion_block(bra, ket, potential, omega):
    """(pairs, functions, pairs, functions) of two groups of shell pairs."""
    hb, hk = _hermites(bra.order), _hermites(ket.order)
    order = bra.order + ket.order
    sign = torch.tensor([(-1.0) ** sum(c) for c in hk], dtype=torch.float64, device=bra.p.device)
    ek = ket.E * sign
    nfb, nfk = bra.E.shape[1], ket.E.shape[1]
    out = torch.zeros((bra.n_pairs, ket.n_pairs, nfb, nfk), dtype=torch.float64,
                      device=bra.p.device)
    step = max(1, int(3e8 / (len(ket.p) * (math.comb(order + 4, 4) + len(hb) * len(hk)))))
    for r0 in range(0, len(bra.p), step):
        r = slice(r0, r0 + step)
        p, q = bra.p[r, None], ket.p[None, :]
        alpha = p * q / (p + q)
        pref = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        x = [bra.P[r, d, None] - ket.P[None, :, d] for d in range(3)]
        t = alpha * (x[0] ** 2 + x[1] ** 2 + x[2] ** 2)
        f = alpha_f = None
        if potential != "erf":
            f, alpha_f = _boys(order, t), alpha
        values = _hermite_integrals(order, alpha_f, x, f) if f else None
        if potential in ("erf", "erfc"):
            s = omega ** 2 / (omega ** 2 + alpha)
            long = _hermite_integrals(order, alpha * s, x,
                                      [torch.sqrt(s) * v for v in _boys(order, s * t)])
            values = ({k: values[k] - v for k, v in long.items() if k[3] == 0} if values
                      else long)
        rpq = torch.stack([torch.stack([values[(*(a + b for a, b in zip(c, d)), 0)] for d in hk], -1)
                           for c in hb], -2) * pref[..., None, None]
        half = torch.einsum("rfh,rshk->rsfk", bra.E[r], rpq)
        full = torch.einsum("rsfk,sgk->rsfg", half, ek)
        per_ket = torch.zeros((full.shape[0], ket.n_pairs, nfb, nfk), dtype=torch.float64,
                              device=full.device).index_add_(1, ket.owner, full)
        out.index_add_(0, bra.owner[r], per_ket)
    return out


def _tensor(shells, coord, raw=False, potential="coulomb", omega=0.0):
    """The chemist tensor (N, N, N, N) of plain shells."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    groups = _groups(shells, coord, raw, device)
    width = [2 * l + 1 if coord == "spherical" else _ncart(l) for l, *_ in shells]
    first = np.cumsum([0] + width)
    n = int(first[-1])
    # pair functions, group after group: their place in the matrix of (n, n) function pairs
    place, start = torch.zeros((n, n), dtype=torch.int64, device=device), [0]
    for g in groups:
        na, nb = g.nfun
        for k, (i, j) in enumerate(g.pairs):
            at = (torch.arange(na * nb, device=device).reshape(na, nb) + start[-1] + k * na * nb)
            place[first[i]:first[i] + na, first[j]:first[j] + nb] = at
            place[first[j]:first[j] + nb, first[i]:first[i] + na] = at.T
        start.append(start[-1] + g.n_pairs * na * nb)
    m = torch.empty((start[-1], start[-1]), dtype=torch.float64, device=device)
    for x, bra in enumerate(groups):
        for y, ket in enumerate(groups[:x + 1]):
            b = _repulsion_block(bra, ket, potential, omega).permute(0, 2, 1, 3)
            b = b.reshape(start[x + 1] - start[x], start[y + 1] - start[y])
            m[start[x]:start[x + 1], start[y]:start[y + 1]] = b
            m[start[y]:start[y + 1], start[x]:start[x + 1]] = b.T
    at = place.reshape(-1)
    return m[at][:, at].reshape(n, n, n, n)


def _cost(shells):
    """Primitive quartets times Hermite products: about what _tensor does."""
    rows = {}
    for (la, *_, ca), (lb, *_, cb) in itertools.combinations_with_replacement(shells, 2):
        rows[la + lb] = rows.get(la + lb, 0) + len(ca) * len(cb)
    return sum(n1 * n2 * (160 + math.comb(a + b + 4, 4) + 6 * math.comb(a + 3, 3) * math.comb(b + 3, 3))
               for a, n1 in rows.items() for b, n2 in rows.items() if a >= b)


def exact(case, seed):
    kind, coord = case["kind"], case.get("coord", "cartesian")
    mols = _molecules(case, seed)
    if kind == "nuclear":
        return _attraction(mols[0], coord, *_points(case, seed)).cpu().numpy()
    # the whole case within a few seconds on a GPU, and its tensors within its memory
    if sum(_cost(m) for m in mols) > 4e11 or max(sum(_ncart(l) for l, *_ in m) for m in mols) > 125:
        return None
    if kind in ("batch", "batch_call"):
        return [_tensor(m, coord) for m in mols]
    if kind == "attenuated":
        return _tensor(mols[0], coord, potential=case["potential"], omega=case["omega"]).cpu().numpy()
    eri = _tensor(mols[0], coord, raw=kind == "quartet")
    if kind == "resident":
        return eri
    if kind == "tensor":
        eri = eri.cpu().numpy()
        return eri.transpose(0, 2, 1, 3) if case["notation"] == "physicist" else eri
    n = eri.shape[0]
    if kind == "quartet":
        w = [_ncart(l) for l, *_ in mols[0]]
        o = np.cumsum([0] + w)
        block = eri[o[0]:o[1], o[1]:o[2], o[2]:o[3], o[3]:o[4]]
        return block.cpu().numpy().reshape(1, w[0], 1, w[1], 1, w[2], 1, w[3])
    if kind in ("coulomb", "jk"):
        d = torch.tensor(_density(case, n, seed), device=eri.device)
        j = torch.einsum("abcd,cd->ab", eri, d).cpu().numpy()
        return j if kind == "coulomb" else (j, torch.einsum("abcd,bd->ac", eri, d).cpu().numpy())
    t = torch.tensor(_transform(case, n, seed), device=eri.device)
    for _ in range(4):
        eri = torch.tensordot(eri, t, dims=([0], [1]))
    return eri.cpu().numpy()


def _attraction(shells, coord, points, charges):
    """The sum over the points of -q (a| 1/|r - R| |b)."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    width = [2 * l + 1 if coord == "spherical" else _ncart(l) for l, *_ in shells]
    first = np.cumsum([0] + width)
    out = torch.zeros((int(first[-1]),) * 2, dtype=torch.float64, device=device)
    pts, q = torch.tensor(points, device=device), torch.tensor(charges, device=device)
    for g in _groups(shells, coord, False, device):
        x = [g.P[:, d, None] - pts[None, :, d] for d in range(3)]
        p = g.p[:, None]
        f = _boys(g.order, p * (x[0] ** 2 + x[1] ** 2 + x[2] ** 2))
        r = _hermite_integrals(g.order, p, x, f)
        v = torch.stack([(r[(*c, 0)] * (-2.0 * math.pi / p) * q).sum(1) for c in _hermites(g.order)], -1)
        rows = torch.einsum("rfh,rh->rf", g.E, v)
        total = torch.zeros((g.n_pairs, rows.shape[1]), dtype=torch.float64,
                            device=device).index_add_(0, g.owner, rows)
        na, nb = g.nfun
        for k, (i, j) in enumerate(g.pairs):
            b = total[k].reshape(na, nb)
            out[first[i]:first[i] + na, first[j]:first[j] + nb] = b
            out[first[j]:first[j] + nb, first[i]:first[i] + na] = b.T
    return out
