"""Performance cases: the calls that programs on top of lible_b200 spend their time in, over the range
of sizes they are made with.

Inputs are the seeded water clusters and densities of lible_b200.workloads.  What stands for what:

- "jk": one direct J/K build of an SCF iteration, with the density and the outputs on the device and the
  structure and its screening plan kept between iterations.  From one water molecule, where launches and
  latency count, to 32 molecules; double- and triple-zeta bases; FP64 and mixed precision.
- "batch": J/K of many molecules at once, replayed as one graph.
- "grad": the J/K energy gradient of a geometry step.
- "rij", "rik": the Coulomb and exchange builds of an SCF iteration with the resolution of the identity, host
  arrays in and out, the tensors and the metric factor kept from the first iteration.
- "rijgrad": the RI-J gradient of a geometry step.
- "one": the overlap, kinetic-energy and nuclear-attraction matrices of a new structure.
- "eri4": the whole four-centre tensor of a small molecule in host memory.
"""
import math
import os

import numpy as np
import torch

from lible_b200 import ints
from lible_b200.workloads import random_density, water_cluster

JKFIT = "def2-universal-jkfit"
SCHWARZ = 1e-12


def listed():
    return [
        # the smallest build: a water molecule, 24 functions
        {"name": "jk_h2o_dz", "kind": "jk", "waters": 1, "basis": "cc-pvdz", "precision": "fp64"},
        # an odd, ordinary molecule in a basis without shared core exponents
        {"name": "jk_h2o5_svp", "kind": "jk", "waters": 5, "basis": "def2-svp", "precision": "fp64"},
        # the cluster of the J/K configuration, 384 functions
        {"name": "jk_h2o16_dz", "kind": "jk", "waters": 16, "basis": "cc-pvdz", "precision": "fp64"},
        # the headline workload of the benchmark, 768 functions, mixed precision
        {"name": "jk_h2o32_dz_mixed", "kind": "jk", "waters": 32, "basis": "cc-pvdz", "precision": "mixed"},
        # the triple-zeta cluster (f functions, every class to (ff|ff)), 464 functions
        {"name": "jk_h2o8_tz", "kind": "jk", "waters": 8, "basis": "cc-pvtz", "precision": "fp64"},
        # a batch of small clusters, half double-, half triple-zeta
        {"name": "batch_24", "kind": "batch", "molecules": 24, "max_waters": 4, "precision": "fp64"},
        # the gradient configuration
        {"name": "grad_h2o8_tz", "kind": "grad", "waters": 8, "basis": "cc-pvtz"},
        # RI with the universal fitting set: 3,616 / 1,808 / 1,356 auxiliary functions
        {"name": "rij_h2o32_dz", "kind": "rij", "waters": 32, "basis": "cc-pvdz", "aux": JKFIT},
        {"name": "rik_h2o16_dz", "kind": "rik", "waters": 16, "basis": "cc-pvdz", "aux": JKFIT},
        {"name": "rijgrad_h2o12_dz", "kind": "rijgrad", "waters": 12, "basis": "cc-pvdz", "aux": JKFIT},
        # set-up matrices of the largest cluster
        {"name": "one_h2o32_dz", "kind": "one", "waters": 32, "basis": "cc-pvdz"},
        # the full tensor of a water molecule
        {"name": "eri4_h2o_dz", "kind": "eri4", "waters": 1, "basis": "cc-pvdz"},
    ]


def draw(rng):
    def size(hi):
        return min(hi, int(math.exp(rng.uniform(0.0, math.log(hi + 1.0)))))

    kind = rng.choice(["jk", "jk", "jk", "batch", "grad", "rij", "rik", "rijgrad", "one", "eri4"])
    case = {"kind": kind}
    if kind == "batch":
        case.update(molecules=rng.randint(2, 24), max_waters=rng.randint(1, 4), precision=rng.choice(["fp64", "mixed"]))
        return case
    if kind == "eri4":
        waters, basis = rng.choice([(1, "6-31+g"), (2, "6-31+g"), (1, "def2-svp"), (2, "def2-svp"), (2, "cc-pvdz"),
                                    (1, "def2-tzvp"), (1, "cc-pvtz")])
        case.update(waters=waters, basis=basis)
        return case
    basis = rng.choice(["6-31+g", "def2-svp", "cc-pvdz", "def2-tzvp", "cc-pvtz"])
    large = basis in ("cc-pvtz", "def2-tzvp")
    if kind == "jk":
        case.update(waters=size(8 if large else 32), basis=basis, precision=rng.choice(["fp64", "mixed"]))
    elif kind == "grad":
        case.update(waters=size(7 if large else 14), basis=basis)
    elif kind == "one":
        case.update(waters=size(12 if large else 32), basis=basis)
    else:
        aux = rng.choice([JKFIT, "cc-pvdz-rifit"])
        case.update(waters=size(6 if large else 16), basis=basis, aux=aux)
    return case


def _clusters(case, seed):
    """The molecules of a case: [(basis, atomic numbers, coordinates in bohr, generator)]."""
    if case["kind"] == "batch":
        out = []
        for i in range(case["molecules"]):
            Z, xyz, rng = water_cluster(1 + i // 2 % case["max_waters"], seed * 1000 + i)
            out.append(("cc-pvtz" if i % 2 else "cc-pvdz", Z, xyz, rng))
        return out
    Z, xyz, rng = water_cluster(case["waters"], seed)
    return [(case["basis"], Z, xyz, rng)]


def _structure(case, seed):
    basis, Z, xyz, rng = _clusters(case, seed)[0]
    return ints.Structure(basis, Z, xyz, case.get("aux"), units="bohr"), rng


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "batch":
        mols = _clusters(case, seed)
        s = ints.Batch([(b, Z, xyz) for b, Z, xyz, _ in mols], units="bohr")
        D = s.pack([random_density(int(n), 5 * len(m[1]) // 3, m[3]) for n, m in zip(s.nao, mols)])
        state.update(s=s, D=torch.tensor(D, device="cuda"), precision=case["precision"])
    else:
        s, rng = _structure(case, seed)
        occ = 5 * case["waters"]
        state["s"] = s
        if kind in ("jk", "grad", "rij", "rijgrad"):
            D = random_density(s.nao, occ, rng)
            state["D"] = torch.tensor(D, device="cuda") if kind == "jk" else D
        if kind == "rik":
            state["C"] = np.ascontiguousarray(np.linalg.qr(rng.standard_normal((s.nao, occ)))[0])
        if kind == "jk":
            state["precision"] = case["precision"]
    if kind in ("jk", "batch"):
        state["J"], state["K"] = torch.empty_like(state["D"]), torch.empty_like(state["D"])
        ints.jk_plan(s, SCHWARZ, case["precision"])
        torch.cuda.synchronize()
    elif kind == "grad":
        ints.jk_plan(s, SCHWARZ, "fp64", 0.0)
    elif kind == "rij":
        ints.rij(s, state["D"], SCHWARZ)
    elif kind == "rik":
        ints.rik(s, C=state["C"], schwarz=SCHWARZ)
    elif kind == "rijgrad":
        ints.rij_grad(s, state["D"], SCHWARZ)
    return state


def run(state):
    kind, s = state["kind"], state["s"]
    if kind in ("jk", "batch"):
        J, K, _ = ints.jk(s, state["D"], SCHWARZ, state["precision"], J=state["J"], K=state["K"],
                          use_graph=kind == "batch")
        return J, K
    if kind == "grad":
        return ints.jk_energy_backward(s, state["D"], SCHWARZ)
    if kind == "rij":
        return ints.rij(s, state["D"], SCHWARZ)
    if kind == "rik":
        return ints.rik(s, C=state["C"], schwarz=SCHWARZ)
    if kind == "rijgrad":
        return ints.rij_grad(s, state["D"], SCHWARZ)
    if kind == "one":
        return ints.one_electron(s)
    return ints.eri4(s)


def work(case):
    """Bytes: inputs read and outputs written once; for the RI builds also the resident tensors that every call
    has to stream.  Operations: the multiply-adds of the McMurchie-Davidson evaluation of the quartets
    that survive the screening (three times as many for a gradient, one per independent centre),
    or of the tensor contractions."""
    kind = case["kind"]
    if kind == "batch":
        s = ints.Batch([(b, Z, xyz) for b, Z, xyz, _ in _clusters(case, 1)], units="bohr")
        plan = ints.jk_plan(s, SCHWARZ, case["precision"])
        return {"bytes": 24.0 * s.packed, "flops": plan["flops_fp64"] + plan["flops_fp32"]}
    s, _ = _structure(case, 1)
    n, na, occ, nat = float(s.nao), float(s.naux), 5.0 * case["waters"], float(s.n_atoms)
    tri = n * (n + 1) / 2
    if kind in ("jk", "grad", "eri4"):
        plan = ints.jk_plan(s, 0.0 if kind == "eri4" else SCHWARZ, case.get("precision", "fp64"))
        f = plan["flops_fp64"] + plan["flops_fp32"]
        if kind == "jk":
            return {"bytes": 24.0 * n * n, "flops": f}
        return {"bytes": 8.0 * n ** 4, "flops": f} if kind == "eri4" else {"bytes": 8.0 * n * n + 24.0 * nat, "flops": 3.0 * f}
    if kind == "rij":
        return {"bytes": 16.0 * na * tri + 8.0 * na * na + 16.0 * n * n, "flops": 4.0 * na * tri + 2.0 * na * na}
    if kind == "rik":
        return {"bytes": 8.0 * na * n * n + 8.0 * n * n, "flops": 2.0 * na * n * n * occ + 2.0 * na * occ * tri}
    if kind == "rijgrad":
        # about a hundred operations for each three-centre derivative integral and density product
        return {"bytes": 8.0 * n * n + 8.0 * na * na, "flops": 100.0 * na * tri}
    # one-electron: about ten primitive pairs a function pair, a hundred operations for each with a nucleus
    return {"bytes": 24.0 * n * n, "flops": 1000.0 * tri * nat}


# ------------------------------------------------------------------------------------------------
# Reference values in 64 bits: the same integrals in plain torch, from the basis files' numbers.

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_DATA = os.path.join("lible_b200", "basis")


def _basis_shells(group, name, Z, xyz):
    """[(l, centre, exponents, coefficients, first function)] in the order atom, shell."""
    for family in sorted(os.listdir(os.path.join(_DATA, group))):
        path = os.path.join(_DATA, group, family, name + ".txt")
        if os.path.exists(path):
            break
    elements, z = {}, None
    lines = iter(open(path))
    for line in lines:
        line = line.strip()
        if line.startswith("element="):
            z = int(line[8:])
            elements[z] = []
        elif line.startswith("l="):
            l, n = (int(x.split("=")[1]) for x in line.split())
            rows = [[float(v) for v in next(lines).split()] for _ in range(n)]
            elements[z].append((l, [r[0] for r in rows], [r[1] for r in rows]))
    out, ofs = [], 0
    for z, r in zip(Z, xyz):
        for l, e, c in elements[z]:
            # coefficients of normalised primitives, scaled to a normalised contraction (radial part)
            e, c = np.array(e), np.array(c)
            prim = c * (2 * e) ** (0.5 * l + 0.75)
            s = (prim[:, None] * prim[None, :] * (e[:, None] + e[None, :]) ** (-l - 1.5)).sum()
            out.append((l, np.asarray(r, dtype=float), e, prim / math.sqrt(s), ofs))
            ofs += 2 * l + 1
    return out, ofs


def _carts(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _double_factorial(n):
    return math.prod(range(n, 0, -2)) if n > 0 else 1


def _solid(l):
    """Rows m = 0, +1, -1, ... of the real solid harmonics over x^i y^j z^k, each row scaled so that the
    function with radial normalisation 1 as in _basis_shells is normalised."""
    carts, rows = _carts(l), []
    for r in range(2 * l + 1):
        m = 0 if r == 0 else (r + 1) // 2 if r % 2 else -(r // 2)
        am, row = abs(m), np.zeros(len(carts))
        for t in range((l - am) // 2 + 1):
            for u in range(t + 1):
                for w in range(1 if m < 0 else 0, am + 1, 2):
                    k = carts.index((2 * t + am - 2 * u - w, 2 * u + w, l - 2 * t - am))
                    row[k] += (-1.0) ** (t + w // 2) * 0.25 ** t * math.comb(l, t) * math.comb(l - t, am + t) * math.comb(t, u) * math.comb(am, w)
        # squared norm of the polynomial times e^{-r^2/2 * 2 a}, with the radial factor taken out
        q = 0.0
        for i, a in enumerate(carts):
            for j, b in enumerate(carts):
                p = [x + y for x, y in zip(a, b)]
                if row[i] and row[j] and not any(x % 2 for x in p):
                    q += row[i] * row[j] * math.prod(_double_factorial(x - 1) for x in p) / 2.0 ** l
        rows.append(row / math.sqrt(q * math.pi ** 1.5))
    return np.array(rows)


def _herm(L):
    return [(t, u, n - t - u) for n in range(L + 1) for t in range(n, -1, -1) for u in range(n - t, -1, -1)]


class _Pairs:
    """All shell pairs of one class (la, lb) of two shell lists, with their primitive pairs flattened."""

    def __init__(self, bra, ket, la, lb, same, raise_b=0, unit=False):
        self.la, self.lb, self.pairs = la, lb, []
        prim = []
        for i, A in enumerate(bra):
            for j, B in enumerate(ket):
                if A[0] != la or B[0] != lb or (same and j > i):
                    continue
                for a, ca in zip(A[2], A[3]):
                    for b, cb in zip(B[2], B[3]):
                        mu = a * b / (a + b)
                        if abs(ca * cb) * math.exp(-mu * float(((A[1] - B[1]) ** 2).sum())) > 1e-20:
                            prim.append((a, b, *A[1], *B[1], ca * cb, len(self.pairs)))
                self.pairs.append((A[4], B[4]))
        p = torch.tensor(prim, dtype=torch.float64, device=_DEV).reshape(-1, 10)
        self.a, self.b, self.A, self.B, self.c = p[:, 0], p[:, 1], p[:, 2:5], p[:, 5:8], p[:, 8]
        self.of = p[:, 9].long()
        self.p = self.a + self.b
        self.P = (self.a[:, None] * self.A + self.b[:, None] * self.B) / self.p[:, None]
        mu = self.a * self.b / self.p
        lbx = lb + raise_b
        self.E1 = []
        for x in range(3):
            pa, pb = self.P[:, x] - self.A[:, x], self.P[:, x] - self.B[:, x]
            E = {(0, 0): [torch.exp(-mu * (self.A[:, x] - self.B[:, x]) ** 2)]}
            for i in range(la + 1):
                for j in range(lbx + 1):
                    if (i, j) == (0, 0):
                        continue
                    src, d = (E[(i, j - 1)], pb) if j else (E[(i - 1, j)], pa)
                    n = i + j
                    E[(i, j)] = [(src[t] * d if t < n else 0) + (src[t - 1] * (0.5 / self.p) if t else 0) +
                                 ((t + 1) * src[t + 1] if t + 1 < n else 0) for t in range(n + 1)]
            self.E1.append(E)
        self.Ta = torch.tensor(_solid(la), device=_DEV)
        self.Tb = torch.ones(1, 1, dtype=torch.float64, device=_DEV) if unit else torch.tensor(_solid(lb), device=_DEV)

    def spherical(self, cart):
        """[primitive, cart a, cart b, ...] -> [primitive, m a * m b, ...] with the coefficients."""
        r = torch.einsum("mi,nj,pij...->pmn...", self.Ta, self.Tb, cart)
        return (r.flatten(1, 2).transpose(0, -1) * self.c).transpose(0, -1)

    def hermite(self):
        """E [primitive, m a * m b, tuv]."""
        hs = _herm(self.la + self.lb)
        cart = torch.zeros(len(self.p), len(_carts(self.la)), len(_carts(self.lb)), len(hs), dtype=torch.float64, device=_DEV)
        for i, ca in enumerate(_carts(self.la)):
            for j, cb in enumerate(_carts(self.lb)):
                e = [self.E1[x][(ca[x], cb[x])] for x in range(3)]
                for h, tuv in enumerate(hs):
                    if all(tuv[x] <= ca[x] + cb[x] for x in range(3)):
                        cart[:, i, j, h] = e[0][tuv[0]] * e[1][tuv[1]] * e[2][tuv[2]]
        return self.spherical(cart)


def _boys(M, x):
    """F_0 .. F_M: the ascending series and downward recursion below 36, upward recursion above."""
    big = x > 36.0
    s = torch.where(big, torch.ones_like(x), x)
    term = torch.full_like(s, 1.0 / (2 * M + 1))
    top = term.clone()
    for k in range(1, 170):
        term = term * (2.0 * s) / (2 * M + 2 * k + 1)
        top += term
    ex = torch.exp(-s)
    F = [None] * (M + 1)
    F[M] = top * ex
    for m in range(M - 1, -1, -1):
        F[m] = (2.0 * s * F[m + 1] + ex) / (2 * m + 1)
    g, exb = torch.where(big, x, torch.full_like(x, 40.0)), torch.exp(-x)
    up = 0.5 * torch.sqrt(math.pi / g)
    for m in range(M + 1):
        F[m] = torch.where(big, up, F[m])
        up = ((2 * m + 1) * up - exb) / (2.0 * g)
    return F


def _coulomb(L, alpha, r):
    """R_tuv [..., tuv] of distance vectors r [..., 3]."""
    F = _boys(L, alpha * (r * r).sum(-1))
    level = {(0, 0, 0): None}
    for n in range(L, -1, -1):
        new = {}
        for t, u, v in _herm(L - n):
            if t + u + v == 0:
                new[(0, 0, 0)] = (-2.0 * alpha) ** n * F[n]
                continue
            x = 0 if t else 1 if u else 2
            k = [t, u, v]
            k[x] -= 1
            val = r[..., x] * level[tuple(k)]
            if k[x]:
                m = list(k)
                m[x] -= 1
                val = val + k[x] * level[tuple(m)]
            new[(t, u, v)] = val
        level = new
    return torch.stack([level[h] for h in _herm(L)], -1)


def _contract(X, Y):
    """(X|Y) of two pair classes: [pair x, m, pair y, m']."""
    EX, EY = X.hermite(), Y.hermite()
    hx, hy = _herm(X.la + X.lb), _herm(Y.la + Y.lb)
    L = X.la + X.lb + Y.la + Y.lb
    where = {h: i for i, h in enumerate(_herm(L))}
    at = torch.tensor([[where[tuple(a + b for a, b in zip(h, g))] for g in hy] for h in hx], device=_DEV)
    EY = EY * torch.tensor([(-1.0) ** sum(g) for g in hy], dtype=torch.float64, device=_DEV)
    out = torch.zeros(len(X.pairs), EX.shape[1], len(Y.pairs), EY.shape[1], dtype=torch.float64, device=_DEV)
    step = max(1, int(4e7) // max(1, len(Y.p) * len(hx) * len(hy)))
    for i in range(0, len(X.p), step):
        px, py = X.p[i:i + step, None], Y.p[None, :]
        alpha = px * py / (px + py)
        R = _coulomb(L, alpha, X.P[i:i + step, None, :] - Y.P[None, :, :])
        R = R * (2.0 * math.pi ** 2.5 / (px * py * torch.sqrt(px + py)))[..., None]
        g = torch.einsum("pqhk,qck->pqhc", R[..., at], EY)
        k = torch.zeros(g.shape[0], len(Y.pairs), g.shape[2], g.shape[3], dtype=torch.float64, device=_DEV).index_add_(1, Y.of, g)
        out.index_add_(0, X.of[i:i + step], torch.einsum("psh,pyhc->psyc", EX[i:i + step], k))
    return out


def _classes(shells):
    top = max(s[0] for s in shells)
    return [_Pairs(shells, shells, la, lb, la == lb) for la in range(top + 1) for lb in range(la + 1)
            if any(s[0] == la for s in shells) and any(s[0] == lb for s in shells)]


def _tensor4(shells, n):
    V = torch.zeros(n, n, n, n, dtype=torch.float64, device=_DEV)
    cls = _classes(shells)
    for i, X in enumerate(cls):
        for Y in cls[:i + 1]:
            sa, sb, sc, sd = (2 * l + 1 for l in (X.la, X.lb, Y.la, Y.lb))
            blocks = _contract(X, Y)
            for x, (oa, ob) in enumerate(X.pairs):
                for y, (oc, od) in enumerate(Y.pairs):
                    v = blocks[x, :, y, :].reshape(sa, sb, sc, sd)
                    a, b, c, d = slice(oa, oa + sa), slice(ob, ob + sb), slice(oc, oc + sc), slice(od, od + sd)
                    for w, p, q in ((v, a, b), (v.transpose(0, 1), b, a)):
                        V[p, q, c, d] = w
                        V[p, q, d, c] = w.transpose(2, 3)
                        V[c, d, p, q] = w.permute(2, 3, 0, 1)
                        V[d, c, p, q] = w.permute(3, 2, 0, 1)
    return V


def _tensors_ri(shells, n, aux, na):
    unit = (0, None, np.zeros(1), np.ones(1), 0)
    cls = []
    for l in range(max(s[0] for s in aux) + 1):
        of_l = [s for s in aux if s[0] == l]
        X = None
        for s in of_l:
            Y = _Pairs([s], [(0, s[1], unit[2], unit[3], 0)], l, 0, False, unit=True)
            if X is None:
                X = Y
            else:
                Y.of = Y.of + len(X.pairs)
                X.pairs += Y.pairs
                for k in ("a", "b", "A", "B", "c", "of", "p", "P"):
                    setattr(X, k, torch.cat([getattr(X, k), getattr(Y, k)]))
                X.E1 = [{ij: [torch.cat([u, v]) for u, v in zip(X.E1[x][ij], Y.E1[x][ij])] for ij in X.E1[x]} for x in range(3)]
        if X is not None:
            cls.append(X)
    T = torch.zeros(n, n, na, dtype=torch.float64, device=_DEV)
    M = torch.zeros(na, na, dtype=torch.float64, device=_DEV)
    for X in _classes(shells):
        for Y in cls:
            sa, sb, sc = 2 * X.la + 1, 2 * X.lb + 1, 2 * Y.la + 1
            blocks = _contract(X, Y)
            at = torch.tensor([o + k for o, _ in Y.pairs for k in range(sc)], device=_DEV)
            for x, (oa, ob) in enumerate(X.pairs):
                v = blocks[x].reshape(sa, sb, -1)
                T[oa:oa + sa, ob:ob + sb, at] = v
                T[ob:ob + sb, oa:oa + sa, at] = v.transpose(0, 1)
    for X in cls:
        ax = torch.tensor([o + k for o, _ in X.pairs for k in range(2 * X.la + 1)], device=_DEV)
        for Y in cls:
            ay = torch.tensor([o + k for o, _ in Y.pairs for k in range(2 * Y.la + 1)], device=_DEV)
            M[ax[:, None], ay[None, :]] = _contract(X, Y).flatten(2, 3).flatten(0, 1)
    return T, M


def _one_electron(shells, n, Z, xyz):
    out = torch.zeros(3, n, n, dtype=torch.float64, device=_DEV)
    q = torch.tensor([float(z) for z in Z], device=_DEV, dtype=torch.float64)
    C = torch.tensor(np.asarray(xyz, dtype=float), device=_DEV)
    top = max(s[0] for s in shells)
    for la in range(top + 1):
        for lb in range(la + 1):
            X = _Pairs(shells, shells, la, lb, la == lb, raise_b=2)
            if not X.pairs:
                continue
            root = torch.sqrt(math.pi / X.p)

            def s1(x, i, j):
                return X.E1[x][(i, j)][0] * root if j >= 0 else 0.0 * root

            def t1(x, i, j):
                r = -2.0 * X.b ** 2 * s1(x, i, j + 2) + X.b * (2 * j + 1) * s1(x, i, j)
                return r - 0.5 * j * (j - 1) * s1(x, i, j - 2) if j > 1 else r

            S = torch.zeros(len(X.p), len(_carts(la)), len(_carts(lb)), dtype=torch.float64, device=_DEV)
            T = torch.zeros_like(S)
            for i, a in enumerate(_carts(la)):
                for j, b in enumerate(_carts(lb)):
                    s, t = ([f(x, a[x], b[x]) for x in range(3)] for f in (s1, t1))
                    S[:, i, j] = s[0] * s[1] * s[2]
                    T[:, i, j] = t[0] * s[1] * s[2] + s[0] * t[1] * s[2] + s[0] * s[1] * t[2]
            L = la + lb
            R = torch.zeros(len(X.p), len(_herm(L)), dtype=torch.float64, device=_DEV)
            step = max(1, int(1e7) // (len(q) * len(_herm(L))))
            for k in range(0, len(X.p), step):
                r = _coulomb(L, X.p[k:k + step, None], X.P[k:k + step, None, :] - C[None])
                R[k:k + step] = torch.einsum("pch,c->ph", r, -q) * (2.0 * math.pi / X.p[k:k + step])[:, None]
            for k, prim in enumerate((X.spherical(S), X.spherical(T), torch.einsum("psh,ph->ps", X.hermite(), R))):
                sa, sb = 2 * la + 1, 2 * lb + 1
                v = torch.zeros(len(X.pairs), sa * sb, dtype=torch.float64, device=_DEV).index_add_(0, X.of, prim)
                v = v.reshape(-1, sa, sb)
                ab = torch.tensor(X.pairs, device=_DEV)
                rows = (ab[:, 0, None, None] + torch.arange(sa, device=_DEV)[None, :, None]).expand_as(v)
                cols = (ab[:, 1, None, None] + torch.arange(sb, device=_DEV)[None, None, :]).expand_as(v)
                out[k][rows, cols] = v
                out[k][cols, rows] = v
    return [m.cpu().numpy() for m in out]


def exact(case, seed):
    """The same results from dense tensors; None where those would take too long (more than 60 functions,
    and the gradients)."""
    kind = case["kind"]
    if kind in ("batch", "grad", "rijgrad"):
        return None
    basis, Z, xyz, rng = _clusters(case, seed)[0]
    shells, n = _basis_shells("main", basis, Z, xyz)
    if kind == "one":
        return _one_electron(shells, n, Z, xyz) if len(Z) <= 48 else None
    if n > 60:
        return None
    occ = 5 * case["waters"]
    if kind == "eri4":
        return _tensor4(shells, n).cpu().numpy()
    if kind == "jk":
        D = torch.tensor(random_density(n, occ, rng), device=_DEV)
        V = _tensor4(shells, n)
        return [torch.einsum("mnls,ls->mn", V, D), torch.einsum("mlns,ls->mn", V, D)]
    aux, na = _basis_shells("aux", case["aux"], Z, xyz)
    T, M = _tensors_ri(shells, n, aux, na)
    if kind == "rij":
        D = torch.tensor(random_density(n, occ, rng), device=_DEV)
        gamma = torch.einsum("mnP,mn->P", T, D)
        d = torch.linalg.solve(M, gamma)
        return [(T @ d).cpu().numpy(), gamma.cpu().numpy(), d.cpu().numpy()]
    C = torch.tensor(np.linalg.qr(rng.standard_normal((n, occ)))[0], device=_DEV)
    Y = torch.einsum("mlP,li->miP", T, C).reshape(n * occ, na)
    W = torch.linalg.solve(M, Y.T).T
    return (Y.reshape(n, -1) @ W.reshape(n, -1).T).cpu().numpy()
