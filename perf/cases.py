"""Timed workloads of the two-electron engine, through its public entry points.

Each case is one call (or, for the whole SCF, one run) that a user's program repeats: the
host-pointer Fock hooks, the device-pointer J/K build of an SCF loop (FP64 and mixed
precision), the UHF Fock build, the adjoint gradient and Hessian, the batched J/K build, and a
complete SCF with its gradient.  Molecules and basis sets are those of ``hfscf_b200.molecules``
(water clusters, all-trans alkanes, anthracene, the seeded batch mix), displaced and turned by
the seed.  Densities are core-guess densities, the SCF loop's own first density, formed on the
host from the one-electron matrices.

``exact`` recomputes the same quantities in 64 bits without the engine: McMurchie-Davidson
Hermite expansions (J. Comput. Phys. 26, 218 (1978)) in plain torch, derivatives by autograd.
"""
from __future__ import annotations

import itertools
import math

import numpy as np
import torch

from hfscf_b200 import basis as B
from hfscf_b200 import batch as BT
from hfscf_b200 import engine as E
from hfscf_b200 import flopmodel
from hfscf_b200 import molecules as M
from hfscf_b200 import scf

PRECISION = {"fp64": E.FP64, "mixed": E.MIXED}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(name, op, molecule, size, basis, precision="fp64"):
    c = {"op": op, "molecule": molecule, "size": size, "basis": basis, "precision": precision}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest everyday calls: one water, host matrices in and out, where launches,
        # copies and latency are the time
        _case("water-fock", "fock", "water", 1, "cc-pvdz"),
        _case("water-grad", "grad", "water", 1, "6-31g*"),
        # one J/K build of the SCF loop of a mid-size organic molecule, device matrices: the
        # headline workload, and the same build in mixed precision
        _case("octane-jk", "jk", "alkane", 8, "6-31g**"),
        _case("octane-jk-mixed", "jk", "alkane", 8, "6-31g**", "mixed"),
        # spherical d and long contractions (cc-pVDZ)
        _case("anthracene-jk", "jk", "anthracene", 1, "cc-pvdz"),
        # an open-shell cation: J of the total density, K of both spins, host matrices
        _case("octamer-uhf", "uhf", "water", 8, "6-31g*"),
        # forces of a geometry step
        _case("octane-grad", "grad", "alkane", 8, "6-31g**"),
        _case("anthracene-grad-mixed", "grad", "anthracene", 1, "cc-pvdz", "mixed"),
        # second derivatives for frequencies, a small cluster and the largest call of all
        _case("tetramer-hess", "hess", "water", 4, "6-31g*"),
        _case("octane-hess", "hess", "alkane", 8, "6-31g**"),
        # many small molecules in one handle: one J/K build for all of them
        _case("batch-jk", "batch", "mix", 512, "mix"),
        # a whole calculation: SAD guess, SCF to tight convergence, gradient
        _case("dimer-scf", "scf", "water", 2, "6-31g*"),
    ]


def draw(rng):
    """One more case of the same ranges: every operation, molecules from one atom group to the
    largest listed, every basis set the molecules ship with."""
    op = rng.choice(["fock", "jk", "jk", "uhf", "grad", "grad", "hess", "batch", "scf"])
    if op == "batch":
        return _case(None, op, "mix", int(round(math.exp(rng.uniform(math.log(16), math.log(512))))), "mix",
                     rng.choice(["fp64", "mixed"]))
    if op == "scf":
        return _case(None, op, rng.choice(["water", "alkane"]), rng.randint(1, 4),
                     rng.choice(["sto-3g", "6-31g*", "6-31g**", "cc-pvdz"]))
    molecule = rng.choice(["water", "alkane", "alkane", "anthracene"] if op in ("fock", "jk", "grad")
                          else ["water", "alkane"])
    size = 1 if molecule == "anthracene" else int(round(math.exp(rng.uniform(0.0, math.log(8.4)))))
    basis = rng.choice(["sto-3g", "6-31g*", "6-31g**", "cc-pvdz"])
    if op == "hess" and basis == "cc-pvdz":
        size = min(size, 4)
    precision = "fp64" if op == "hess" else rng.choice(["fp64", "fp64", "mixed"])
    return _case(None, op, molecule, size, basis, precision)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _basis(case, seed):
    rng = np.random.default_rng([seed, case["size"]])
    if case["molecule"] == "water":
        Z, xyz = M.water_cluster(case["size"], 2.9, rng, 0.1)
    elif case["molecule"] == "alkane":
        Z, xyz = M.n_alkane(case["size"]) if case["size"] > 1 else M.methane()
    else:
        Z, xyz = M.anthracene()
    xyz = np.asarray(xyz, dtype=np.float64)
    xyz = (xyz + rng.normal(scale=0.02, size=xyz.shape)) @ M.random_rotation(rng).T
    return B.build_basis(case["basis"], Z, xyz * B.ANGSTROM_TO_BOHR, pure=case["basis"] == "cc-pvdz")


def _batch(case, seed):
    """The seeded mix of small molecules (its composition fixed by the count), moved by the seed."""
    rng = np.random.default_rng([seed, case["size"]])
    mix = M.batch_molecules(case["size"])
    return BT.batch_bases([(Z, x + rng.normal(scale=0.03, size=x.shape), name, pure) for Z, x, name, pure in mix])


def _core_guess(bs):
    """Core Hamiltonian and the occupied orbitals that diagonalise it (host, numpy)."""
    S, T, V = E.one_electron(bs)
    H = T + V
    X = scf.sym_orth(S)
    _, C = np.linalg.eigh(X.T @ H @ X)
    return H, X @ C


def _density(C, nocc):
    return np.ascontiguousarray(C[:, :nocc] @ C[:, :nocc].T)


def _inputs(case, seed):
    """Basis and host matrices of a single-molecule case."""
    bs = _basis(case, seed)
    H, C = _core_guess(bs)
    nel = int(np.sum(bs.Z))
    if case["op"] == "uhf":  # the doublet cation
        return bs, H, (_density(C, nel // 2), _density(C, (nel - 1) // 2))
    return bs, H, (_density(C, nel // 2),)


_STREAM = None


def _stream():
    """The stream a program shares between torch and its engines."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def prepare(case, seed):
    op = case["op"]
    st = {"op": op, "prec": PRECISION[case["precision"]], "stream": _stream()}
    f64 = dict(dtype=torch.float64, device="cuda")
    if op == "batch":
        bases = _batch(case, seed)
        eng = BT.BatchEngine(bases)
        D = np.concatenate([_density(_core_guess(b)[1], int(np.sum(b.Z)) // 2).ravel() for b in bases])
        st["D"] = torch.from_numpy(D).cuda()
        st["J"], st["K"] = torch.empty_like(st["D"]), torch.empty_like(st["D"])
    elif op == "scf":
        bs = _basis(case, seed)
        eng = E.Engine(bs)
        st["basis"] = bs
    else:
        bs, H, Ds = _inputs(case, seed)
        eng = E.Engine(bs)
        st["H"], st["host_D"] = H, Ds
        if op in ("jk", "grad", "hess"):
            st["D"] = torch.from_numpy(Ds[0]).cuda()
            n, na = bs.nbf, bs.natoms
            if op == "jk":
                st["J"], st["K"] = torch.empty((n, n), **f64), torch.empty((n, n), **f64)
            elif op == "grad":
                st["g"] = torch.zeros((na, 3), **f64)
            else:
                st["h"] = torch.zeros((3 * na, 3 * na), **f64)
    if op != "scf":
        eng.set_stream(st["stream"].cuda_stream)
    st["engine"] = eng
    torch.cuda.synchronize()
    return st


def run(st):
    op, eng, prec = st["op"], st["engine"], st["prec"]
    if op == "fock":
        return eng.fock_rhf(st["host_D"][0], st["H"], prec)
    if op == "uhf":
        return eng.fock_uhf(st["host_D"][0], st["host_D"][1], st["H"], prec)
    if op == "scf":
        # tight thresholds, as for derivatives, so that the result does not depend on which side
        # of a loose threshold the last iteration falls
        res = scf.rhf(st["basis"], engine=eng, guess="sad", e_tol=1e-10, rms_tol=1e-10, precision=prec)
        return {"energy": np.float64(res.energy), "density": res.D, "fock": res.F,
                "gradient": scf.rhf_gradient(st["basis"], res, eng, prec)}
    if op == "batch":
        eng.jk_device(st["D"], st["J"], st["K"], prec)
        return st["J"], st["K"]
    D = st["D"].data_ptr()
    if op == "jk":
        eng.jk_device(D, 1, D, st["J"].data_ptr(), st["K"].data_ptr(), prec)
        return st["J"], st["K"]
    with torch.cuda.stream(st["stream"]):
        if op == "grad":
            st["g"].zero_()
            eng.grad2e_device(D, 2.0, 1, D, 1.0, st["g"].data_ptr(), prec)
            return st["g"]
        st["h"].zero_()
        eng.hess2e_device(D, 2.0, 1, D, 1.0, st["h"].data_ptr())
        return st["h"]


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------
# a Hessian's recurrence runs two orders higher on the ten exponent weights against the
# gradient's one order on four: about this many times its operations
HESS_OVER_GRAD = 6.0


def _pair_work(bs):
    """Surviving (Schwarz bound >= 1e-12) contracted and primitive quartets per class, from the
    engine's own lists of this molecule."""
    with E.Engine(bs) as eng:
        return [eng.class_work(c) for c in range(E.NUM_CLASSES)]


def _flops(bs, kind):
    f = flopmodel.grad_class_flops if kind in ("grad", "hess") else flopmodel.class_flops
    tot = sum(f(c, w["quartets"], w["prim_quartets"], bs.pure) for c, w in enumerate(_pair_work(bs)))
    return tot * (HESS_OVER_GRAD if kind == "hess" else 1.0)


def work(case):
    """Operations: the frozen Head-Gordon-Pople count over the Schwarz-surviving quartets.
    Bytes: the matrices in and out."""
    op = case["op"]
    if op == "batch":
        # a sample of the mix, scaled: the molecules are drawn independently
        bases = _batch(case, 1)
        some = bases[:: max(1, len(bases) // 16)]
        scale = len(bases) / len(some)
        return {"bytes": 24.0 * sum(b.nbf ** 2 for b in bases), "flops": scale * sum(_flops(b, "jk") for b in some)}
    bs = _basis(case, 1)
    n, nc = bs.nbf, 3 * bs.natoms
    if op == "scf":
        # about 15 builds and one gradient; the matrices of the result
        return {"bytes": 8.0 * (2 * n * n + nc), "flops": 15.0 * _flops(bs, "jk") + _flops(bs, "grad")}
    nmat = {"fock": 3, "jk": 3, "uhf": 5, "grad": 1, "hess": 1}[op]
    out = {"grad": nc, "hess": nc * nc}.get(op, 0)
    return {"bytes": 8.0 * (nmat * n * n + out), "flops": _flops(bs, op)}


# ---------------------------------------------------------------------------
# the same quantities in plain torch, 64 bits
# ---------------------------------------------------------------------------
CART = {L: [(L - i, i - j, j) for i in range(L + 1) for j in range(i + 1)] for L in range(5)}
R3 = math.sqrt(3.0)
# real solid harmonics m = -L..L over the Cartesian components above (x^L normalised)
PURE = {0: [[1.0]], 1: [[0, 1, 0], [0, 0, 1], [1, 0, 0]],
        2: [[0, R3, 0, 0, 0, 0], [0, 0, 0, 0, R3, 0], [-0.5, 0, 0, -0.5, 0, 1], [0, 0, R3, 0, 0, 0],
            [R3 / 2, 0, 0, -R3 / 2, 0, 0]]}
CHUNK = 40_000_000   # Hermite integrals held at once
# primitive quartets below which the plain evaluation stays well under 20 s
EXACT_LIMIT = {"fock": 6e8, "jk": 6e8, "uhf": 6e8, "grad": 4e7, "hess": 3e5, "scf": 3e6}


def _hermites(n):
    return [t for s in range(n + 1) for t in itertools.product(range(s + 1), repeat=3) if sum(t) == s]


class _Boys(torch.autograd.Function):
    """F_0..F_M(T) stacked in front; dF_m/dT = -F_{m+1}."""

    @staticmethod
    def forward(ctx, T, M):
        ctx.save_for_backward(T)
        ctx.M = M
        a = M + 0.5
        Ts = T.clamp_min(1.0)
        big = torch.special.gammainc(torch.full_like(T, a), Ts) * math.gamma(a) / (2.0 * Ts ** a)
        term = torch.full_like(T, 1.0 / (2 * M + 1))
        small = term.clone()
        for i in range(1, 24):  # e^-T sum (2T)^i / (2M+1)(2M+3)..., T <= 1
            term = term * 2.0 * T.clamp_max(1.0) / (2 * M + 2 * i + 1)
            small = small + term
        e = torch.exp(-T)
        F = [None] * (M + 1)
        F[M] = torch.where(T < 1.0, e * small, big)
        for m in range(M, 0, -1):
            F[m - 1] = (2.0 * T * F[m] + e) / (2 * m - 1)
        return torch.stack(F)

    @staticmethod
    def backward(ctx, g):
        (T,) = ctx.saved_tensors
        return -(g * _Boys.apply(T, ctx.M + 1)[1:]).sum(0), None


def _hermite_coulomb(alpha, X, L):
    """R_tuv for t+u+v <= L, stacked last in the order of _hermites(L); X: [..., 3]."""
    F = _Boys.apply(alpha * (X * X).sum(-1), L)
    R = {((0, 0, 0), m): F[m] * (-2.0 * alpha) ** m for m in range(L + 1)}
    for s in range(1, L + 1):
        for t in _hermites(s):
            if sum(t) != s:
                continue
            i = max(range(3), key=lambda k: t[k])
            d = [tuple(v - k * (j == i) for j, v in enumerate(t)) for k in (1, 2)]
            for m in range(L + 1 - s):
                r = X[..., i] * R[d[0], m + 1]
                if t[i] > 1:
                    r = r + (t[i] - 1) * R[d[1], m + 1]
                R[t, m] = r
    return torch.stack([R[t, 0] for t in _hermites(L)], dim=-1)


class _Mol:
    """Primitive shell pairs of a basis by pair class, differentiable in the coordinates x."""

    def __init__(self, bs, device):
        self.bs, self.dev, self.n = bs, device, bs.nbf
        self.x = torch.from_numpy(np.array(bs.coords)).to(device)
        self.shells = []
        for s in bs.shells:
            a, c = s.exps, s.coefs
            m = s.L + 1.5
            norm = np.sum(np.outer(c, c) * np.outer(a, a) ** (0.5 * m) / np.add.outer(a, a) ** m)
            norm *= math.pi ** 1.5 * (1.0, 1.0, 3.0)[s.L] / 2.0 ** s.L
            self.shells.append((s.L, s.atom, a, c * a ** (0.5 * m) / math.sqrt(norm), s.ids if bs.pure else s.idx))
        self.nprim = sum(len(s[2]) for s in self.shells)
        self.classes = [self._pairs(la, lb) for la in range(3) for lb in range(la + 1)]
        self.classes = [c for c in self.classes if c["seg"].numel()]

    def _pairs(self, la, lb):
        rows, fab = [], []
        for i, si in enumerate(self.shells):
            for j, sj in enumerate(self.shells):
                if si[0] != la or sj[0] != lb or (la == lb and j < i):
                    continue
                for (a, ca), (b, cb) in itertools.product(zip(si[2], si[3]), zip(sj[2], sj[3])):
                    rows.append((len(fab), si[1], sj[1], a, b, ca * cb))
                fab.append((si[4], sj[4], 1.0 if i == j else 2.0))
        r = torch.tensor(rows, dtype=torch.float64).reshape(-1, 6).to(self.dev)
        f = torch.tensor(fab, dtype=torch.float64).reshape(-1, 3).to(self.dev)
        na, nb = [(2 * L + 1) if self.bs.pure else len(CART[L]) for L in (la, lb)]
        fa = f[:, 0].long()[:, None] + torch.arange(na, device=self.dev).repeat_interleave(nb)
        fb = f[:, 1].long()[:, None] + torch.arange(nb, device=self.dev).repeat(na)
        return {"la": la, "lb": lb, "L": la + lb, "seg": r[:, 0].long(), "A": r[:, 1].long(), "B": r[:, 2].long(),
                "a": r[:, 3], "b": r[:, 4], "c": r[:, 5], "fa": fa, "fb": fb, "twice": f[:, 2]}

    def expand(self, c, x, extra=0):
        """p, P and the 1-D Hermite tables E[dir][(i, j)] (lists over t) of a pair class."""
        a, b = c["a"], c["b"]
        p = a + b
        A, Bc = x[c["A"]], x[c["B"]]
        P = (a[:, None] * A + b[:, None] * Bc) / p[:, None]
        tabs = []
        for d in range(3):
            E0 = {(0, 0): [torch.exp(-a * b / p * (A[:, d] - Bc[:, d]) ** 2)]}
            for i, j in itertools.product(range(c["la"] + 1), range(c["lb"] + 1 + extra)):
                if (i, j) == (0, 0):
                    continue
                prev, Xp = (E0[i - 1, j], P[:, d] - A[:, d]) if j == 0 else (E0[i, j - 1], P[:, d] - Bc[:, d])
                get = lambda t, q=prev: q[t] if 0 <= t < len(q) else None  # noqa: E731
                row = []
                for t in range(i + j + 1):
                    v = 0.0
                    if get(t - 1) is not None:
                        v = v + get(t - 1) / (2 * p)
                    if get(t) is not None:
                        v = v + Xp * get(t)
                    if get(t + 1) is not None:
                        v = v + (t + 1) * get(t + 1)
                    row.append(v)
                E0[i, j] = row
            tabs.append(E0)
        return p, P, tabs

    def to_final(self, c, H):
        """Cartesian component pairs (dim 1) to the basis's own functions."""
        if not self.bs.pure:
            return H
        Ta, Tb = (torch.tensor(PURE[L], dtype=torch.float64, device=self.dev) for L in (c["la"], c["lb"]))
        return torch.einsum("fc,kct->kft", torch.kron(Ta, Tb), H)

    def hermite(self, c, x):
        p, P, tabs = self.expand(c, x)
        zero = torch.zeros_like(p)
        comps = []
        for u, v in itertools.product(CART[c["la"]], CART[c["lb"]]):
            E1 = [tabs[d][u[d], v[d]] for d in range(3)]
            comps.append(torch.stack([E1[0][t[0]] * E1[1][t[1]] * E1[2][t[2]]
                                      if all(t[d] < len(E1[d]) for d in range(3)) else zero
                                      for t in _hermites(c["L"])], -1))
        return p, P, self.to_final(c, torch.stack(comps, 1) * c["c"][:, None, None])

    def blocks(self, x):
        """Contracted blocks over unique class pairs, in chunks of bra shell pairs: yields
        (bra class, bra pairs lo..hi, ket class, block [pairs, ab, pairs, cd])."""
        herm = [self.hermite(c, x) for c in self.classes]
        for ib, cb in enumerate(self.classes):
            pb, Pb, Hb = herm[ib]
            first = torch.searchsorted(cb["seg"], torch.arange(len(cb["twice"]) + 1, device=self.dev)).tolist()
            for ik in range(ib + 1):
                ck = self.classes[ik]
                pk, Pk, Hk = herm[ik]
                tb, tk, tl = _hermites(cb["L"]), _hermites(ck["L"]), _hermites(cb["L"] + ck["L"])
                at = {t: i for i, t in enumerate(tl)}
                idx = torch.tensor([[at[tuple(np.add(s, t))] for t in tk] for s in tb], device=self.dev)
                sign = torch.tensor([(-1.0) ** sum(t) for t in tk], dtype=torch.float64, device=self.dev)
                Hks = Hk * sign
                most = max(1, int(CHUNK / (len(pk) * (len(tb) * len(tk) + 3 * len(tl)))))
                lo = 0
                while lo < len(cb["twice"]):
                    hi = lo + 1
                    while hi < len(cb["twice"]) and first[hi + 1] - first[lo] <= most:
                        hi += 1
                    s = slice(first[lo], first[hi])
                    q = pb[s, None] * pk[None, :]
                    sm = pb[s, None] + pk[None, :]
                    R = _hermite_coulomb(q / sm, Pb[s, None, :] - Pk[None, :, :], cb["L"] + ck["L"])
                    R = R * (2.0 * math.pi ** 2.5 / (q * torch.sqrt(sm)))[..., None]
                    Y = torch.einsum("bktu,kdu->bktd", R[:, :, idx], Hks)
                    Y = torch.einsum("bktd,bct->bckd", Y, Hb[s])
                    Y = torch.zeros(Y.shape[0], Y.shape[1], len(ck["twice"]), Y.shape[3], dtype=Y.dtype,
                                    device=self.dev).index_add(2, ck["seg"], Y)
                    Y = torch.zeros(hi - lo, *Y.shape[1:], dtype=Y.dtype, device=self.dev).index_add(
                        0, cb["seg"][s] - lo, Y)
                    yield cb, lo, hi, ck, Y
                    lo = hi

    def jk(self, DJ, DKs):
        n = self.n
        G = torch.zeros(n * (n + 1) // 2, n * (n + 1) // 2, dtype=torch.float64, device=self.dev)

        def packed(i, j):
            hi, lo = torch.maximum(i, j), torch.minimum(i, j)
            return hi * (hi + 1) // 2 + lo

        for cb, lo, hi, ck, Y in self.blocks(self.x):
            r = packed(cb["fa"][lo:hi], cb["fb"][lo:hi]).reshape(-1)
            s = packed(ck["fa"], ck["fb"]).reshape(-1)
            Y = Y.reshape(len(r), len(s))
            G[r[:, None], s[None, :]] = Y
            G[s[:, None], r[None, :]] = Y.T
        i = torch.arange(n, device=self.dev)
        full = packed(i[:, None], i[None, :])
        fold = torch.zeros(len(G), dtype=torch.float64, device=self.dev).index_add(0, full.reshape(-1), DJ.reshape(-1))
        J = (G @ fold)[full]
        K = [torch.empty_like(J) for _ in DKs]
        for a in range(n):
            rows = G[full[a]][:, full]  # (a b | c d)
            for m, D in enumerate(DKs):
                K[m][a] = torch.einsum("bcd,bd->c", rows, D)
        return J, K

    def energy_terms(self, D, x):
        """E2 = sum D (2J - K) in pieces, differentiable in x."""
        for cb, lo, hi, ck, Y in self.blocks(x):
            a, b = (cb[k][lo:hi][:, :, None, None] for k in ("fa", "fb"))
            c, d = ck["fa"][None, None], ck["fb"][None, None]
            W = 2.0 * D[a, b] * D[c, d] - 0.5 * (D[a, c] * D[b, d] + D[a, d] * D[b, c])
            f = cb["twice"][lo:hi, None, None, None] * ck["twice"][None, None, :, None]
            yield (W * f * Y).sum() * (1.0 if cb is ck else 2.0)

    def gradient(self, D):
        x = self.x.clone().requires_grad_(True)
        for e in self.energy_terms(D, x):
            e.backward(retain_graph=True)
        return x.grad

    def hessian(self, D):
        x = self.x.clone().requires_grad_(True)
        (g,) = torch.autograd.grad(sum(self.energy_terms(D, x)), x, create_graph=True)
        rows = [torch.autograd.grad(v, x, retain_graph=True)[0].reshape(-1) for v in g.reshape(-1)]
        return torch.stack(rows)

    def one_electron(self, x):
        """S, T, V at coordinates x."""
        n = self.n
        out = [torch.zeros(n, n, dtype=torch.float64, device=self.dev) for _ in range(3)]
        Z = torch.from_numpy(np.asarray(self.bs.Z, dtype=np.float64)).to(self.dev)
        for c in self.classes:
            p, P, tabs = self.expand(c, x, extra=2)
            root = torch.sqrt(math.pi / p)
            s1 = [{k: v[0] * root for k, v in tabs[d].items()} for d in range(3)]
            b = c["b"]

            def kin(d, i, j):
                v = b * (2 * j + 1) * s1[d][i, j] - 2.0 * b * b * s1[d][i, j + 2]
                return v - 0.5 * j * (j - 1) * s1[d][i, j - 2] if j > 1 else v

            S, T = [], []
            for u, v in itertools.product(CART[c["la"]], CART[c["lb"]]):
                s = [s1[d][u[d], v[d]] for d in range(3)]
                k = [kin(d, u[d], v[d]) for d in range(3)]
                S.append(s[0] * s[1] * s[2])
                T.append(k[0] * s[1] * s[2] + s[0] * k[1] * s[2] + s[0] * s[1] * k[2])
            _, _, H = self.hermite(c, x)
            R = _hermite_coulomb(p[:, None].expand(-1, len(Z)), P[:, None, :] - x[None], c["L"])
            R = (R * Z[None, :, None]).sum(1) * (-2.0 * math.pi / p)[:, None]
            cc = c["c"][:, None]
            mats = [self.to_final(c, (torch.stack(m, 1) * cc)[..., None])[..., 0] for m in (S, T)]
            mats.append(torch.einsum("kct,kt->kc", H, R))
            for k, m in enumerate(mats):
                m = torch.zeros(len(c["twice"]), m.shape[1], dtype=m.dtype, device=self.dev).index_add(0, c["seg"], m)
                out[k] = out[k].index_put((c["fa"], c["fb"]), m)
                out[k] = out[k].index_put((c["fb"], c["fa"]), m)
        return out

    def scf(self):
        """Closed-shell energy, density, Fock matrix and gradient, converged by DIIS."""
        x, bs = self.x, self.bs
        nocc = int(np.sum(bs.Z)) // 2
        S, T, V = self.one_electron(x)
        H = T + V
        w, U = torch.linalg.eigh(S)
        X = (U / torch.sqrt(w)) @ U.T
        F, Fs, Es = H, [], []
        for _ in range(200):
            C = X @ torch.linalg.eigh(X.T @ F @ X)[1][:, :nocc]
            D = C @ C.T
            J, K = self.jk(D, [D])
            F0 = H + 2.0 * J - K[0]
            err = X.T @ (F0 @ D @ S - S @ D @ F0) @ X
            if err.abs().max() < 1e-12:
                break
            Fs, Es = (Fs + [F0])[-8:], (Es + [err])[-8:]
            m = len(Fs)
            Bm = -torch.ones(m + 1, m + 1, dtype=torch.float64, device=self.dev)
            Bm[m, m] = 0.0
            for i, j in itertools.product(range(m), range(m)):
                Bm[i, j] = (Es[i] * Es[j]).sum()
            scale = Bm[:m, :m].abs().max()
            Bm[:m, :m] /= scale
            rhs = torch.zeros(m + 1, dtype=torch.float64, device=self.dev)
            rhs[m] = -1.0
            cf = torch.linalg.lstsq(Bm.cpu(), rhs.cpu()[:, None], driver="gelsd").solution[:m, 0].tolist()
            F = sum(cf[k] * Fs[k] for k in range(m))
        xg = x.clone().requires_grad_(True)
        Sg, Tg, Vg = self.one_electron(xg)
        Z = torch.from_numpy(np.asarray(bs.Z, dtype=np.float64)).to(self.dev)
        i, j = np.triu_indices(len(Z), 1)
        enuc = (Z[i] * Z[j] / (xg[i] - xg[j]).norm(dim=1)).sum()
        e1 = 2.0 * (D * (Tg + Vg)).sum() - 2.0 * (D @ F0 @ D * Sg).sum() + enuc
        (g1,) = torch.autograd.grad(e1, xg)
        return {"energy": np.float64((D * (H + F0)).sum().item() + enuc.item()), "density": D.cpu(), "fock": F0.cpu(),
                "gradient": (g1 + self.gradient(D)).cpu()}


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if op == "scf":
        bs, H, Ds = _basis(case, seed), None, ()
    else:
        bs, H, Ds = _inputs(case, seed)
    mol = _Mol(bs, dev)
    if (mol.nprim * (mol.nprim + 1) / 2) ** 2 / 2 > EXACT_LIMIT[op]:
        return None
    Ds = [torch.from_numpy(D).to(dev) for D in Ds]
    if op == "scf":
        return mol.scf()
    if op == "grad":
        return mol.gradient(Ds[0])
    if op == "hess":
        return mol.hessian(Ds[0])
    J, K = mol.jk(sum(Ds), Ds)
    if op == "jk":
        return J, K[0]
    Hd = torch.from_numpy(H).to(dev)
    if op == "fock":
        return (Hd + 2.0 * J - K[0]).cpu()
    return tuple((Hd + J - k).cpu() for k in K)
