"""Workloads of the Fock build, the nuclear gradient and their set-up.

Each case is one call that a quantum-chemistry program makes over and over:
a Fock or J/K build per SCF iteration, a gradient per geometry step, response
densities of a CPHF solve, the context and the one-electron matrices of a new
geometry, a batch of geometries, and a whole small SCF.  Molecules are the
package's seeded synthetic ones (``iqcp_b200.molecules``) or its reference
molecules, displaced by the seed; densities have the size and the decay with
distance of converged ones.

``exact`` evaluates small cases in plain torch (FP64) by another method than
the library's: McMurchie-Davidson Hermite expansions of every primitive pair,
no screening, and automatic differentiation for gradients.
"""
import functools
import math

import numpy as np
import torch

from iqcp_b200 import FP64, MIXED, BasisSet, BatchFockEngine, FockEngine, molecules
from iqcp_b200.batch_scf import BatchRHF

BASES = ("sto-3g", "3-21g", "6-31g", "6-31g*", "cc-pvdz", "6-31+g*")
HEAVY = (6, 7, 8, 9)
JITTER = 0.02  # bohr, per coordinate: the step of a geometry scan


def listed():
    return [
        # one Fock build of the smallest molecules people run: launches and host latency
        dict(name="fock_h2o", kind="fock", atoms=3, geom=0, basis="6-31g*"),
        # J and K through the host-array call, as a program without a GPU array library makes it
        dict(name="jk_host_12", kind="jk_host", atoms=12, geom=0, basis="6-31g"),
        # the SCF iteration of an ordinary drug-like molecule, the size of the package's benchmark
        dict(name="fock_40", kind="fock", atoms=40, geom=0, basis="6-31g*"),
        # the same build in the mixed-precision form at the benchmark's cutoff
        dict(name="fock_mixed_40", kind="fock", atoms=40, geom=0, basis="6-31g*", cutoff=1e-3),
        # diffuse functions, where screening keeps most quartets: the largest Fock build
        dict(name="jk_diffuse_44", kind="jk", atoms=44, geom=3, basis="6-31+g*"),
        # two-electron gradient of a small molecule (geometry steps, finite-difference Hessians)
        dict(name="grad_12", kind="grad", atoms=12, geom=1, basis="6-31g*"),
        # the same at the size of the package's benchmark
        dict(name="grad_40", kind="grad", atoms=40, geom=0, basis="6-31g*"),
        # the whole RHF gradient through the host call, in the other common polarised basis
        dict(name="rhf_grad_dz_30", kind="rhf_grad", atoms=30, geom=0, basis="cc-pvdz"),
        # one CPHF step: several response densities at once
        dict(name="cphf_16", kind="multi", atoms=16, geom=2, basis="6-31g", nset=9),
        # a new geometry of an optimisation or a scan: context, Schwarz bounds, S, T and V
        dict(name="new_geometry_30", kind="setup", atoms=30, geom=0, basis="6-31g*"),
        # many small geometries in one context, tuned once as a long scan does: Fock builds and gradients
        dict(name="batch_16", kind="batch", n_mol=16, atoms=20, geom=1, basis="6-31g*"),
        # a whole batched SCF with its gradients, from the SAD guess
        dict(name="scf_batch_6", kind="scf", n_mol=6, basis="6-31g*"),
    ]


def draw(rng):
    kind = rng.choice(("fock", "fock", "jk", "jk_host", "grad", "grad", "rhf_grad", "multi", "setup", "batch", "mixed"))
    hi = {"rhf_grad": 30, "multi": 24, "batch": 20}.get(kind, 40)
    atoms = int(round(math.exp(rng.uniform(math.log(4), math.log(hi)))))
    c = dict(kind=kind, atoms=atoms, geom=rng.randrange(6), basis=rng.choice(BASES[:5] if atoms > 30 else BASES))
    if kind == "multi":
        c["nset"] = rng.randrange(2, 13)
    if kind == "batch":
        c["n_mol"] = rng.randrange(2, 14)
    if kind == "mixed":
        c["kind"], c["cutoff"] = "fock", rng.choice((1e-3, 1e-5))
    return c


# ---------------------------------------------------------------------------
# Inputs
@functools.lru_cache(maxsize=64)
def _molecule(atoms, geom):
    """Seeded synthetic molecule (the package's workload seeds and element mixes)."""
    if atoms == 3:
        return tuple(molecules.REFERENCE_MOLECULES["H2O"])
    n_heavy = max(1, int(round((0.5 + 0.02 * (geom % 6)) * atoms)))
    heavy = HEAVY[:3] if geom % 2 == 0 else HEAVY
    for k in range(50):
        try:
            return tuple(molecules.generate(atoms, heavy, n_heavy, 1000 * k + geom, max_tries=600))
        except RuntimeError:
            continue
    raise RuntimeError("no placeable molecule of %d atoms" % atoms)


def _molecules(case):
    kind, n = case["kind"], case.get("n_mol", 1)
    if kind == "scf":
        names = ("H2O", "NH3", "CH4", "HF", "C6H6", "H2")
        return [tuple(molecules.REFERENCE_MOLECULES[names[m % len(names)]]) for m in range(n)]
    if kind == "batch":
        return [_molecule(max(4, case["atoms"] - 2 * (m % 6)), case["geom"] + m) for m in range(n)]
    return [_molecule(case["atoms"], case["geom"])]


def _geometries(case, seed):
    """The molecules of a case, displaced by the seed, and the generator of its other inputs."""
    rng = np.random.default_rng(seed)
    return [[(z, tuple(np.asarray(x) + rng.uniform(-JITTER, JITTER, 3))) for z, x in mol] for mol in _molecules(case)], rng


def _decaying(basis, rng, diag):
    """Symmetric matrix whose elements fall off with the distance of their centres."""
    at = np.repeat(basis.center, (basis.l + 1) * (basis.l + 2) // 2, axis=0)
    r = np.linalg.norm(at[:, None] - at[None], axis=2)
    a = rng.normal(size=r.shape) * 0.15 * np.exp(-r / 3.0)
    return 0.5 * (a + a.T) + diag * np.diag(rng.uniform(0.1, 1.0, len(r)))


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    geoms, rng = _geometries(case, seed)
    bases = [BasisSet.build(g, case["basis"]) for g in geoms]
    st = dict(case=case, kind=case["kind"], bases=bases, basis=bases[0])
    kind, b = case["kind"], bases[0]
    if kind == "setup":
        return st
    if kind == "scf":
        st["rhf"] = BatchRHF(bases)
        return st
    if kind == "batch":
        eng = BatchFockEngine(bases)
        D = eng.pack([_decaying(x, rng, 1.0) for x in bases])
        st.update(D=_gpu(D), H=_gpu(eng.pack([_decaying(x, rng, -8.0) for x in bases])),
                  F=torch.empty(eng.packed_size, dtype=torch.float64, device="cuda"),
                  g=torch.zeros(eng.n_atoms, 3, dtype=torch.float64, device="cuda"))
        eng.autotune(st["D"].data_ptr(), 1)
    else:
        mixed = "cutoff" in case
        eng = FockEngine(b, precision=MIXED if mixed else FP64, mixed_cutoff=case.get("cutoff", 1e-9))
        n = b.n_basis
        D = _decaying(b, rng, 1.0)
        if kind in ("jk_host", "rhf_grad"):
            st.update(D=D, W=_decaying(b, rng, -1.0))
        elif kind == "multi":
            D = np.stack([_decaying(b, rng, 0.0) for _ in range(case["nset"])])
            st.update(D=_gpu(D), J=_gpu(np.empty_like(D)), K=_gpu(np.empty_like(D)))
        elif kind == "grad":
            st.update(D=_gpu(D), g=torch.zeros(b.n_atoms, 3, dtype=torch.float64, device="cuda"))
        else:
            st.update(D=_gpu(D), H=_gpu(_decaying(b, rng, -8.0)),
                      F=torch.empty(n, n, dtype=torch.float64, device="cuda"),
                      J=torch.empty(n, n, dtype=torch.float64, device="cuda"),
                      K=torch.empty(n, n, dtype=torch.float64, device="cuda"))
    if kind not in ("jk_host", "rhf_grad"):
        eng.set_stream(torch.cuda.current_stream().cuda_stream)
    st["eng"] = eng
    return st


def run(st):
    kind, eng = st["kind"], st.get("eng")
    if kind == "fock":
        eng.fock_device(st["H"].data_ptr(), st["D"].data_ptr(), 1.0, st["F"].data_ptr())
        return st["F"]
    if kind == "jk":
        eng.jk_device(st["D"].data_ptr(), st["J"].data_ptr(), st["K"].data_ptr())
        return st["J"], st["K"]
    if kind == "jk_host":
        return eng.build_jk(st["D"])
    if kind == "grad":
        st["g"].zero_()
        eng.eri_gradient_device(st["D"].data_ptr(), 1.0, st["g"].data_ptr())
        return st["g"]
    if kind == "rhf_grad":
        return eng.rhf_gradient(st["D"], st["W"])
    if kind == "multi":
        eng.jk_multi_device(len(st["D"]), st["D"].data_ptr(), st["J"].data_ptr(), st["K"].data_ptr())
        return st["J"], st["K"]
    if kind == "setup":
        with FockEngine(st["basis"]) as eng:
            return (eng.schwarz(),) + tuple(eng.one_electron())
    if kind == "batch":
        eng.fock_device(st["H"].data_ptr(), st["D"].data_ptr(), 1.0, st["F"].data_ptr())
        st["g"].zero_()
        eng.eri_gradient_device(st["D"].data_ptr(), 1.0, st["g"].data_ptr())
        return st["F"], st["g"]
    rhf = st["rhf"]  # scf: tight thresholds, so that the solution does not depend on the last iteration
    r = rhf.run(e_tol=1e-10, d_tol=1e-9, err_tol=1e-7, D0=rhf.sad_guess())
    return [r.energies, np.concatenate([d.ravel() for d in rhf.densities()]), np.concatenate(rhf.gradients())]


# ---------------------------------------------------------------------------
# What a pass cannot do without: every input read and every output written
# once, and for each primitive quartet within reach the operations of one
# Rys/Boys evaluation of its integrals and their products with the densities.
@functools.lru_cache(maxsize=64)
def _counts(mol, basis):
    """(nbf, primitive pairs with exp(-mu R^2) >= 1e-15, the same times their components) of a molecule."""
    b = BasisSet.build(list(mol), basis)
    first = np.concatenate([[0], np.cumsum(b.nprim)])
    exps = [b.exps[first[s]:first[s + 1]] for s in range(b.n_shells)]
    ncart = (b.l + 1) * (b.l + 2) // 2
    pairs = comps = 0.0
    for i in range(b.n_shells):
        for j in range(i + 1):
            mu = np.multiply.outer(exps[i], exps[j]) / np.add.outer(exps[i], exps[j])
            n = int((mu * float(((b.center[i] - b.center[j]) ** 2).sum()) < 34.5).sum())
            pairs += n
            comps += n * int(ncart[i] * ncart[j])
    return b.n_basis, pairs, comps


def work(case):
    kind = case["kind"]
    n2 = flops = nat = 0.0
    for mol in _molecules(case):
        nbf, pairs, comps = _counts(mol, case["basis"])
        n2 += nbf * nbf
        nat += len(mol)
        quartets, integrals = pairs * pairs / 2, comps * comps / 2
        build, grad = 40 * quartets + 2 * integrals, 80 * quartets + 18 * integrals
        flops += {"setup": 60 * comps * (1 + len(mol)), "grad": grad, "rhf_grad": grad, "batch": build + grad,
                  "scf": 12 * build + grad}.get(kind, build)
    mats = {"fock": 3, "jk": 3, "jk_host": 3, "multi": 3 * case.get("nset", 1), "setup": 3, "batch": 3, "rhf_grad": 2}.get(kind, 1)
    return {"bytes": 8 * (mats * n2 + 3 * nat), "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit values by McMurchie-Davidson in plain torch
def _cart(l):
    return [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]


def _dfact(n):
    return float(np.prod(np.arange(n, 0, -2))) if n > 0 else 1.0


class _Boys(torch.autograd.Function):
    """F_0..F_m(T) along a new last axis; dF_m/dT = -F_{m+1}."""

    @staticmethod
    def forward(ctx, T, m):
        F = _boys(T, m + 1)
        ctx.save_for_backward(F)
        return F[..., : m + 1].clone()

    @staticmethod
    def backward(ctx, g):
        (F,) = ctx.saved_tensors
        return -(g * F[..., 1:]).sum(-1), None


def _boys(T, m):
    out = torch.empty(T.shape + (m + 1,), dtype=T.dtype, device=T.device)
    small = T < 38.0
    t = torch.where(small, T, torch.zeros_like(T))
    e = torch.exp(-t)
    term = torch.full_like(t, 1.0 / (2 * m + 1))
    s = term.clone()
    for k in range(1, 170):
        term = term * (2.0 * t / (2 * m + 2 * k + 1))
        s = s + term
    f = s * e
    big = torch.where(small, torch.full_like(T, 50.0), T)
    eb = torch.exp(-big)
    up = [0.5 * torch.sqrt(math.pi / big) * torch.erf(torch.sqrt(big))]
    for k in range(m):
        up.append(((2 * k + 1) * up[-1] - eb) / (2.0 * big))
    for k in range(m, -1, -1):
        out[..., k] = torch.where(small, f, up[k])
        if k:
            f = (2.0 * t * f + e) / (2 * k - 1)
    return out


def _hermite_list(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _r_tensor(p, d, L):
    """R_tuv (t + u + v <= L) for exponent p and separation d, last axis in _hermite_list order."""
    F = _Boys.apply(p * (d * d).sum(-1), L)
    cur = {(n, 0, 0, 0): F[..., n] * (-2.0 * p) ** n for n in range(L + 1)}

    def get(n, t, u, v):
        if min(t, u, v) < 0:
            return 0.0
        k = (n, t, u, v)
        if k not in cur:
            ax = 0 if t else (1 if u else 2)
            low = [t, u, v]
            low[ax] -= 1
            c = low[ax]
            val = d[..., ax] * get(n + 1, *low)
            if c:
                low2 = list(low)
                low2[ax] -= 1
                val = val + c * get(n + 1, *low2)
            cur[k] = val
        return cur[k]

    return torch.stack([get(0, *h) for h in _hermite_list(L)], -1)


def _e_axis(la, lb, a, b, X):
    """E[i][j] = list over t of the 1D Hermite coefficients, without the exponential."""
    p = a + b
    xa, xb, o = -b / p * X, a / p * X, 0.5 / p
    E = {(0, 0): [torch.ones_like(X)]}

    def step(prev, x, n):
        out = []
        for t in range(n + 1):
            v = x * prev[t] if t < n else 0.0
            if t > 0:
                v = v + o * prev[t - 1]
            if t + 1 < n:
                v = v + (t + 1) * prev[t + 1]
            out.append(v)
        return out

    for i in range(la + 1):
        for j in range(lb + 1):
            if i + j:
                E[i, j] = step(E[i - 1, j], xa, i + j) if i else step(E[i, j - 1], xb, i + j)
    return E


class _Mol:
    """Shell pairs by class with Hermite coefficients; differentiable in the atom positions xyz."""

    def __init__(self, basis, device):
        self.b, self.dev = basis, device
        self.xyz = torch.tensor(basis.xyz, dtype=torch.float64, device=device)
        self.first = np.concatenate([[0], np.cumsum(basis.nprim)])

    def _norm(self, l, a):
        return (2.0 * a / math.pi) ** 0.75 * (4.0 * a) ** (l / 2.0)

    def pairs(self, la, lb, ordered=False, extra=0):
        """Primitive pairs of the shell pairs of class (la, lb): contracted-pair index, E, P, p, shells."""
        b = self.b
        A = [s for s in range(b.n_shells) if b.l[s] == la]
        B = [s for s in range(b.n_shells) if b.l[s] == lb]
        sp = [(i, j) for i in A for j in B if ordered or la != lb or j <= i]
        if not sp:
            return None
        idx, pa, pb = [], [], []
        for k, (i, j) in enumerate(sp):
            for x in range(self.first[i], self.first[i + 1]):
                for y in range(self.first[j], self.first[j + 1]):
                    idx.append(k)
                    pa.append(x)
                    pb.append(y)
        idx = np.array(idx)
        sh = np.array(sp)
        e, c = b.exps, b.coefs
        t = lambda v: torch.tensor(v, dtype=torch.float64, device=self.dev)  # noqa: E731
        a_, b_ = t(e[pa]), t(e[pb])
        w = t(c[pa] * c[pb] * self._norm(la, e[pa]) * self._norm(lb, e[pb]))
        cA = self.xyz[b.atom_of_shell[sh[idx, 0]]]
        cB = self.xyz[b.atom_of_shell[sh[idx, 1]]]
        p = a_ + b_
        P = (a_[:, None] * cA + b_[:, None] * cB) / p[:, None]
        w = w * torch.exp(-a_ * b_ / p * ((cA - cB) ** 2).sum(-1))
        ax = [_e_axis(la, lb + extra, a_, b_, cA[:, d] - cB[:, d]) for d in range(3)]
        H = _hermite_list(la + lb)
        rows = []
        for i in _cart(la):
            for j in _cart(lb):
                n = 1.0 / math.sqrt(np.prod([_dfact(2 * q - 1) for q in i + j]))
                rows.append(torch.stack([w * n * ax[0][i[0], j[0]][h[0]] * ax[1][i[1], j[1]][h[1]] * ax[2][i[2], j[2]][h[2]]
                                         if all(h[d] <= i[d] + j[d] for d in range(3)) else torch.zeros_like(w) for h in H], -1))
        E = torch.stack(rows, 1)  # [prim pair, component, hermite]
        return dict(idx=torch.tensor(idx, device=self.dev), n=len(sp), E=E, P=P, p=p, sh=sh, la=la, lb=lb, ax=ax, w=w, a=a_, b=b_)

    def func(self, cl):
        """Basis-function indices [pair, component] of both members."""
        off = self.b.offsets[cl["sh"]]
        na, nb = (cl["la"] + 1) * (cl["la"] + 2) // 2, (cl["lb"] + 1) * (cl["lb"] + 2) // 2
        i = np.repeat(off[:, 0][:, None] + np.arange(na), nb, axis=1)
        j = np.tile(off[:, 1][:, None] + np.arange(nb), (1, na))
        return torch.tensor(i, device=self.dev), torch.tensor(j, device=self.dev)

    def blocks(self, budget=3e7):
        """(class X, class Y, contracted-pair slice of X, integrals [pairs of the slice, comps, pairs of Y, comps])."""
        names = [(x, y) for x in range(3) for y in range(x + 1)]
        for X in names:
            for Y in names:
                first = self.pairs(*X)
                ky = self.pairs(*Y)
                if first is None or ky is None:
                    continue
                L = sum(X) + sum(Y)
                hx, hy = _hermite_list(sum(X)), _hermite_list(sum(Y))
                pos = {h: k for k, h in enumerate(_hermite_list(L))}
                at = torch.tensor([[pos[tuple(np.add(g, h))] for h in hy] for g in hx], device=self.dev)
                sign = torch.tensor([(-1.0) ** sum(h) for h in hy], dtype=torch.float64, device=self.dev)
                counts = torch.bincount(first["idx"], minlength=first["n"]).cumsum(0).cpu().tolist()
                per = len(ky["p"]) * (len(hx) * len(hy) + len(pos) + 4 * L + 8)
                step = max(1, int(budget / per / max(1, counts[-1] / first["n"])))
                for lo in range(0, first["n"], step):
                    hi = min(lo + step, first["n"])
                    kx = self.pairs(*X) if self.xyz.requires_grad else first
                    kk = self.pairs(*Y) if self.xyz.requires_grad else ky
                    s = slice(counts[lo - 1] if lo else 0, counts[hi - 1])
                    p, q = kx["p"][s, None], kk["p"][None]
                    al = p * q / (p + q)
                    R = _r_tensor(al, kx["P"][s, None] - kk["P"][None], L)
                    R = R * (2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q)))[..., None]
                    T = torch.einsum("xygh,ych->xgyc", R[..., at.reshape(-1)].reshape(R.shape[:2] + at.shape), kk["E"] * sign)
                    T = torch.zeros(T.shape[:2] + (ky["n"], T.shape[3]), dtype=T.dtype, device=T.device).index_add(2, kk["idx"], T)
                    V = torch.einsum("xag,xgyc->xayc", kx["E"][s], T)
                    V = torch.zeros((hi - lo,) + V.shape[1:], dtype=V.dtype, device=V.device).index_add(0, kx["idx"][s] - lo, V)
                    yield kx, kk, slice(lo, hi), V

    def jk(self, Ds):
        n = self.b.n_basis
        J, K = torch.zeros_like(Ds), torch.zeros_like(Ds)
        for kx, ky, s, V in self.blocks():
            (i, j), (k, l) = self.func(kx), self.func(ky)
            i, j = i[s], j[s]
            # weight of a pair (both orders of its two functions are in the full sum)
            wy = torch.where(torch.tensor(ky["sh"][:, 0] != ky["sh"][:, 1], device=self.dev), 1.0, 0.5)
            wx = torch.where(torch.tensor(kx["sh"][s, 0] != kx["sh"][s, 1], device=self.dev), 1.0, 0.5)
            V = V * wy[None, None, :, None] * wx[:, None, None, None]
            for m in range(len(Ds)):
                D = Ds[m]
                v = torch.einsum("xayc,yc->xa", V, D[k, l] + D[l, k])
                J[m].view(-1).index_add_(0, torch.cat([(i * n + j).reshape(-1), (j * n + i).reshape(-1)]), v.reshape(-1).repeat(2))
                I, Jx, Kx, Lx = (torch.broadcast_to(t, V.shape) for t in (i[:, :, None, None], j[:, :, None, None], k[None, None], l[None, None]))
                for a, b2 in ((I, Jx), (Jx, I)):
                    for c, d in ((Kx, Lx), (Lx, Kx)):
                        K[m].view(-1).index_add_(0, (a * n + c).reshape(-1), (V * D[b2, d]).reshape(-1))
        return J, K

    def eri_gradient(self, D, hf=1.0):
        self.xyz.requires_grad_(True)
        g = torch.zeros_like(self.xyz)
        for kx, ky, s, V in self.blocks(6e6):
            (i, j), (k, l) = self.func(kx), self.func(ky)
            i, j = i[s][:, :, None, None], j[s][:, :, None, None]
            k, l = k[None, None], l[None, None]
            wy = torch.where(torch.tensor(ky["sh"][:, 0] != ky["sh"][:, 1], device=self.dev), 2.0, 1.0)
            wx = torch.where(torch.tensor(kx["sh"][s, 0] != kx["sh"][s, 1], device=self.dev), 2.0, 1.0)
            W = 0.5 * D[i, j] * D[k, l] - 0.125 * hf * (D[i, k] * D[j, l] + D[i, l] * D[j, k])
            W = W * wy[None, None, :, None] * wx[:, None, None, None]
            g += torch.autograd.grad((W * V).sum(), self.xyz)[0]
        self.xyz = self.xyz.detach()
        return g

    def one_electron(self, charges=True):
        """S, T, V (full matrices), differentiable."""
        n, dev = self.b.n_basis, self.dev
        S, T, V = (torch.zeros(n * n, dtype=torch.float64, device=dev) for _ in range(3))
        z = torch.tensor(self.b.z, dtype=torch.float64, device=dev)
        for la in range(3):
            for lb in range(3):
                cl = self.pairs(la, lb, ordered=True, extra=2)
                if cl is None:
                    continue
                L, (i, j) = la + lb, self.func(cl)
                r = torch.zeros(len(cl["p"]), len(_hermite_list(L)), dtype=torch.float64, device=dev)
                for c in range(len(z)):
                    r = r - z[c] * _r_tensor(cl["p"], cl["P"] - self.xyz[c], L)
                v = torch.einsum("xah,xh->xa", cl["E"], r) * (2.0 * math.pi / cl["p"])[:, None]
                sq, be = torch.sqrt(math.pi / cl["p"]), cl["b"]
                srow, trow = [], []
                for x in _cart(la):
                    for y in _cart(lb):
                        nn = cl["w"] / math.sqrt(np.prod([_dfact(2 * q - 1) for q in x + y]))
                        s1 = [sq * cl["ax"][d][x[d], y[d]][0] for d in range(3)]
                        t1 = []
                        for d in range(3):
                            q = y[d]
                            e = -2.0 * be * (2 * q + 1) * cl["ax"][d][x[d], q][0] + 4.0 * be * be * cl["ax"][d][x[d], q + 2][0]
                            if q > 1:
                                e = e + q * (q - 1) * cl["ax"][d][x[d], q - 2][0]
                            t1.append(-0.5 * sq * e)
                        srow.append(nn * s1[0] * s1[1] * s1[2])
                        trow.append(nn * (t1[0] * s1[1] * s1[2] + s1[0] * t1[1] * s1[2] + s1[0] * s1[1] * t1[2]))
                out = []
                for m in (torch.stack(srow, 1), torch.stack(trow, 1), v):
                    m = torch.zeros((cl["n"], m.shape[1]), dtype=m.dtype, device=dev).index_add(0, cl["idx"], m)
                    out.append(m.reshape(-1))
                f = (i * n + j).reshape(-1)
                S, T, V = S.index_add(0, f, out[0]), T.index_add(0, f, out[1]), V.index_add(0, f, out[2])
        return S.view(n, n), T.view(n, n), V.view(n, n)

    def one_electron_gradient(self, D, W):
        self.xyz.requires_grad_(True)
        S, T, V = self.one_electron()
        z = torch.tensor(self.b.z, dtype=torch.float64, device=self.dev)
        iu = torch.triu_indices(len(z), len(z), 1, device=self.dev)
        e = (z[iu[0]] * z[iu[1]] / (self.xyz[iu[0]] - self.xyz[iu[1]]).norm(dim=1)).sum()
        e = e + (D * (T + V)).sum() - (W * S).sum()
        g = torch.autograd.grad(e, self.xyz)[0]
        self.xyz = self.xyz.detach()
        return g

    def schwarz(self):
        n = self.b.n_shells
        Q = torch.zeros(n, n, dtype=torch.float64, device=self.dev)
        for la in range(3):
            for lb in range(la + 1):
                cl = self.pairs(la, lb)
                if cl is None:
                    continue
                L, hx = la + lb, _hermite_list(la + lb)
                pos = {h: k for k, h in enumerate(_hermite_list(2 * L))}
                at = torch.tensor([[pos[tuple(np.add(g, h))] for h in hx] for g in hx], device=self.dev)
                sign = torch.tensor([(-1.0) ** sum(h) for h in hx], dtype=torch.float64, device=self.dev)
                npp = torch.bincount(cl["idx"], minlength=cl["n"])
                first = torch.cumsum(npp, 0) - npp
                out = torch.zeros(cl["n"], cl["E"].shape[1], dtype=torch.float64, device=self.dev)
                for x in range(int(npp.max())):
                    for y in range(int(npp.max())):
                        k = torch.nonzero((npp > x) & (npp > y)).reshape(-1)
                        u, v = first[k] + x, first[k] + y
                        p, q = cl["p"][u], cl["p"][v]
                        R = _r_tensor(p * q / (p + q), cl["P"][u] - cl["P"][v], 2 * L)[:, at.reshape(-1)].view((-1,) + at.shape)
                        R = R * (2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q)))[:, None, None]
                        out.index_add_(0, k, torch.einsum("xag,xgh,xah->xa", cl["E"][u], R, cl["E"][v] * sign))
                q = out.abs().amax(1).sqrt()
                i, j = torch.tensor(cl["sh"], device=self.dev).T
                Q[i, j] = q
                Q[j, i] = q
        return Q


def exact(case, seed):
    kind = case["kind"]
    if kind in ("scf", "batch"):
        return None
    geoms, rng = _geometries(case, seed)
    b = BasisSet.build(geoms[0], case["basis"])
    if b.n_basis > (450 if kind == "setup" else 110):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    mol = _Mol(b, dev)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    if kind == "setup":
        return (mol.schwarz(),) + tuple(mol.one_electron())
    D = _decaying(b, rng, 1.0)
    if kind == "grad":
        return mol.eri_gradient(t(D))
    if kind == "rhf_grad":
        W = _decaying(b, rng, -1.0)
        return mol.eri_gradient(t(D)) + mol.one_electron_gradient(t(D), t(W))
    if kind == "multi":
        D = np.stack([_decaying(b, rng, 0.0) for _ in range(case["nset"])])
        return mol.jk(t(D))
    if kind == "fock":
        H = t(_decaying(b, rng, -8.0))
        J, K = mol.jk(t(D)[None])
        return H + J[0] - 0.5 * K[0]
    J, K = mol.jk(t(D)[None])
    return J[0], K[0]
