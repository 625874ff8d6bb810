"""The work that programs built on this library have it do, as measurable cases.

Each case is one call (or the few calls of one step) through the public entry
points, on seeded water clusters and alkanes in the bundled basis sets.  A case
names its path (which entry point), its system (kind and size) and its basis;
``draw`` gives further cases of the same paths over the whole range of sizes.

``exact`` evaluates the same quantities by another method (McMurchie-Davidson
Hermite expansions with the Boys function from its series, everything in 64 bits
in plain torch) for the systems small enough for it.
"""
import functools
import importlib
import math

import numpy as np
import torch

lai = importlib.import_module("libaccint-public_b200")

THRESHOLD = 1e-12       # Schwarz cut of every engine (its default)
FP32_CUT = 1e-7         # mixed-precision builds: quartets below this bound in FP32
AUX = "cc-pvdz-ri"      # auxiliary basis of the density-fitted builds


def listed():
    return [
        # a single molecule in a minimal basis: the smallest call, launches and latency only
        {"name": "water1_sto3g", "path": "jk", "system": "water", "n": 1, "basis": "sto-3g"},
        # a cluster in a minimal basis (the repository's smallest benchmark system)
        {"name": "water8_sto3g", "path": "jk", "system": "water", "n": 8, "basis": "sto-3g"},
        # the drop-in Engine.compute(op, FockBuilder) with host matrices, split-valence, odd size
        {"name": "water5_631g_host", "path": "host", "system": "water", "n": 5, "basis": "6-31g"},
        # an ordinary J/K build, once per SCF iteration
        {"name": "water16_ccpvdz", "path": "jk", "system": "water", "n": 16, "basis": "cc-pvdz"},
        # the repository's headline system: the largest build
        {"name": "water64_ccpvdz", "path": "jk", "system": "water", "n": 64, "basis": "cc-pvdz"},
        # f shells, a chain molecule off its ideal geometry
        {"name": "alkane6_ccpvtz", "path": "jk", "system": "alkane", "n": 6, "basis": "cc-pvtz"},
        # g shells: every class up to (gg|gg)
        {"name": "water1_ccpvqz", "path": "jk", "system": "water", "n": 1, "basis": "cc-pvqz"},
        # a mixed-precision build, the early SCF iterations of a larger cluster
        {"name": "water23_ccpvdz_mixed", "path": "mixed", "system": "water", "n": 23, "basis": "cc-pvdz"},
        # the nuclear gradient of a geometry step, host matrices
        {"name": "water6_ccpvdz_gradient", "path": "gradient", "system": "water", "n": 6, "basis": "cc-pvdz"},
        # many independent small systems in one engine
        {"name": "clusters32_ccpvdz", "path": "batched", "system": "water", "n": 32, "basis": "cc-pvdz"},
        # the one-shot jk(basis, D): a new geometry, engine set-up included
        {"name": "water6_ccpvdz_oneshot", "path": "oneshot", "system": "water", "n": 6, "basis": "cc-pvdz"},
        # density-fitted J and K of a new geometry: three-centre integrals, fit and contraction
        {"name": "water8_ccpvdz_df", "path": "df", "system": "water", "n": 8, "basis": "cc-pvdz"},
    ]


# (path, system, basis, smallest n, largest n): the ranges the listed cases stand for
RANGES = [
    ("jk", "water", "sto-3g", 1, 48),
    ("jk", "water", "6-31g", 1, 32),
    ("jk", "water", "cc-pvdz", 1, 40),
    ("jk", "water", "aug-cc-pvdz", 1, 8),
    ("jk", "water", "cc-pvtz", 1, 6),
    ("jk", "alkane", "cc-pvdz", 1, 12),
    ("jk", "alkane", "cc-pvtz", 1, 7),
    ("jk", "water", "cc-pvqz", 1, 2),
    ("host", "water", "sto-3g", 1, 24),
    ("host", "water", "6-31g", 1, 12),
    ("host", "alkane", "cc-pvdz", 1, 8),
    ("mixed", "water", "cc-pvdz", 2, 40),
    ("mixed", "alkane", "cc-pvtz", 1, 6),
    ("gradient", "water", "sto-3g", 1, 16),
    ("gradient", "water", "cc-pvdz", 1, 8),
    ("gradient", "alkane", "6-31g", 1, 8),
    ("batched", "water", "cc-pvdz", 3, 48),
    ("batched", "water", "sto-3g", 3, 96),
    ("oneshot", "water", "cc-pvdz", 1, 12),
    ("oneshot", "alkane", "6-31g", 1, 10),
    ("df", "water", "cc-pvdz", 1, 10),
    ("df", "alkane", "cc-pvdz", 1, 8),
]


def draw(rng):
    path, system, basis, lo, hi = rng.choice(RANGES)
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return {"path": path, "system": system, "n": n, "basis": basis}


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------

def _atoms(system, n, rng):
    if system == "water":
        return lai.molecules.water_cluster_n(n, rng)
    Z, xyz = lai.molecules.alkane(n)
    return Z, xyz + rng.normal(0.0, 0.05, xyz.shape)


def _nocc(system, n):
    return 5 * n if system == "water" else 4 * n + 1


def _systems(case, seed):
    """[(Z, xyz, occupied orbitals)] of the case: one system, or the batch's."""
    rng = np.random.default_rng(seed)
    if case["path"] == "batched":  # one to six molecules each
        sizes = rng.permutation([1 + i % 6 for i in range(case["n"])])
    else:
        sizes = [case["n"]]
    out = []
    for n in sizes:
        Z, xyz = _atoms(case["system"], int(n), rng)
        nbf = _nbf(Z, case["basis"])
        C = rng.normal(0.0, 1.0 / math.sqrt(nbf), size=(nbf, min(nbf, _nocc(case["system"], int(n)))))
        out.append((Z, xyz, C))
    return out


_SYMBOL = {1: "H", 6: "C", 8: "O"}


def _nbf(Z, basis):
    data = lai.basis_data(basis)
    return sum((l + 1) * (l + 2) // 2 for z in Z for l, _, _ in data[_SYMBOL[int(z)]])


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    path = case["path"]
    systems = _systems(case, seed)
    bases = [lai.BasisSet.from_atoms(Z, xyz, case["basis"]) for Z, xyz, _ in systems]
    state = {"path": path, "basis": bases[0]}
    if path == "batched":
        eng = lai.BatchedEngine(bases, threshold=THRESHOLD)
        D = torch.from_numpy(eng.pack([C @ C.T for _, _, C in systems])).to(dev)
    else:
        Cn = systems[0][2]
        eng = None if path == "oneshot" else lai.Engine(bases[0], threshold=THRESHOLD)
        if path == "df":
            state["aux"] = lai.BasisSet.from_atoms(systems[0][0], systems[0][1], AUX)
            state["C"] = torch.from_numpy(Cn).to(dev)
        if path == "host":
            state["builder"] = lai.FockBuilder(bases[0].nbf)
        D = Cn @ Cn.T
        if path in ("jk", "mixed"):
            D = torch.from_numpy(D).to(dev)
    state["engine"], state["D"] = eng, D
    if path in ("jk", "mixed", "batched"):
        state["J"], state["K"] = torch.empty_like(D), torch.empty_like(D)
    return state


def run(state):
    path, eng, D = state["path"], state["engine"], state["D"]
    if path in ("jk", "mixed", "batched"):
        J, K = state["J"], state["K"]
        eng.jk_device(D.data_ptr(), J.data_ptr(), K.data_ptr(), stream=torch.cuda.current_stream().cuda_stream,
                      fp32_cut=FP32_CUT if path == "mixed" else 0.0)
        return J, K
    if path == "host":
        fb = state["builder"]
        fb.reset()
        fb.set_density(D)
        eng.compute(lai.Operator.coulomb(), fb)
        return fb.get_coulomb_matrix(), fb.get_exchange_matrix()
    if path == "gradient":
        return eng.gradient(D)
    if path == "oneshot":
        return lai.jk(state["basis"], D, threshold=THRESHOLD)
    df = lai.df.DFFockBuilder(eng, state["aux"])
    df.set_orbitals(state["C"])
    return df.compute_coulomb(), df.compute_exchange()


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------

def _shell_list(Z, xyz, basis):
    """(l, centre, exponents, normalized coefficients) of every shell, zero
    coefficients dropped."""
    data = lai.basis_data(basis)
    out = []
    for z, r in zip(Z, xyz):
        for l, e, c in data[_SYMBOL[int(z)]]:
            e, c = np.array(e, float), np.array(c, float)
            df = float(np.prod(np.arange(2 * l - 1, 0, -2))) if l else 1.0
            c = c * (2 * e / math.pi) ** 0.75 * (4 * e) ** (0.5 * l) / math.sqrt(df)
            z2 = e[:, None] + e[None, :]
            c = c / math.sqrt(float(np.sum(c[:, None] * c[None, :] * (math.pi / z2) ** 1.5 * (0.5 / z2) ** l)))
            out.append((l, np.asarray(r, float), e[c != 0.0], c[c != 0.0]))
    return out


_DEC = 4  # histogram bins per decade of the bounds


def _pair_histograms(shells):
    """Per (la, lb) class: 2-D counts of primitive pairs over (decade of the
    primitive bound, decade of the shell pair's bound), and 1-D counts of shell
    pairs; bounds sqrt((ab|ab)) estimated from s functions."""
    nb = 20 * _DEC
    out = {}
    by_l = {}
    for i, s in enumerate(shells):
        by_l.setdefault((s[0], len(s[2])), []).append(i)
    bin_of = lambda q: np.clip((-np.log10(np.maximum(q, 1e-30)) + 2.0) * _DEC, 0, nb - 1).astype(int)  # noqa: E731
    for (la, Ka), ia in by_l.items():
        for (lb, Kb), ib in by_l.items():
            if (la, Ka) < (lb, Kb):
                continue
            I, J = np.meshgrid(ia, ib, indexing="ij")
            keep = I >= J if (la, Ka) == (lb, Kb) else np.ones_like(I, bool)
            I, J = I[keep], J[keep]
            R = np.array([s[1] for s in shells])
            r2 = np.sum((R[I] - R[J]) ** 2, axis=1)[:, None, None]
            ea, ca = (np.array([shells[i][k] for i in range(len(shells)) if i in set(ia)]) for k in (2, 3))
            eb, cb = (np.array([shells[i][k] for i in range(len(shells)) if i in set(ib)]) for k in (2, 3))
            pa, pb = {i: k for k, i in enumerate(sorted(ia))}, {i: k for k, i in enumerate(sorted(ib))}
            ai, bi = np.array([pa[i] for i in I], int), np.array([pb[j] for j in J], int)
            a, b = ea[ai][:, :, None], eb[bi][:, None, :]
            p = a + b
            q = (np.abs(ca[ai][:, :, None] * cb[bi][:, None, :]) * np.exp(-a * b / p * r2) *
                 np.sqrt(2 * math.pi ** 2.5 / (p * p * np.sqrt(2 * p))) * (0.25 / p) ** (0.5 * (la + lb)))
            q = q.reshape(len(I), -1)
            qs = bin_of(q.sum(axis=1))
            h2 = np.zeros((nb, nb))
            np.add.at(h2, (bin_of(q).ravel(), np.repeat(qs, q.shape[1])), 1.0)
            key = (max(la, lb), min(la, lb))
            o = out.setdefault(key, [np.zeros((nb, nb)), np.zeros(nb)])
            o[0] += h2
            o[1] += np.bincount(qs, minlength=nb)
    return out


def _counts(shells):
    """{(la, lb, lc, ld): (contracted, primitive) quartets above the cuts}, canonical."""
    H = sorted(_pair_histograms(shells).items())
    out = {}
    for i, (ab, (h2, h1)) in enumerate(H):
        nb = len(h1)
        lim = lambda thr: int((-math.log10(thr) + 4.0) * _DEC)  # noqa: E731  sum of two bins below it passes
        for cd, (g2, g1) in H[:i + 1]:
            w = 0.5 if ab == cd else 1.0
            nq = float(np.convolve(h1, g1)[:lim(THRESHOLD)].sum())
            s = (2 * nb, 2 * nb)
            conv = np.fft.irfft2(np.fft.rfft2(h2, s) * np.fft.rfft2(g2, s), s)
            npq = float(conv[:lim(1e-3 * THRESHOLD), :lim(THRESHOLD)].sum())
            out[ab + cd] = (w * nq, w * npq)
    return out


def _ncart(l):
    return (l + 1) * (l + 2) // 2


def _per_primitive(la, lb, lc, ld, der):
    """Operations of one primitive quartet: prefactors, n roots and weights, the
    2-D tables and the (e0|f0) products of every root."""
    L1, L2 = la + lb + (1 if der else 0), lc + ld
    n = (L1 + L2) // 2 + 1
    ne = sum(_ncart(e) for e in range(la, L1 + 1))
    nf = sum(_ncart(f) for f in range(lc, L2 + 1))
    one = 40.0 + 48.0 * n + n * (20.0 + 15.0 * (L1 + 1) * (L2 + 1) + 3.0 * ne * nf)
    return 3.0 * one if der else one


@functools.lru_cache(maxsize=None)
def _flops(path, system, n, basis):
    if path == "batched":
        per = [_flops("jk", system, k, basis) for k in range(1, 7)]
        return sum(per[i % 6] for i in range(n))
    Z, xyz = _atoms(system, n, np.random.default_rng(0))
    shells = _shell_list(Z, xyz, basis)
    nbf = _nbf(Z, basis)
    if path == "df":
        naux, nocc = _nbf(Z, AUX), _nocc(system, n)
        # metric, triangular solve, J by two products with the tensor, K by two contractions
        return naux ** 3 / 3.0 + float(nbf) ** 2 * naux ** 2 + 4.0 * nbf ** 2 * naux + \
            2.0 * naux * nbf ** 2 * nocc + float(nbf) ** 2 * naux * nocc
    der = path == "gradient"
    total = 0.0
    for (la, lb, lc, ld), (nq, npq) in _counts(shells).items():
        nc = _ncart(la) * _ncart(lb) * _ncart(lc) * _ncart(ld)
        total += npq * _per_primitive(la, lb, lc, ld, der) + nq * (75.0 if der else 25.0) * nc
    return total


def work(case):
    path = case["path"]
    rng = np.random.default_rng(0)
    if path == "batched":
        elems = sum(_nbf(_atoms(case["system"], 1 + i % 6, rng)[0], case["basis"]) ** 2 for i in range(case["n"]))
    else:
        elems = _nbf(_atoms(case["system"], case["n"], rng)[0], case["basis"]) ** 2
    moved = 1 if path == "gradient" else 3  # D in, J and K out
    return {"bytes": 8.0 * moved * elems, "flops": _flops(path, case["system"], case["n"], case["basis"])}


def tolerance(case):
    # Against exact(): the screened builds are off by what the Schwarz cut leaves out,
    # up to 3e-12 of J and K and 5e-12 of the gradient (run to run 1e-15); the
    # density-fitted J and K, unscreened, by 1.4e-15.  About four times that.
    path = case["path"]
    if path == "df":
        return {"rel": 5e-14}
    return {"rel": 2e-11 if path == "gradient" else 1e-11}


# ----------------------------------------------------------------------------
# the same quantities by another method, in 64 bits
# ----------------------------------------------------------------------------

def _boys(T, M):
    """[F_0 .. F_M](T): the ascending series of F_M and downward recursion for T < 36,
    erf and upward recursion above."""
    lo = T < 36.0
    t = torch.where(lo, T, torch.zeros_like(T))
    ex = torch.exp(-t)
    term = torch.full_like(t, 1.0 / (2 * M + 1))
    s = term.clone()
    for k in range(1, 130):
        term = term * (2.0 * t / (2 * M + 2 * k + 1))
        s = s + term
    down = [None] * (M + 1)
    down[M] = ex * s
    for m in range(M, 0, -1):
        down[m - 1] = (2.0 * t * down[m] + ex) / (2 * m - 1)
    u = torch.where(lo, torch.full_like(T, 36.0), T)
    exu = torch.exp(-u)
    up = [0.5 * torch.sqrt(math.pi / u) * torch.erf(torch.sqrt(u))]
    for m in range(M):
        up.append(((2 * m + 1) * up[m] - exu) / (2.0 * u))
    return torch.stack([torch.where(lo, d, v) for d, v in zip(down, up)])


class _Boys(torch.autograd.Function):
    @staticmethod
    def forward(ctx, T, M):
        F = _boys(T, M + 1)
        ctx.save_for_backward(F)
        return F[:-1]

    @staticmethod
    def backward(ctx, g):
        (F,) = ctx.saved_tensors
        return -(g * F[1:]).sum(0), None


@functools.lru_cache(maxsize=None)
def _herm(L):
    return [(t, u, n - t - u) for n in range(L + 1) for t in range(n, -1, -1) for u in range(n - t, -1, -1)]


def _cart(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _E_tables(la, lb, a, b, AB):
    """E[i][j][t] of one direction (without the exponential prefactor)."""
    p = a + b
    pa, pb, h = -b / p * AB, a / p * AB, 0.5 / p
    one = torch.ones_like(pa)
    E = {(0, 0): [one]}
    get = lambda v, t: v[t] if 0 <= t < len(v) else 0.0  # noqa: E731
    for i in range(la + 1):
        for j in range(lb + 1):
            if i == j == 0:
                continue
            src, x = (E[(i - 1, j)], pa) if i else (E[(i, j - 1)], pb)
            E[(i, j)] = [h * get(src, t - 1) + x * get(src, t) + (t + 1) * get(src, t + 1) for t in range(i + j + 1)]
    return E


def _norm(c):
    d = 1.0
    for k in c:
        for m in range(2 * k - 1, 1, -2):
            d *= m
    return 1.0 / math.sqrt(d)


class _Pairs:
    """Shell pairs (i >= j) of one (la, Ka, lb, Kb) class: function indices, and per
    primitive pair the exponent, the centre and the Hermite coefficients."""

    def __init__(self, shells, func, R, idx, dev):
        I, J = idx[:, 0], idx[:, 1]
        self.n = len(idx)
        self.la, self.lb = shells[I[0]][0], shells[J[0]][0]
        A, B = R[torch.as_tensor(I, device=dev)], R[torch.as_tensor(J, device=dev)]
        put = lambda k, at: torch.as_tensor(np.array([shells[i][k] for i in at]), device=dev)  # noqa: E731
        a, b = put(2, I)[:, :, None], put(2, J)[:, None, :]
        cab = put(3, I)[:, :, None] * put(3, J)[:, None, :]
        p = a + b
        AB = A - B
        K = torch.exp(-a * b / p * (AB ** 2).sum(1)[:, None, None])
        self.p = p.reshape(self.n, -1)
        self.P = ((a[..., None] * A[:, None, None] + b[..., None] * B[:, None, None]) / p[..., None]).reshape(self.n, -1, 3)
        E = [_E_tables(self.la, self.lb, a, b, AB[:, x][:, None, None]) for x in range(3)]
        hs = _herm(self.la + self.lb)
        rows = []
        zero = torch.zeros_like(K)
        for ca in _cart(self.la):
            for cb in _cart(self.lb):
                nrm = _norm(ca) * _norm(cb)
                e = [E[x][(ca[x], cb[x])] for x in range(3)]
                rows.append(torch.stack([nrm * cab * K * e[0][t] * e[1][u] * e[2][v]
                                         if t < len(e[0]) and u < len(e[1]) and v < len(e[2]) else zero
                                         for t, u, v in hs], -1).reshape(self.n, -1, len(hs)))
        self.E = torch.stack(rows, 2)                       # [pair, prim, component, hermite]
        na, nb = len(_cart(self.la)), len(_cart(self.lb))
        fa = torch.as_tensor(func[I], device=dev)[:, None, None] + torch.arange(na, device=dev)[None, :, None]
        fb = torch.as_tensor(func[J], device=dev)[:, None, None] + torch.arange(nb, device=dev)[None, None, :]
        self.fa = (fa + 0 * fb).reshape(self.n, -1)
        self.fb = (fb + 0 * fa).reshape(self.n, -1)
        self.w = torch.as_tensor(np.where(I == J, 0.5, 1.0), device=dev)

    def detached(self):
        self.leaf = [t.detach().requires_grad_(t.requires_grad) for t in (self.P, self.E)]
        return self


def _all_pairs(shells, func, R, dev):
    by = {}
    for i, s in enumerate(shells):
        by.setdefault((s[0], len(s[2])), []).append(i)
    keys = sorted(by)
    out = []
    for x, ka in enumerate(keys):
        for kb in keys[:x + 1]:
            idx = np.array([(i, j) for i in by[ka] for j in by[kb] if ka != kb or i >= j], dtype=int)
            out.append(_Pairs(shells, func, R, idx, dev))
    return out


def _hermite_R(L, alpha, PQ):
    """R_tuv of all t + u + v <= L, stacked last in the order of _herm(L)."""
    F = _Boys.apply(alpha * (PQ ** 2).sum(-1), L)
    memo = {}

    def R(n, t, u, v):
        k = (n, t, u, v)
        if k in memo:
            return memo[k]
        if t == u == v == 0:
            r = (-2.0 * alpha) ** n * F[n]
        else:
            x = 0 if t else 1 if u else 2
            lo = [t, u, v]
            lo[x] -= 1
            r = PQ[..., x] * R(n + 1, *lo)
            if lo[x] > 0:
                m = lo[x]
                lo[x] -= 1
                r = r + m * R(n + 1, *lo)
        memo[k] = r
        return r

    return torch.stack([R(0, *h) for h in _herm(L)], -1)


def _block(b, bs, k, ks, bP, bE, kP, kE):
    """(ab|cd) of bra pairs bs against ket pairs ks: [bra, comp, ket, comp]."""
    Lb, Lk = b.la + b.lb, k.la + k.lb
    hb, hk = _herm(Lb), _herm(Lk)
    at = {h: i for i, h in enumerate(_herm(Lb + Lk))}
    p, q = b.p[bs].reshape(-1)[:, None], k.p[ks].reshape(-1)[None, :]
    PQ = bP[bs].reshape(-1, 1, 3) - kP[ks].reshape(1, -1, 3)
    R = _hermite_R(Lb + Lk, p * q / (p + q), PQ)
    pre = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
    ix = torch.tensor([[at[tuple(x + y for x, y in zip(g, h))] for h in hk] for g in hb], device=R.device)
    sg = torch.tensor([(-1.0) ** sum(h) for h in hk], dtype=R.dtype, device=R.device)
    R = (R * pre[..., None])[..., ix] * sg                    # [bra prim, ket prim, Hb, Hk]
    Eb, Ek = bE[bs], kE[ks]
    nb, Kb, nk, Kk = Eb.shape[0], Eb.shape[1], Ek.shape[0], Ek.shape[1]
    R = R.reshape(nb, Kb, nk, Kk, len(hb), len(hk))
    X = torch.einsum("bpkqgh,kqdh->bpkgd", R, Ek)
    return torch.einsum("bpkgd,bpcg->bckd", X, Eb)


def _quartet_cost(b, k):
    L = b.la + b.lb + k.la + k.lb
    per = 3 * len(_herm(b.la + b.lb)) * len(_herm(k.la + k.lb)) + 6 * len(_herm(L)) + 300
    return float(b.p.numel()) * k.p.numel() * per


def _chunks(b, k, budget):
    """Bra and ket slices whose Hermite tensors stay within budget elements."""
    per = b.p.shape[1] * k.p.shape[1] * (3 * len(_herm(b.la + b.lb)) * len(_herm(k.la + k.lb)) + 200)
    nk = max(1, min(k.n, budget // per))
    nb = max(1, min(b.n, budget // (per * nk)))
    for i in range(0, b.n, nb):
        for j in range(0, k.n, nk):
            yield slice(i, min(b.n, i + nb)), slice(j, min(k.n, j + nk))


def _exact_jk(shells, D, dev, grad_R=None):
    """J and K of the density, or with grad_R (centres that require gradients, and
    the shells' atoms) the gradient of 1/2 tr DJ - 1/4 tr DK."""
    func = np.concatenate([[0], np.cumsum([_ncart(s[0]) for s in shells])])
    n = int(func[-1])
    D = torch.as_tensor(D, device=dev)
    if grad_R is None:
        R = torch.as_tensor(np.array([s[1] for s in shells]), device=dev)
    else:
        R = grad_R[0][torch.as_tensor(grad_R[1], device=dev)]
    pairs = [p.detached() for p in _all_pairs(shells, func, R, dev)]
    J, K = torch.zeros((n, n), dtype=torch.float64, device=dev), torch.zeros((n, n), dtype=torch.float64, device=dev)
    flat = lambda M, r, c, v: M.view(-1).index_add_(0, (r * n + c).reshape(-1), v.reshape(-1))  # noqa: E731
    for x, b in enumerate(pairs):
        for k in pairs[:x + 1]:
            w0 = 0.5 if b is k else 1.0
            for bs, ks in _chunks(b, k, 1 << 26):
                (bP, bE), (kP, kE) = b.leaf, k.leaf
                V = _block(b, bs, k, ks, bP, bE, kP, kE)
                V = V * (w0 * b.w[bs][:, None, None, None] * k.w[ks][None, None, :, None])
                fa, fb = b.fa[bs][:, :, None, None], b.fb[bs][:, :, None, None]
                fc, fd = k.fa[ks][None, None], k.fb[ks][None, None]
                if grad_R is not None:
                    G = 4.0 * D[fa, fb] * D[fc, fd] - D[fa, fc] * D[fb, fd] - D[fa, fd] * D[fb, fc]
                    (V * G).sum().backward()
                    continue
                z = 0 * (fa + fc)
                # every distinct integral feeds its whole orbit; J and K are symmetrized at the end
                flat(J, fa + z, fb + z, 2.0 * V * D[fc, fd])
                flat(J, fc + z, fd + z, 2.0 * V * D[fa, fb])
                flat(K, fa + z, fc + z, V * D[fb, fd])
                flat(K, fa + z, fd + z, V * D[fb, fc])
                flat(K, fb + z, fc + z, V * D[fa, fd])
                flat(K, fb + z, fd + z, V * D[fa, fc])
    if grad_R is None:
        return J + J.T, K + K.T
    todo = [(t, l.grad) for p in pairs for t, l in zip((p.P, p.E), p.leaf) if l.grad is not None]
    torch.autograd.backward([t for t, _ in todo], [g for _, g in todo])
    return grad_R[0].grad


def _exact_df(shells, aux, C, dev):
    func = np.concatenate([[0], np.cumsum([_ncart(s[0]) for s in shells])])
    n = int(func[-1])
    unit = (0, np.zeros(3), np.zeros(1), np.ones(1))  # the constant function 1 beside each auxiliary shell
    ash = aux + [unit]
    afunc = np.concatenate([[0], np.cumsum([_ncart(s[0]) for s in ash])])
    R = torch.as_tensor(np.array([s[1] for s in shells]), device=dev)
    aR = torch.as_tensor(np.array([s[1] for s in ash]), device=dev)
    naux = int(afunc[-1]) - 1
    by = {}
    for i, s in enumerate(aux):
        by.setdefault((s[0], len(s[2])), []).append(i)
    axp = [_Pairs(ash, afunc, aR, np.array([(i, len(aux)) for i in v]), dev) for v in by.values()]
    T = torch.zeros((n, n, naux), dtype=torch.float64, device=dev)
    V = torch.zeros((naux, naux), dtype=torch.float64, device=dev)
    for k in axp:
        for b in _all_pairs(shells, func, R, dev):
            for bs, ks in _chunks(b, k, 1 << 26):
                X = _block(b, bs, k, ks, b.P, b.E, k.P, k.E)
                r, c, a = b.fa[bs][:, :, None, None], b.fb[bs][:, :, None, None], k.fa[ks][None, None]
                T[r, c, a] = X
                T[c, r, a] = X
        for b in axp:
            V[b.fa.reshape(-1)[:, None], k.fa.reshape(-1)[None, :]] = \
                _block(b, slice(0, b.n), k, slice(0, k.n), b.P, b.E, k.P, k.E).reshape(b.fa.numel(), -1)
    C = torch.as_tensor(C, device=dev)
    L = torch.linalg.cholesky(0.5 * (V + V.T))
    B = torch.linalg.solve_triangular(L, T.reshape(n * n, naux).T, upper=False).reshape(naux, n, n)
    D = C @ C.T
    J = torch.einsum("pab,p->ab", B, torch.einsum("pcd,cd->p", B, D))
    X = torch.matmul(B, C)
    return J, torch.einsum("pai,pci->ac", X, X)


_MOST = 2e12  # operations (as _quartet_cost counts them) an exact evaluation may take


def exact(case, seed):
    path = case["path"]
    dev = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    systems = _systems(case, seed)
    shells = [_shell_list(Z, xyz, case["basis"]) for Z, xyz, _ in systems]
    if path == "df":
        Z, xyz, C = systems[0]
        return _exact_df(shells[0], _shell_list(Z, xyz, AUX), C, dev)
    cost = 0.0
    for sh in shells:
        prims = [(s[0], len(s[2])) for s in sh]
        # all primitive quartets, at the mean cost of one
        k = sum(x for _, x in prims)
        lm = sum(l * x for l, x in prims) / k
        cost += (k * (k + 1) / 2) ** 2 / 2 * (300 + 60 * (1 + lm) ** 6) * (4 if path == "gradient" else 1)
    if cost > _MOST:
        return None
    out = []
    for (Z, xyz, C), sh in zip(systems, shells):
        D = C @ C.T
        if path == "gradient":
            R = torch.as_tensor(np.asarray(xyz, float), device=dev).requires_grad_()
            data = lai.basis_data(case["basis"])
            atom = np.concatenate([[a] * len(data[_SYMBOL[int(z)]]) for a, z in enumerate(Z)]).astype(int)
            return _exact_jk(sh, D, dev, (R, atom)).cpu().numpy()
        out.append(_exact_jk(sh, D, dev))
    if path == "batched":
        return tuple(torch.cat([m[i].reshape(-1) for m in out]) for i in (0, 1))
    if path in ("host", "oneshot"):
        return tuple(m.cpu().numpy() for m in out[0])
    return out[0]
