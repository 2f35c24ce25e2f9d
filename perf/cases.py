"""The work that a user of this library has it do, as measurable cases.

Every case goes through the public Python entry points (Engine, Context) on
the synthetic water clusters and basis sets of the repository's benchmark and
tests.  `exact` restates the integrals in 64-bit torch by the
McMurchie-Davidson scheme (Hermite Gaussians; J. Comput. Phys. 26, 218
(1978)), which shares no formula or code with the library's kernels beyond
the definition of the integrals.
"""
import math

import numpy as np
import torch

import libint_gb300 as lg

FP64, MIXED, MIXED_FP32_BOYS = 0, 1, 2
MODES = {"fp64": FP64, "mixed": MIXED, "mixed_fp32_boys": MIXED_FP32_BOYS}
SCHWARZ = 1e-12
MIXED_THRESH = 1e-4


def listed():
    return [
        # one shell set per call, as a program written against libint's Engine asks for them:
        # contracted p shells, where the call's latency is everything
        {"name": "engine_pppp", "kind": "engine", "ls": "1111", "nprim": 3, "deriv": 0},
        # the same for nuclear gradients: 12 first-derivative sets of one shell quartet
        {"name": "engine_dpds_d1", "kind": "engine", "ls": "2120", "nprim": 2, "deriv": 1},
        # every unique quartet of a small cluster left on the GPU, no screening (a conventional,
        # integral-storing method; 692,076 quartets, 11.3M integrals)
        {"name": "batch_h2o4_dz", "kind": "batch", "waters": 4, "basis": "cc-pVDZ", "deriv": 0,
         "mode": "fp64", "quartets": 0, "host": False},
        # first-derivative sets of every unique quartet of a dimer
        {"name": "batch_h2o2_dz_d1", "kind": "batch", "waters": 2, "basis": "cc-pVDZ", "deriv": 1,
         "mode": "fp64", "quartets": 0, "host": False},
        # an explicit list of quartets up to (ff|ff), mixed precision, sets copied to host memory
        {"name": "batch_h2o3_tz_mixed", "kind": "batch", "waters": 3, "basis": "cc-pVTZ",
         "deriv": 0, "mode": "mixed", "quartets": 30001, "host": True},
        # density fitting: every (P|ab) of a cluster and its fitting basis, left on the GPU
        {"name": "df_h2o8_dz", "kind": "df", "waters": 8, "basis": "cc-pVDZ"},
        # the J/K build of one molecule in a small basis (SCF on host arrays): launches and latency
        {"name": "jk_h2o1_631g", "kind": "jk", "waters": 1, "basis": "6-31G", "mode": "fp64",
         "omega": 0.0, "host": True, "fock": 0.0},
        # range-separated exchange: erfc-attenuated J/K
        {"name": "jk_h2o16_dz_erfc", "kind": "jk", "waters": 16, "basis": "cc-pVDZ",
         "mode": "fp64", "omega": 0.4, "host": True, "fock": 0.0},
        # an ordinary double-zeta Fock build, mixed precision, matrices on the GPU
        {"name": "jk_h2o32_dz_mixed", "kind": "jk", "waters": 32, "basis": "cc-pVDZ",
         "mode": "mixed", "omega": 0.0, "host": False, "fock": 0.0},
        # an FP64 Fock build in the basis of the headline benchmark
        {"name": "jk_h2o8_tz_fp64", "kind": "jk", "waters": 8, "basis": "cc-pVTZ",
         "mode": "fp64", "omega": 0.0, "host": False, "fock": 0.0},
        # the headline pass (mixed precision, cc-pVTZ) at a size whose pass stays near a second
        {"name": "jk_h2o20_tz_mixed", "kind": "jk", "waters": 20, "basis": "cc-pVTZ",
         "mode": "mixed", "omega": 0.0, "host": False, "fock": 0.0},
        # nuclear gradients of the Coulomb and exchange energies
        {"name": "grad_h2o12_dz", "kind": "grad", "waters": 12, "basis": "cc-pVDZ"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["jk", "jk", "jk", "jk", "jk", "grad", "batch", "batch", "df", "engine"])
    if kind == "engine":
        return {"kind": kind, "ls": "".join(str(rng.randint(0, 3)) for _ in range(4)),
                "nprim": rng.randint(1, 5), "deriv": rng.randint(0, 2)}
    if kind == "df":
        return {"kind": kind, "waters": _log_int(rng, 1, 8), "basis": rng.choice(["6-31G", "cc-pVDZ"])}
    if kind == "grad":
        return {"kind": kind, "waters": _log_int(rng, 1, 12),
                "basis": rng.choice(["6-31G", "cc-pVDZ"])}
    if kind == "batch":
        deriv = rng.choice([0, 0, 1])
        return {"kind": kind, "waters": rng.randint(1, 4),
                "basis": rng.choice(["6-31G", "cc-pVDZ", "cc-pVTZ"]), "deriv": deriv,
                "mode": "fp64" if deriv else rng.choice(["fp64", "mixed", "mixed_fp32_boys"]),
                "quartets": _log_int(rng, 1, 20000 if deriv else 200000),
                "host": rng.random() < 0.5}
    basis, mode = rng.choice([("6-31G", "fp64"), ("6-31G", "mixed"), ("cc-pVDZ", "fp64"),
                              ("cc-pVDZ", "mixed"), ("cc-pVDZ", "mixed_fp32_boys"),
                              ("cc-pVTZ", "fp64"), ("cc-pVTZ", "mixed"),
                              ("cc-pVTZ", "mixed_fp32_boys"), ("aug-cc-pVDZ", "mixed")])
    top = {"6-31G": 40, "cc-pVDZ": 24, "cc-pVTZ": 18, "aug-cc-pVDZ": 12}[basis]
    if mode == "fp64":
        top //= 2
    omega = round(rng.uniform(0.1, 1.0), 3) if basis == "cc-pVDZ" and rng.random() < 0.3 else 0.0
    return {"kind": kind, "waters": _log_int(rng, 1, top), "basis": basis, "mode": mode,
            "omega": omega, "host": rng.random() < 0.5,
            "fock": 1e-9 if rng.random() < 0.2 else 0.0}


# ------------------------------------------------------------------ inputs
def _cluster(n, seed):
    """n water molecules on the smallest near-cubic grid that holds them."""
    nx = max(1, round(n ** (1.0 / 3.0)))
    ny = max(1, round(math.sqrt(n / nx)))
    nz = -(-n // (nx * ny))
    return lg.water_cluster(nx, ny, nz, seed=seed)[:3 * n]


def _engine_shells(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for c in case["ls"]:
        ex = np.exp(rng.uniform(math.log(0.15), math.log(12.0), case["nprim"]))
        co = rng.uniform(0.2, 1.0, case["nprim"])
        out.append(lg.Shell(int(c), list(zip(ex, co)), rng.uniform(-1.5, 1.5, 3), pure=int(c) > 1))
    return out


def _unique_quartets(ns):
    i, j = np.tril_indices(ns)
    b, k = np.tril_indices(len(i))
    return np.stack([i[b], j[b], i[k], j[k]], axis=1).astype(np.int32)


def _df_basis(case, seed):
    """Orbital basis, fitting basis and a unit shell (exponent 0) in one list, as the library's
    batched entry takes three-centre quartets (P unit|a b)."""
    atoms = _cluster(case["waters"], seed)
    bs, fit = lg.BasisSet(case["basis"], atoms), lg.BasisSet("cc-pVDZ-JKFIT", atoms)
    return lg.BasisSet(list(bs) + list(fit) + [lg.Shell.unit()]), len(bs), len(fit)


def _df_quartets(nb, nf):
    i, j = np.tril_indices(nb)
    P = np.repeat(np.arange(nb, nb + nf), len(i))
    n = len(P)
    return np.stack([P, np.full(n, nb + nf), np.tile(i, nf), np.tile(j, nf)],
                    axis=1).astype(np.int32)


def _list_inputs(case, seed):
    """Basis and quartet list of the explicit-list cases."""
    if case["kind"] == "df":
        bs, nb, nf = _df_basis(case, seed)
        return bs, _df_quartets(nb, nf)
    bs = lg.BasisSet(case["basis"], _cluster(case["waters"], seed))
    if case["quartets"] == 0:
        return bs, _unique_quartets(len(bs))
    rng = np.random.default_rng(case["quartets"])  # the list belongs to the case, the geometry to the seed
    return bs, rng.integers(0, len(bs), (case["quartets"], 4)).astype(np.int32)


def _density(case, nbf, seed):
    return lg.random_density(nbf, 5 * case["waters"], seed=seed + 2)


def prepare(case, seed):
    kind = case["kind"]
    ctx = lg.Context(0)
    st = {"case": case, "ctx": ctx}
    if kind == "engine":
        st["shells"] = _engine_shells(case, seed)
        st["engine"] = lg.Engine(lg.Operator.coulomb, case["nprim"],
                                 max(s.l for s in st["shells"]), case["deriv"], context=ctx)
        return st
    if kind in ("batch", "df"):
        bs, st["quartets"] = _list_inputs(case, seed)
        ctx.set_basis(bs)
        if not case.get("host", False):
            q = st["quartets"]
            sizes = np.array([s.size() for s in bs], np.int64)
            nv = np.prod(sizes[q], axis=1) * (12 if case.get("deriv", 0) else 1)
            st["offsets"] = np.concatenate([[0], np.cumsum(nv)[:-1]]).astype(np.int64)
            st["out"] = torch.empty(int(nv.sum()), dtype=torch.float64, device="cuda")
            st["null"] = torch.empty(len(q), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
        return st
    bs = lg.BasisSet(case["basis"], _cluster(case["waters"], seed))
    ctx.set_basis(bs)
    D = _density(case, bs.nbf, seed)
    if kind == "jk":
        if case["omega"] > 0:
            ctx.set_operator(lg.Operator.erfc_coulomb, case["omega"])
        if case["fock"] > 0:
            ctx.set_fock_precision(case["fock"])
        if not case["host"]:
            D = torch.from_numpy(D).cuda()
            st["J"], st["K"] = torch.empty_like(D), torch.empty_like(D)
            torch.cuda.synchronize()
    st["D"] = D
    return st


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "engine":
        r = st["engine"].compute(*st["shells"])
        return np.stack(r) if case["deriv"] else r
    if kind in ("batch", "df"):
        deriv, mode = case.get("deriv", 0), MODES[case.get("mode", "fp64")]
        if case.get("host", False):
            out, _, null = ctx.compute_batch(st["quartets"], deriv, mode, MIXED_THRESH)
            return {"sets": out, "null": null}
        ctx.compute_batch_device(st["quartets"], st["out"].data_ptr(), st["out"].numel(), deriv,
                                 mode, MIXED_THRESH, st["offsets"], st["null"].data_ptr())
        return {"sets": st["out"], "null": st["null"]}
    if kind == "grad":
        gJ, gK, _ = ctx.jk_grad(st["D"], schwarz_thresh=SCHWARZ)
        return {"gJ": gJ, "gK": gK}
    if case["host"]:
        J, K, _ = ctx.jk(st["D"], SCHWARZ, MODES[case["mode"]], MIXED_THRESH)
        return {"J": J, "K": K}
    ctx.jk_device(st["D"].data_ptr(), st["J"].data_ptr(), st["K"].data_ptr(), SCHWARZ,
                  MODES[case["mode"]], MIXED_THRESH)
    return {"J": st["J"], "K": st["K"]}


# -------------------------------------------------------------------- work
def _ncart(l):
    return (l + 1) * (l + 2) // 2


def _prim_flops(la, lb, lc, ld, deriv=0):
    """One primitive quartet: the prologue (exponent sums, P - Q, the Boys functions) and one
    recurrence of 8 operations for each (e0|f0) component below the targets."""
    L = la + lb + lc + ld + deriv
    e = sum(_ncart(l) for l in range(la + lb + 1))
    f = sum(_ncart(l) for l in range(lc + ld + 1))
    return 50 + 4 * L + 8 * e * f * (4 if deriv else 1)


def _pair_groups(bs):
    """{(la, lb, primitive pairs, functions): descending bounds sqrt (ab|ab) of the (ss|ss) part}
    over the unique shell pairs, an estimate of the Schwarz factors for the operation count."""
    kinds = {}
    for s in bs:
        kinds.setdefault((s.l, s.nprim(), s.size()), []).append(s)
    keys = sorted(kinds)
    groups = {}
    for x, kx in enumerate(keys):
        for ky in keys[: x + 1]:
            A, B = kinds[kx], kinds[ky]
            OA, OB = np.array([s.O for s in A]), np.array([s.O for s in B])
            R2 = np.sum((OA[:, None] - OB[None]) ** 2, axis=-1)
            Q2 = np.zeros_like(R2)
            for i in range(kx[1]):
                for j in range(ky[1]):
                    a, b = (np.array([s.alpha[t] for s in S]) for S, t in ((A, i), (B, j)))
                    ca, cb = (np.array([s.coeff[t] for s in S]) for S, t in ((A, i), (B, j)))
                    p = a[:, None] + b[None]
                    c = np.abs(ca / (4 * a) ** (kx[0] / 2))[:, None] * np.abs(cb / (4 * b) ** (ky[0] / 2))
                    K = c * np.exp(-a[:, None] * b[None] / p * R2)
                    Q2 = np.maximum(Q2, K * K * 2 * math.pi ** 2.5 / (p * p * np.sqrt(2 * p)))
            q = Q2[np.tril_indices(len(A))] if kx == ky else Q2.ravel()
            key = (max(kx[0], ky[0]), min(kx[0], ky[0]), kx[1] * ky[1], kx[2] * ky[2])
            groups.setdefault(key, []).append(np.sqrt(q))
    return {k: np.sort(np.concatenate(v))[::-1] for k, v in groups.items()}


def work(case):
    kind = case["kind"]
    if kind == "engine":
        ls, d = [int(c) for c in case["ls"]], case["deriv"]
        nf = math.prod(2 * l + 1 for l in ls)
        sets = {0: 1, 1: 12, 2: 78}[d]
        return {"bytes": 4 * (16 * case["nprim"] + 40) + 8 * nf * sets,
                "flops": case["nprim"] ** 4 * _prim_flops(*ls, d) + 10 * nf * sets}
    if kind in ("batch", "df"):
        bs, q = _list_inputs(case, 0)
        d = case.get("deriv", 0)
        l, n, size = bs.l, bs.nprim.astype(np.int64), np.array([s.size() for s in bs], np.int64)
        cls = np.sort(l[q].reshape(-1, 2, 2), axis=2)[:, :, ::-1].reshape(-1, 4)
        code = cls @ np.array([64, 16, 4, 1])
        np4 = np.prod(n[q], axis=1)
        vals = int(np.prod(size[q], axis=1).sum()) * (12 if d else 1)
        fl = sum(float(np4[code == c].sum()) * _prim_flops(c >> 6, c >> 4 & 3, c >> 2 & 3, c & 3, d)
                 for c in np.unique(code).tolist())
        return {"bytes": 16 * len(q) + 8 * vals, "flops": fl + 4.0 * vals}
    bs = lg.BasisSet(case["basis"], _cluster(case["waters"], 0))
    d = 1 if kind == "grad" else 0
    G = sorted(_pair_groups(bs).items())
    fl = 0.0
    for x, (kx, qx) in enumerate(G):
        for y, (ky, qy) in enumerate(G[: x + 1]):
            # quartets whose bounds multiply to the threshold (half of them within one group)
            asc = qy[::-1]
            nq = float(len(qy) * len(qx) - np.searchsorted(asc, SCHWARZ / np.maximum(qx, 1e-300)).sum())
            nq *= 0.5 if x == y else 1.0
            fl += nq * (kx[2] * ky[2] * _prim_flops(kx[0], kx[1], ky[0], ky[1], d) +
                        12 * kx[3] * ky[3] * (12 if d else 1))
    nn = 8 * bs.nbf ** 2
    return {"bytes": nn + 48 * case["waters"] * 3 if d else 3 * nn, "flops": fl}


# ------------------------------------------------------------------- exact
# Operations (elements of the Hermite interaction matrices) and shells above which `exact` gives
# None: it would take too long, or its quartet list too much memory.
EXACT_MOST = 3e10
EXACT_SHELLS = 100

_SQ3, _SQ15 = math.sqrt(3.0), math.sqrt(15.0)
# real solid harmonics m = -l..l over {(lx, ly, lz): coefficient}
_SOLID = {
    2: [{(1, 1, 0): _SQ3}, {(0, 1, 1): _SQ3},
        {(0, 0, 2): 1.0, (2, 0, 0): -0.5, (0, 2, 0): -0.5}, {(1, 0, 1): _SQ3},
        {(2, 0, 0): 0.5 * _SQ3, (0, 2, 0): -0.5 * _SQ3}],
    3: [{(2, 1, 0): 3 * math.sqrt(0.625), (0, 3, 0): -math.sqrt(0.625)}, {(1, 1, 1): _SQ15},
        {(0, 1, 2): 4 * math.sqrt(0.375), (2, 1, 0): -math.sqrt(0.375), (0, 3, 0): -math.sqrt(0.375)},
        {(0, 0, 3): 1.0, (2, 0, 1): -1.5, (0, 2, 1): -1.5},
        {(1, 0, 2): 4 * math.sqrt(0.375), (3, 0, 0): -math.sqrt(0.375), (1, 2, 0): -math.sqrt(0.375)},
        {(2, 0, 1): 0.5 * _SQ15, (0, 2, 1): -0.5 * _SQ15},
        {(3, 0, 0): math.sqrt(0.625), (1, 2, 0): -3 * math.sqrt(0.625)}],
}


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _carts(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _solid(l, pure):
    """Transform of the Cartesian components of one shell (identity when Cartesian)."""
    cs = _carts(l)
    if not pure:
        return torch.eye(len(cs), dtype=torch.float64, device=_dev())
    M = torch.zeros(2 * l + 1, len(cs), dtype=torch.float64, device=_dev())
    rows = _SOLID[l] if l in _SOLID else [{c: 1.0} for c in ([(0, 0, 0)] if l == 0 else
                                                             [(0, 1, 0), (0, 0, 1), (1, 0, 0)])]
    for p, row in enumerate(rows):
        for c, v in row.items():
            M[p, cs.index(c)] = v
    return M


def _herm(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


class _Pairs:
    """Hermite expansions of a list of shell pairs of one kind, differentiated `da` / `db` times
    (per direction) with respect to the first / second centre."""

    def __init__(self, A, B, da=(0, 0, 0), db=(0, 0, 0)):
        t = dict(dtype=torch.float64, device=_dev())
        la, lb = A[0].l, B[0].l
        self.L = la + lb + sum(da) + sum(db)
        a = torch.tensor(np.array([s.alpha for s in A]), **t)[:, :, None]
        b = torch.tensor(np.array([s.alpha for s in B]), **t)[:, None, :]
        c = (torch.tensor(np.array([s.coeff for s in A]), **t)[:, :, None] *
             torch.tensor(np.array([s.coeff for s in B]), **t)[:, None, :])
        OA = torch.tensor(np.array([s.O for s in A]), **t)[:, None, None]
        OB = torch.tensor(np.array([s.O for s in B]), **t)[:, None, None]
        p = a + b
        P = (a[..., None] * OA + b[..., None] * OB) / p[..., None]
        E = []
        for x in range(3):
            ni, nj = la + da[x], lb + db[x]
            PA, PB = P[..., x] - OA[..., x], P[..., x] - OB[..., x]
            zero = torch.zeros_like(p)
            e = {(0, 0, 0): torch.exp(-a * b / p * (OA - OB)[..., x] ** 2)}
            get = lambda i, j, k: e.get((i, j, k), zero)  # noqa: E731
            for i in range(ni + 1):
                for j in range(nj + 1):
                    if i + j == 0:
                        continue
                    i0, j0, X = (i - 1, j, PA) if i else (i, j - 1, PB)
                    for k in range(i + j + 1):
                        e[i, j, k] = (get(i0, j0, k - 1) / (2 * p) + X * get(i0, j0, k) +
                                      (k + 1) * get(i0, j0, k + 1))
            # d/dA x^i exp(-a x^2) = 2a x^(i+1) - i x^(i-1), the same for B
            for _ in range(da[x]):
                ni -= 1
                e = {(i, j, k): 2 * a * get(i + 1, j, k) - i * get(i - 1, j, k)
                     for i in range(ni + 1) for j in range(nj + 1) for k in range(self.L + 1)}
            for _ in range(db[x]):
                nj -= 1
                e = {(i, j, k): 2 * b * get(i, j + 1, k) - j * get(i, j - 1, k)
                     for i in range(ni + 1) for j in range(nj + 1) for k in range(self.L + 1)}
            E.append(e)
        n, k = len(A), a.shape[1] * b.shape[2]
        ca, cb, hs = _carts(la), _carts(lb), _herm(self.L)
        H = torch.zeros(n, k, len(ca), len(cb), len(hs), **t)
        for ia, u in enumerate(ca):
            for ib, w in enumerate(cb):
                for ih, h in enumerate(hs):
                    f = [E[x].get((u[x], w[x], h[x])) for x in range(3)]
                    if all(g is not None for g in f):
                        H[:, :, ia, ib, ih] = (c * f[0] * f[1] * f[2]).reshape(n, k)
        Ma, Mb = _solid(la, A[0].pure), _solid(lb, B[0].pure)
        self.nf = (Ma.shape[0], Mb.shape[0])
        self.H = torch.einsum("pa,qb,nkabh->nkpqh", Ma, Mb, H).reshape(n, k, -1, len(hs)).contiguous()
        self.p, self.P, self.k = p.reshape(n, k), P.reshape(n, k, 3), k


def _boys(L, T):
    """F_0..F_L(T), T >= 0."""
    big = T > 45.0
    Ts = torch.where(big, torch.zeros_like(T), T)
    eT = torch.exp(-Ts)
    term = torch.full_like(T, 1.0 / (2 * L + 1))
    s = term.clone()
    for i in range(1, 190):
        term = term * (2.0 * Ts) / (2 * L + 2 * i + 1)
        s = s + term
    F = [None] * (L + 1)
    F[L] = eT * s
    for m in range(L - 1, -1, -1):
        F[m] = (2 * Ts * F[m + 1] + eT) / (2 * m + 1)
    Tb = torch.where(big, T, torch.full_like(T, 50.0))
    eb, f = torch.exp(-Tb), 0.5 * torch.sqrt(math.pi / Tb)
    for m in range(L + 1):
        F[m] = torch.where(big, f, F[m])
        f = ((2 * m + 1) * f - eb) / (2 * Tb)
    return F


def _eri(X, Y, ix, iy, omega=0.0):
    """(ab|cd) of bra pairs X[ix] with ket pairs Y[iy]: n x (functions ab) x (functions cd)."""
    L = X.L + Y.L
    p, q = X.p[ix][:, :, None], Y.p[iy][:, None, :]
    R = X.P[ix][:, :, None, :] - Y.P[iy][:, None, :, :]
    al = p * q / (p + q)
    pre = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
    T = al * (R * R).sum(-1)
    F = _boys(L, T)
    if omega > 0:  # erfc(omega r)/r
        s = omega * omega / (omega * omega + al)
        G = _boys(L, T * s)
        F = [F[m] - s ** (m + 0.5) * G[m] for m in range(L + 1)]
    r = {(0, 0, 0): [pre * (-2 * al) ** m * F[m] for m in range(L + 1)]}
    hs = _herm(L)
    for h in sorted(hs, key=sum):
        if h == (0, 0, 0):
            continue
        x = 0 if h[0] else (1 if h[1] else 2)
        h1 = tuple(v - (y == x) for y, v in enumerate(h))
        h2 = tuple(v - 2 * (y == x) for y, v in enumerate(h))
        r[h] = [R[..., x] * r[h1][m + 1] + ((h[x] - 1) * r[h2][m + 1] if h[x] > 1 else 0)
                for m in range(L + 1 - sum(h))]
    hb, hk = _herm(X.L), _herm(Y.L)
    n, kx, ky = T.shape
    M = torch.empty(n, kx, len(hb), ky, len(hk), dtype=torch.float64, device=T.device)
    for i, u in enumerate(hb):
        for j, w in enumerate(hk):
            M[:, :, i, :, j] = (-1) ** sum(w) * r[u[0] + w[0], u[1] + w[1], u[2] + w[2]][0]
    Hb = X.H[ix].permute(0, 2, 1, 3).reshape(n, -1, kx * len(hb))
    Hk = Y.H[iy].permute(0, 1, 3, 2).reshape(n, ky * len(hk), -1)
    return torch.bmm(torch.bmm(Hb, M.reshape(n, kx * len(hb), ky * len(hk))), Hk)


def _kind(s):
    return (s.l, bool(s.pure), s.nprim())


def _group(shells, quartets):
    """Quartet indices by the kinds of the four shells."""
    kinds = sorted({_kind(s) for s in shells})
    kid = np.array([kinds.index(_kind(s)) for s in shells])
    code = kid[quartets] @ (len(kinds) ** np.arange(3, -1, -1))
    order = np.argsort(code, kind="stable")
    cuts = np.flatnonzero(np.diff(code[order])) + 1
    return np.split(order, cuts)


def _cost(shells, groups, quartets, extra=0):
    c = 0.0
    for g in groups:
        s = [shells[i] for i in quartets[g[0]]]
        hb, hk = (len(_herm(s[i].l + s[i + 1].l + extra)) for i in (0, 2))
        c += len(g) * hb * hk * math.prod(x.nprim() for x in s)
    return c


def _blocks(shells, quartets, g, d=((0, 0, 0),) * 4, omega=0.0):
    """Yields (quartet indices, values n x nf1 x nf2 x nf3 x nf4) over one group in chunks."""
    q = quartets[g]
    X, ix = np.unique(q[:, :2], axis=0, return_inverse=True)
    Y, iy = np.unique(q[:, 2:], axis=0, return_inverse=True)
    bra = _Pairs([shells[i] for i in X[:, 0]], [shells[i] for i in X[:, 1]], d[0], d[1])
    ket = _Pairs([shells[i] for i in Y[:, 0]], [shells[i] for i in Y[:, 1]], d[2], d[3])
    per = bra.k * ket.k * (len(_herm(bra.L)) * len(_herm(ket.L)) + 6 * len(_herm(bra.L + ket.L)))
    step = max(1, int(2e8 // per))
    ix, iy = (torch.as_tensor(v.reshape(-1), device=_dev()) for v in (ix, iy))
    for k in range(0, len(g), step):
        v = _eri(bra, ket, ix[k:k + step], iy[k:k + step], omega)
        yield g[k:k + step], v.reshape(v.shape[0], *bra.nf, *ket.nf)


def _unit(c):
    """Derivative orders (per shell and direction) of coordinates in `c`."""
    d = [[0, 0, 0] for _ in range(4)]
    for k in c:
        d[k // 3][k % 3] += 1
    return tuple(tuple(x) for x in d)


def _coords(deriv):
    if deriv == 0:
        return [()]
    if deriv == 1:
        return [(k,) for k in range(12)]
    return [(i, j) for i in range(12) for j in range(i, 12)]


def _exact_list(shells, quartets, deriv):
    groups = _group(shells, quartets)
    if _cost(shells, groups, quartets, deriv) * len(_coords(deriv)) > EXACT_MOST:
        return None
    size = np.array([s.size() for s in shells], np.int64)
    nv = np.prod(size[quartets], axis=1)
    ns = len(_coords(deriv))
    off = np.concatenate([[0], np.cumsum(nv * ns)])
    out = torch.zeros(int(off[-1]), dtype=torch.float64, device=_dev())
    for g in groups:
        n1 = int(nv[g[0]])
        at = torch.as_tensor(off[g], device=_dev())
        ar = torch.arange(n1, device=_dev())
        for s, c in enumerate(_coords(deriv)):
            done = 0
            for idx, v in _blocks(shells, quartets, g, _unit(c)):
                m = len(idx)
                out[at[done:done + m, None] + s * n1 + ar] = v.reshape(m, -1)
                done += m
    return out.cpu().numpy()


def _exact_jk(bs, D, omega):
    if len(bs) > EXACT_SHELLS:
        return None
    q = _unique_quartets(len(bs))
    groups = _group(bs, q)
    if _cost(bs, groups, q) > EXACT_MOST:
        return None
    D = torch.as_tensor(D, device=_dev())
    J, K = torch.zeros_like(D), torch.zeros_like(D)
    bf = np.array(bs.shell2bf())
    N = D.shape[0]

    def fn(idx, k, n):
        return torch.as_tensor(bf[q[idx, k]], device=_dev())[:, None] + torch.arange(n, device=_dev())

    for g in groups:
        for idx, v in _blocks(bs, q, g, omega=omega):
            s = q[idx]
            deg = (np.where(s[:, 0] == s[:, 1], 1.0, 2.0) * np.where(s[:, 2] == s[:, 3], 1.0, 2.0) *
                   np.where((s[:, 0] == s[:, 2]) & (s[:, 1] == s[:, 3]), 1.0, 2.0))
            v = v * torch.as_tensor(deg, device=_dev())[:, None, None, None, None]
            f = [fn(idx, k, v.shape[k + 1]) for k in range(4)]
            for M, (x, y), (z, w), eq in ((J, (0, 1), (2, 3), "nabcd,ncd->nab"),
                                          (J, (2, 3), (0, 1), "nabcd,nab->ncd"),
                                          (K, (0, 2), (1, 3), "nabcd,nbd->nac"),
                                          (K, (1, 3), (0, 2), "nabcd,nac->nbd"),
                                          (K, (0, 3), (1, 2), "nabcd,nbc->nad"),
                                          (K, (1, 2), (0, 3), "nabcd,nad->nbc")):
                Dz = D[f[z][:, :, None], f[w][:, None, :]]
                r = torch.einsum(eq, v, Dz)
                M.view(-1).index_add_(0, (f[x][:, :, None] * N + f[y][:, None, :]).reshape(-1),
                                      r.reshape(-1))
    return {"J": ((J + J.T) / 4).cpu().numpy(), "K": ((K + K.T) / 8).cpu().numpy()}


def _exact_grad(bs, D, natoms):
    """Each of the four positions of a differentiated function gives the same sum."""
    ns = len(bs)
    if ns > EXACT_SHELLS // 2:
        return None
    i, j = np.tril_indices(ns)
    a, b = (v.reshape(-1) for v in np.meshgrid(np.arange(ns), np.arange(ns), indexing="ij"))
    q = np.stack([np.repeat(a, len(i)), np.repeat(b, len(i)), np.tile(i, ns * ns),
                  np.tile(j, ns * ns)], axis=1)
    groups = _group(bs, q)
    if 3 * _cost(bs, groups, q, 1) > EXACT_MOST:
        return None
    D = torch.as_tensor(D, device=_dev())
    bf, atom = np.array(bs.shell2bf()), np.array(bs.atom_of_shell)
    g2 = [torch.zeros(natoms, 3, dtype=torch.float64, device=_dev()) for _ in range(2)]
    for g in groups:
        for x in range(3):
            d = tuple(tuple(int(y == x and k == 0) for y in range(3)) for k in range(4))
            for idx, v in _blocks(bs, q, g, d):
                s = q[idx]
                v = v * torch.as_tensor(np.where(s[:, 2] == s[:, 3], 1.0, 2.0),
                                        device=_dev())[:, None, None, None, None]
                f = [torch.as_tensor(bf[s[:, k]], device=_dev())[:, None] +
                     torch.arange(v.shape[k + 1], device=_dev()) for k in range(4)]
                d2 = lambda y, z: D[f[y][:, :, None], f[z][:, None, :]]  # noqa: E731
                at = torch.as_tensor(atom[s[:, 0]], device=_dev())
                eJ = torch.einsum("nabcd,nab,ncd->n", v, d2(0, 1), d2(2, 3))
                eK = (torch.einsum("nabcd,nac,nbd->n", v, d2(0, 2), d2(1, 3)) +
                      torch.einsum("nabcd,nad,nbc->n", v, d2(0, 3), d2(1, 2))) / 2
                g2[0][:, x].index_add_(0, at, 2.0 * eJ)
                g2[1][:, x].index_add_(0, at, -1.0 * eK)
    return {"gJ": g2[0].cpu().numpy(), "gK": g2[1].cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "engine":
        sh = _engine_shells(case, seed)
        v = _exact_list(sh, np.arange(4, dtype=np.int32)[None], case["deriv"])
        v = v.reshape([-1] + [s.size() for s in sh])
        return v if case["deriv"] else v[0]
    if kind in ("batch", "df"):
        bs, q = _list_inputs(case, seed)
        v = _exact_list(bs, q, case.get("deriv", 0))
        return None if v is None else {"sets": v, "null": None}
    bs = lg.BasisSet(case["basis"], _cluster(case["waters"], seed))
    D = _density(case, bs.nbf, seed)
    if kind == "grad":
        return _exact_grad(bs, D, 3 * case["waters"])
    return _exact_jk(bs, D, case["omega"])
