"""The J/K calls whose speed is measured, with their inputs and exact results.

Every case goes through the package's public entry points: IntBox.coulomb and
exchange (and their Multi, Grad and eriJ forms) on host tensors, the pair list
and one-electron set-up of a new geometry, and the device entry points an SCF
over many molecules uses. Molecules are water clusters and all-trans alkanes,
the basis sets those shipped with the package. The seed moves the atoms (bond
noise) and draws the densities: sums over localised orbitals, so that the
density decays with distance as that of a converged closed-shell molecule does
(the decay decides how many quartets the screens keep).
"""
import math

import numpy as np
import torch

import lightspeed_b200 as ls
from lightspeed_b200 import geometry

BOHR = 1.0 / 0.52917720859
KINDS = ("jk", "multi", "grad", "setup", "eri", "lockstep")


def _case(name, kind, system, n, basis, precision="fp64", thre=1.0e-14, thredp=1.0e-6, omega=-1.0, merge=False,
          ndens=1):
    c = dict(kind=kind, system=system, n=n, basis=basis, precision=precision, thre=thre, thredp=thredp, omega=omega,
             merge=merge, ndens=ndens)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one Fock build of a single small molecule: the smallest call, where launches and latency count
        _case("jk_water1_631gs", "jk", "water", 1, "6-31gs"),
        # an ordinary cluster in a Cartesian split-valence basis, all FP64
        _case("jk_water8_631gs", "jk", "water", 8, "6-31gs"),
        # a medium molecule in a correlation-consistent basis, the default mixed precision
        _case("jk_alkane10_ccpvdz_mixed", "jk", "alkane", 10, "cc-pvdz", "mixed", thredp=1.0e-5),
        # the same family larger, FP64 over the exact quartet set
        _case("jk_alkane20_ccpvdz", "jk", "alkane", 20, "cc-pvdz"),
        # the largest build: mixed precision, K over merged s exponents (the opt-in mode for large molecules)
        _case("jk_alkane40_ccpvdz_mixed", "jk", "alkane", 40, "cc-pvdz", "mixed", thredp=1.0e-5, merge=True),
        # response-type work: a batch of non-symmetric transition densities, attenuated operator
        _case("multi_water8_16dens_erf", "multi", "water", 8, "6-31gs", "mixed", thredp=1.0e-5, omega=0.3, ndens=16),
        # f shells in a triple-zeta basis
        _case("jk_water4_ccpvtz", "jk", "water", 4, "cc-pvtz", thre=1.0e-12),
        # nuclear gradients: f shells on a dimer, and a medium alkane
        _case("grad_water2_ccpvtz", "grad", "water", 2, "cc-pvtz", thre=1.0e-12),
        _case("grad_alkane10_ccpvdz", "grad", "alkane", 10, "cc-pvdz", thre=1.0e-12),
        # what every new geometry needs before its first Fock build: pair list, S, T and V
        _case("setup_alkane20_ccpvdz", "setup", "alkane", 20, "cc-pvdz"),
        # active-space integrals: J builds of many orbital pairs at once
        _case("eri_water8_active8", "eri", "water", 8, "6-31gs", thre=1.0e-12, ndens=8),
        # one lockstep SCF iteration of many small molecules on device tensors over several streams
        _case("lockstep_water12_631gs", "lockstep", "water", 12, "6-31gs", thre=1.0e-12),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(("jk", "jk", "jk", "multi", "grad", "setup", "eri", "lockstep"))
    prec = rng.choice(("fp64", "mixed"))
    omega = rng.choice((-1.0, -1.0, round(rng.uniform(0.1, 1.0), 3)))
    thre = rng.choice((1.0e-14, 1.0e-12, 1.0e-10))
    thredp = rng.choice((1.0e-6, 1.0e-5, 1.0e-4))
    system = rng.choice(("water", "alkane"))
    basis = rng.choice(("sto-3g", "6-31gs", "6-31gs", "cc-pvdz", "cc-pvdz", "cc-pvtz"))
    if kind == "multi":
        basis = rng.choice(("sto-3g", "6-31gs", "cc-pvdz"))
        n = _log_int(rng, 1, 8 if system == "water" else 4)
        return _case(None, kind, system, n, basis, prec, thre, thredp, omega, False, rng.randint(2, 17))
    if kind == "grad":
        n = _log_int(rng, 1, {"cc-pvtz": 2, "cc-pvdz": 6}.get(basis, 8))
        return _case(None, kind, system, n, basis, "fp64", thre)
    if kind == "setup":
        return _case(None, kind, system, _log_int(rng, 1, 4 if basis == "cc-pvtz" else 20), basis, "fp64", thre)
    if kind == "eri":
        basis = rng.choice(("sto-3g", "6-31gs", "cc-pvdz"))
        return _case(None, kind, system, _log_int(rng, 1, 8), basis, prec, thre, thredp, omega, False,
                     rng.randint(2, 8))
    if kind == "lockstep":
        return _case(None, kind, "water", _log_int(rng, 2, 12), rng.choice(("sto-3g", "6-31gs")), "fp64", thre)
    n = _log_int(rng, 1, {"cc-pvtz": 4, "sto-3g": 30}.get(basis, 16 if system == "water" else 24))
    return _case(None, kind, system, n, basis, prec, thre, thredp, omega, rng.random() < 0.3)


# ---- inputs -----------------------------------------------------------------------


def _molecule(system, n, rng):
    if system == "water":
        return geometry.water_cluster(n, seed=int(rng.integers(1 << 30)), noise=(0.03, 3.0))
    mol = geometry.alkane(n)
    xyz = mol.xyz + rng.uniform(-0.02, 0.02, size=(mol.natom, 3)) * BOHR
    return ls.Molecule.from_arrays([a.symbol for a in mol.atoms], xyz, name=mol.name)


def _ao_centres(bas):
    """Position of each atomic orbital."""
    R = np.zeros((bas.nao, 3))
    for p in bas.primitives:
        R[p.aoIdx:p.aoIdx + p.nao] = (p.x, p.y, p.z)
    return R


def _occupied_density(mol, bas, rng):
    """sum of one localised orbital per electron pair: normal coefficients that decay
    with the distance from a heavy atom. The length, 1.7 Bohr, was chosen so that the
    screens keep about as many quartets as at a converged RHF density."""
    R = _ao_centres(bas)
    heavy = [a for a in range(mol.natom) if mol.Z[a] > 1.5] or [0]
    nocc = int(mol.nuclear_charge) // 2
    C = rng.standard_normal((bas.nao, nocc))
    for i in range(nocc):
        d = np.linalg.norm(R - mol.xyz[heavy[i % len(heavy)]], axis=1)
        C[:, i] *= np.exp(-d / 1.7)
    C *= 0.9 / np.linalg.norm(C, axis=0)
    return C @ C.T


def _transition_density(bas, rng):
    X = rng.standard_normal((bas.nao, 10)) / math.sqrt(bas.nao)
    Y = rng.standard_normal((bas.nao, 10)) / math.sqrt(bas.nao)
    return X @ Y.T


def _inputs(case, seed):
    """Molecule(s), basis/bases and the numpy arrays of one case."""
    rng = np.random.default_rng([seed, 20])
    kind = case["kind"]
    sizes = range(1, case["n"] + 1) if kind == "lockstep" else (case["n"],)
    systems = []
    for n in sizes:
        mol = _molecule(case["system"], n, rng)
        bas = ls.Basis.from_gbs_file(mol, case["basis"])
        if kind == "multi":
            arrays = [_transition_density(bas, rng) for _ in range(case["ndens"])]
        elif kind == "eri":
            q, _ = np.linalg.qr(rng.standard_normal((bas.nao, min(case["ndens"], bas.nao))))
            arrays = [q]
        elif kind == "setup":
            arrays = [mol.xyzZ]
        else:
            arrays = [_occupied_density(mol, bas, rng)]
        systems.append((mol, bas, arrays))
    return systems


def prepare(case, seed):
    systems = _inputs(case, seed)
    st = dict(case=case, res=ls.ResourceList.build(), ewald=ls.Ewald([1.0], [case["omega"]]))
    mol, bas, arrays = systems[0]
    if case["kind"] == "lockstep":
        st["streams"] = [ls.Stream() for _ in range(4)]
        st["torch_streams"] = [torch.cuda.ExternalStream(x.stream_handle()) for x in st["streams"]]
        st["pairs"] = [ls.PairList.build_schwarz(b, b, True, case["thre"]) for _, b, _ in systems]
        st["D"] = [torch.tensor(a[0], device="cuda") for _, _, a in systems]
        st["JK"] = [torch.zeros((2,) + tuple(d.shape), dtype=torch.float64, device="cuda") for d in st["D"]]
    else:
        st["basis"] = bas
        st["in"] = [ls.Tensor.array(np.ascontiguousarray(a)) for a in arrays]
        if case["kind"] != "setup":
            st["pairs"] = ls.PairList.build_schwarz(bas, bas, True, case["thre"])
    return st


def run(st):
    case, res, ew = st["case"], st["res"], st["ewald"]
    kind, thre, thredp = case["kind"], case["thre"], case["thredp"]
    prec = ls.PREC_MIXED if case["precision"] == "mixed" else ls.PREC_FP64
    ls.set_precision(prec)
    ls.set_merge(case["merge"])
    if kind == "lockstep":
        cur = torch.cuda.current_stream()
        for x, s in zip(st["streams"], st["torch_streams"]):
            x.set_precision(prec)
        for jk in st["JK"]:
            jk.zero_()
        for s in st["torch_streams"]:
            s.wait_stream(cur)
        for k, (pl, d, jk) in enumerate(zip(st["pairs"], st["D"], st["JK"])):
            x = st["streams"][k % len(st["streams"])]
            x.coulomb_device(ew, pl, pl, [d.data_ptr()], [jk[0].data_ptr()], thre, thredp)
            x.exchange_device(ew, pl, pl, [d.data_ptr()], True, [jk[1].data_ptr()], thre, thredp)
        for s in st["torch_streams"]:
            cur.wait_stream(s)
        return st["JK"]
    if kind == "setup":
        pl = ls.PairList.build_schwarz(st["basis"], st["basis"], True, thre)
        S = ls.IntBox.overlap(res, pl)
        T = ls.IntBox.kinetic(res, pl)
        V = ls.IntBox.potential(res, ew, pl, st["in"][0])
        return [S.np, T.np, V.np]
    pl, D = st["pairs"], st["in"]
    if kind == "jk":
        J = ls.IntBox.coulomb(res, ew, pl, pl, D[0], thre, thredp)
        K = ls.IntBox.exchange(res, ew, pl, pl, D[0], True, thre, thredp)
        return [J.np, K.np]
    if kind == "multi":
        J = ls.IntBox.coulombMulti(res, ew, pl, pl, D, thre, thredp)
        K = ls.IntBox.exchangeMulti(res, ew, pl, pl, D, False, thre, thredp)
        return [t.np for t in J + K]
    if kind == "grad":
        GJ = ls.IntBox.coulombGrad(res, ew, pl, D[0], D[0], thre, thredp)
        GK = ls.IntBox.exchangeGrad(res, ew, pl, D[0], D[0], True, True, True, thre, thredp)
        return [GJ.np, GK.np]
    C = D[0]
    return ls.IntBox.eriJ(res, ew, pl, pl, C, C, C, C, thre, thredp).np


def tolerance(case):
    # FP64: sums in another order (1e-14 seen), and single quartets that a rounding of their estimate
    # moves across a screen (each at most thre); the screens themselves are part of the call
    fp64 = {1.0e-14: 1.0e-11, 1.0e-12: 1.0e-10, 1.0e-10: 1.0e-9}[case["thre"]]
    if case["precision"] == "mixed":
        # quartets below thredp may be FP32: up to 2e-11, 1.2e-9 and 1.7e-9 from the exact result were seen
        return {"rel": max(fp64, {1.0e-6: 1.0e-10, 1.0e-5: 5.0e-9, 1.0e-4: 1.0e-8}[case["thredp"]])}
    return {"rel": fp64}


# ---- work: quartets that pass the screens, counted from the Schwarz bounds -----------


def _ncart(L):
    return (L + 1) * (L + 2) // 2


def _nherm(L):
    return (L + 1) * (L + 2) * (L + 3) // 6


def _j_flops(LB, LK):
    L = LB + LK
    return 33.0 + 3.0 * L + 2.0 * sum(_nherm(L - n) for n in range(L + 1)) + 2.0 * _nherm(LB) * _nherm(LK)


def _k_flops(L1, L2, L3, L4, deriv):
    nr = (L1 + L2 + L3 + L4 + deriv) // 2 + 1
    n1d = 3.0 * (L1 + L2 + 1 + deriv) * (L3 + L4 + 1 + deriv) + 3.0 * (L1 + 1 + deriv) * (L2 + 1 + deriv) * \
        (L3 + 1 + deriv) * (L4 + 1)
    nc = _ncart(L1) * _ncart(L2) * _ncart(L3) * _ncart(L4)
    return 40.0 + nr * (28.0 + 2.0 * n1d + (24.0 if deriv else 4.0) * nc)


def _bounds(prims):
    c = np.array([p[0] for p in prims])
    e = np.array([p[1] for p in prims])
    R = np.array([p[2] for p in prims])
    L = np.array([p[3] for p in prims])
    r2 = ((R[:, None] - R[None]) ** 2).sum(-1)
    p = e[:, None] + e[None]
    return np.abs(c[:, None] * c[None]) * np.exp(-e[:, None] * e[None] / p * r2) * 2.0 ** 0.25 * \
        (math.pi / p) ** 1.25, L


def _system_work(case, mol, bas, arrays):
    kind, thre = case["kind"], case["thre"]
    deriv = 1 if kind == "grad" else 0
    prims = [(p.c, p.e, (p.x, p.y, p.z), p.L, p.aoIdx, p.nao) for p in bas.primitives]
    B, L = _bounds(prims)
    nao, npr = bas.nao, len(prims)
    keep = B > thre
    npair = int(np.tril(keep).sum())
    lo = np.tril(keep)
    if kind == "setup":
        nherm = np.array([_nherm(l) for l in range(7)])
        ii, jj = np.nonzero(lo)
        H = float(nherm[L[ii] + L[jj]].sum())
        return {"bytes": 8.0 * 3 * nao * nao + 24.0 * npair, "flops": (60.0 * npair + 8.0 * H) * (2 + mol.natom)}
    if kind == "eri":
        C = arrays[0]
        D = np.abs(C).max(1)[:, None] * np.abs(C).max(1)[None]
        ndens = C.shape[1] * (C.shape[1] + 1) // 2
    else:
        D = np.abs(np.stack(arrays)).max(0)
        ndens = len(arrays)
    ao = np.array([p[4] for p in prims])
    Dm = np.zeros((npr, npr))
    width = np.array([p[5] for p in prims])
    for a in range(width.max()):
        for b in range(width.max()):
            ia, ib = np.minimum(ao + a, ao + width - 1), np.minimum(ao + b, ao + width - 1)
            Dm = np.maximum(Dm, D[np.ix_(ia, ib)])
    Dm = np.maximum(Dm, Dm.T)
    ii, jj = np.nonzero(lo)
    cls, b = L[ii] + L[jj], B[ii, jj]
    flops = 0.0
    per = float(ndens)
    for LK in range(cls.max() + 1):
        k = np.sort((b * Dm[ii, jj])[cls == LK])
        for LB in range(cls.max() + 1):
            bb = b[cls == LB]
            if len(k) and len(bb):
                n = float((len(k) - np.searchsorted(k, thre / bb)).sum())
                shared = _j_flops(LB + deriv, LK) - 2.0 * _nherm(LB + deriv) * _nherm(LK)
                flops += n * (shared + per * 2.0 * _nherm(LB + deriv) * _nherm(LK))
    if kind != "eri":
        # sampled (prim2, prim4) tasks, over distinct s exponents when they are merged
        sel = np.ones(npr, bool)
        if case["merge"]:
            seen = set()
            for q, pr in enumerate(prims):
                key = (pr[1], pr[2])
                sel[q] = pr[3] != 0 or key not in seen
                seen.add(key)
        idx = np.nonzero(sel)[0]
        Bs, Ls, Dk = np.where(keep, B, 0.0)[np.ix_(idx, idx)], L[idx], Dm[np.ix_(idx, idx)]
        m = len(idx)
        rows = [[np.sort(Bs[q][(Ls == l) & (Bs[q] > 0)]) for l in range(Ls.max() + 1)] for q in range(m)]
        r = np.random.default_rng(1)
        ns = min(m * m, 3000)
        pick = r.permutation(m * m)[:ns] if m * m <= 4000000 else r.integers(m * m, size=ns)
        tot = 0.0
        for q in pick:
            q2, q4 = divmod(int(q), m)
            for L1, r1 in enumerate(rows[q2]):
                for L3, r3 in enumerate(rows[q4]):
                    if len(r1) and len(r3) and r1[-1] * r3[-1] * Dk[q2, q4] >= thre:
                        n = float((len(r3) - np.searchsorted(r3, thre / (r1 * Dk[q2, q4]))).sum())
                        f = _k_flops(L1, int(Ls[q2]), L3, int(Ls[q4]), deriv)
                        nr = (L1 + Ls[q2] + L3 + Ls[q4] + deriv) // 2 + 1
                        con = nr * 2.0 * _ncart(L1) * _ncart(Ls[q2]) * _ncart(L3) * _ncart(Ls[q4])
                        tot += n * (f + (per - 1.0) * con)
        half = 1.0 if kind == "multi" else 0.5    # a symmetric density needs prim2 <= prim4 only
        flops += tot * half * m * m / ns
    out = {"grad": 2 * 3 * mol.natom, "eri": arrays[0].shape[1] ** 4}.get(kind, 2 * ndens * nao * nao)
    return {"bytes": 8.0 * (ndens * nao * nao + out) + 32.0 * npair, "flops": flops}


def work(case):
    tot = {"bytes": 0.0, "flops": 0.0}
    for s in _inputs(case, 0):
        w = _system_work(case, *s)
        tot = {k: tot[k] + w[k] for k in tot}
    return tot


# ---- exact results: McMurchie-Davidson integrals in plain FP64 torch, no screening ----


def _cart(L):
    return [(L - i, i - j, j) for i in range(L + 1) for j in range(i + 1)]


def _pure(L):
    """Real solid harmonics (m = 0, 1c, 1s, 2c, 2s, ...) over the Cartesian components."""
    s = math.sqrt
    terms = {
        0: [{(0, 0, 0): 1.0}],
        1: [{(0, 0, 1): 1.0}, {(1, 0, 0): 1.0}, {(0, 1, 0): 1.0}],
        2: [{(0, 0, 2): 1.0, (2, 0, 0): -0.5, (0, 2, 0): -0.5}, {(1, 0, 1): s(3)}, {(0, 1, 1): s(3)},
            {(2, 0, 0): s(3) / 2, (0, 2, 0): -s(3) / 2}, {(1, 1, 0): s(3)}],
        3: [{(0, 0, 3): 1.0, (2, 0, 1): -1.5, (0, 2, 1): -1.5},
            {(1, 0, 2): 2 * s(1.5), (3, 0, 0): -s(1.5) / 2, (1, 2, 0): -s(1.5) / 2},
            {(0, 1, 2): 2 * s(1.5), (2, 1, 0): -s(1.5) / 2, (0, 3, 0): -s(1.5) / 2},
            {(2, 0, 1): s(15) / 2, (0, 2, 1): -s(15) / 2}, {(1, 1, 1): s(15)},
            {(3, 0, 0): s(2.5) / 2, (1, 2, 0): -1.5 * s(2.5)}, {(2, 1, 0): 1.5 * s(2.5), (0, 3, 0): -s(2.5) / 2}],
    }[L]
    return np.array([[t.get(c, 0.0) for c in _cart(L)] for t in terms])


_BOYS = {}


def _boys_grid(dev):
    """F_m on a grid of step 0.05 up to T = 45 by the (all positive) series."""
    if dev not in _BOYS:
        T = np.arange(0, 901) * 0.05
        out = []
        for m in range(22):
            term = np.ones_like(T) / (2 * m + 1)
            tot = term.copy()
            for k in range(1, 260):
                term = term * 2.0 * T / (2 * m + 2 * k + 1)
                tot += term
            out.append(np.exp(-T) * tot)
        _BOYS[dev] = torch.tensor(np.stack(out, 1), device=dev)
    return _BOYS[dev]


def _boys_values(L, T):
    """[F_0 .. F_L] at T."""
    grid = _boys_grid(T.device)
    big = T > 44.9
    Ts = torch.where(big, torch.zeros_like(T), T)
    k = (Ts * 20.0 + 0.5).to(torch.int64)
    d = k.to(T.dtype) * 0.05 - Ts
    top = grid[:, L + 7][k]
    for j in range(6, -1, -1):
        top = grid[:, L + j][k] + top * d / (j + 1)
    F = [None] * L + [top]
    e = torch.exp(-T)
    for m in range(L - 1, -1, -1):
        F[m] = (2.0 * Ts * F[m + 1] + e) / (2 * m + 1)
    a = 0.5 * torch.sqrt(math.pi / T.clamp(min=1.0))
    for m in range(L + 1):
        F[m] = torch.where(big, a, F[m])
        a = ((2 * m + 1) * a - e) / (2.0 * T.clamp(min=1.0))
    return F


class _Boys(torch.autograd.Function):
    @staticmethod
    def forward(ctx, T, L):
        F = _boys_values(L + 1, T)
        ctx.save_for_backward(*F[1:])
        return torch.stack(F[:L + 1])

    @staticmethod
    def backward(ctx, g):
        return -sum(gm * F for gm, F in zip(g, ctx.saved_tensors)), None


def _hermite_coulomb(L, alpha, PQ, pref):
    """R_tuv, |tuv| <= L, of the Coulomb interaction with exponent alpha times pref."""
    X = PQ.unbind(-1)
    F = _Boys.apply(alpha * (PQ * PQ).sum(-1), L)
    R = {(m, 0, 0, 0): pref * (-2.0 * alpha) ** m * F[m] for m in range(L + 1)}
    for N in range(1, L + 1):
        for m in range(L - N + 1):
            for t in _cart(N):
                d = next(k for k in range(3) if t[k])
                one = tuple(t[k] - (k == d) for k in range(3))
                v = X[d] * R[(m + 1,) + one]
                if one[d]:
                    v = v + one[d] * R[(m + 1,) + tuple(one[k] - (k == d) for k in range(3))]
                R[(m,) + t] = v
    return {k[1:]: v for k, v in R.items() if k[0] == 0}


def _herm(L):
    return [t for N in range(L + 1) for t in _cart(N)]


class _ShellType:
    """All contracted shells with one angular momentum and contraction length."""

    def __init__(self, L, K, shells, dev):
        f = dict(dtype=torch.float64, device=dev)
        self.L, self.n = L, len(shells)
        self.c = torch.tensor([[p.c for p in s] for s in shells], **f)
        self.e = torch.tensor([[p.e for p in s] for s in shells], **f)
        self.atom = torch.tensor([s[0].atomIdx for s in shells], device=dev)
        pure = shells[0][0].is_pure and L > 0
        self.T = torch.tensor(_pure(L) if pure else np.eye(_ncart(L)), **f)
        w = self.T.shape[0]
        self.w = w
        self.ao = torch.tensor([[s[0].aoIdx + k for k in range(w)] for s in shells], device=dev).reshape(-1)


def _shell_types(bas, dev):
    shells, groups = {}, {}
    for p in bas.primitives:
        shells.setdefault(p.shellIdx, []).append(p)
    for s in shells.values():
        groups.setdefault((s[0].L, len(s)), []).append(s)
    return [_ShellType(L, K, g, dev) for (L, K), g in sorted(groups.items())]


def _pair_data(a, b, ia, ib, xyz):
    """Exponents, centres and Hermite coefficients E[pair, a, b, K, t] of shell pairs."""
    e1, e2 = a.e[ia][:, :, None], b.e[ib][:, None, :]
    p = e1 + e2
    A, B = xyz[a.atom[ia]], xyz[b.atom[ib]]
    P = (e1[..., None] * A[:, None, None] + e2[..., None] * B[:, None, None]) / p[..., None]
    kab = a.c[ia][:, :, None] * b.c[ib][:, None, :] * torch.exp(-e1 * e2 / p * ((A - B) ** 2).sum(-1)[:, None, None])
    h = 0.5 / p
    E = []
    for d in range(3):
        XA, XB = P[..., d] - A[:, None, None, d], P[..., d] - B[:, None, None, d]
        tab = {(0, 0): [torch.ones_like(p)]}
        for i in range(a.L + 1):
            for j in range(b.L + 1):
                if i + j == 0:
                    continue
                src, X = (tab[(i - 1, j)], XA) if i else (tab[(i, j - 1)], XB)
                z = torch.zeros_like(p)
                get = lambda t: src[t] if 0 <= t < len(src) else z
                tab[(i, j)] = [X * get(t) + h * get(t - 1) + (t + 1) * get(t + 1) for t in range(i + j + 1)]
        E.append(tab)
    ca, cb, hm = _cart(a.L), _cart(b.L), _herm(a.L + b.L)
    z = torch.zeros_like(p)
    out = []
    for x in ca:
        for y in cb:
            for t in hm:
                if all(t[d] <= x[d] + y[d] for d in range(3)):
                    out.append(kab * E[0][(x[0], y[0])][t[0]] * E[1][(x[1], y[1])][t[1]] * E[2][(x[2], y[2])][t[2]])
                else:
                    out.append(z)
    np_, K = p.shape[0], p.shape[1] * p.shape[2]
    out = torch.stack(out, -1).reshape(np_, K, len(ca), len(cb), len(hm))
    out = torch.einsum("nkabt,xa,yb->nxykt", out, a.T, b.T)
    return p.reshape(np_, K), P.reshape(np_, K, 3), out.reshape(np_, a.w * b.w, K, len(hm))


def _eri_block(bra, ket, Lb, Lk, omega):
    """(ab|cd) of all bra and ket shell pairs: [nb, ab, nk, cd]."""
    p, P, Eb = bra
    q, Q, Ek = ket
    nb, Kb, nk, Kk = p.shape[0], p.shape[1], q.shape[0], q.shape[1]
    pf, qf = p.reshape(-1, 1), q.reshape(1, -1)
    rho = pf * qf / (pf + qf)
    pref = 2.0 * math.pi ** 2.5 / (pf * qf * torch.sqrt(pf + qf))
    if omega > 0:
        s = omega * omega / (rho + omega * omega)
        pref, rho = pref * torch.sqrt(s), rho * s
    R = _hermite_coulomb(Lb + Lk, rho, P.reshape(-1, 1, 3) - Q.reshape(1, -1, 3), pref)
    hb, hk = _herm(Lb), _herm(Lk)
    nab, ncd = Eb.shape[1], Ek.shape[1]
    El = Eb.reshape(nb, nab, Kb * len(hb))
    half = []
    for u in hk:
        Ru = torch.stack([R[tuple(t[d] + u[d] for d in range(3))] for t in hb], 1)   # [nb*Kb, H, nk*Kk]
        sign = -1.0 if sum(u) % 2 else 1.0
        half.append(sign * torch.bmm(El, Ru.reshape(nb, Kb * len(hb), nk * Kk)))
    X = torch.stack(half, -1).reshape(nb * nab, nk, Kk * len(hk)).transpose(0, 1)     # [nk, nb*ab, K*H]
    Y = torch.bmm(X, Ek.reshape(nk, ncd, Kk * len(hk)).transpose(1, 2))
    return Y.reshape(nk, nb, nab, ncd).permute(1, 2, 0, 3)


def _blocks(types, xyz, omega, limit=3.0e7):
    """The integrals over every quadruple of shell types (type 1 <= type 2, type 3 <= type 4)
    in pieces (some shells 1, all 2 | some shells 3, all 4): function indices of 1, 2, 3, 4
    and [n1, n2, n3, n4]."""
    dev = xyz.device
    pairs = [(a, b) for k, a in enumerate(types) for b in types[k:]]
    for ta, tb in pairs:
        for tc, td in pairs:
            Lb, Lk = ta.L + tb.L, tc.L + td.L
            Kb, Kk = ta.c.shape[1] * tb.c.shape[1], tc.c.shape[1] * td.c.shape[1]
            cost = float(tb.n * Kb * Kk * (_nherm(Lb + Lk) * (Lb + Lk + 2) / 2 + 12 + _nherm(Lb) * _nherm(Lk)))
            n3 = max(1, min(tc.n, int(limit / (cost * td.n))))
            n1 = max(1, min(ta.n, int(limit / (cost * td.n * n3))))
            for i in range(0, ta.n, n1):
                sa = torch.arange(i, min(i + n1, ta.n), device=dev)
                ia, ib = sa.repeat_interleave(tb.n), torch.arange(tb.n, device=dev).repeat(len(sa))
                bra = _pair_data(ta, tb, ia, ib, xyz)
                for k in range(0, tc.n, n3):
                    sc = torch.arange(k, min(k + n3, tc.n), device=dev)
                    ic, id_ = sc.repeat_interleave(td.n), torch.arange(td.n, device=dev).repeat(len(sc))
                    ket = _pair_data(tc, td, ic, id_, xyz)
                    I = _eri_block(bra, ket, Lb, Lk, omega)
                    I = I.reshape(len(sa), tb.n, ta.w, tb.w, len(sc), td.n, tc.w, td.w)
                    I = I.permute(0, 2, 1, 3, 4, 6, 5, 7).reshape(len(sa) * ta.w, tb.n * tb.w, len(sc) * tc.w,
                                                                 td.n * td.w)
                    yield (ta.ao.reshape(ta.n, -1)[sa].reshape(-1), tb.ao, tc.ao.reshape(tc.n, -1)[sc].reshape(-1),
                           td.ao, I, ta is not tb, tc is not td)


def _orders(block):
    """The block and its transposes in 1, 2 and in 3, 4 that _blocks leaves out."""
    a1, a2, a3, a4, I, flip12, flip34 = block
    out = [(a1, a2, a3, a4, I)]
    if flip12:
        out.append((a2, a1, a3, a4, I.transpose(0, 1)))
    if flip34:
        out += [(b1, b2, a4, a3, X.transpose(2, 3)) for b1, b2, _, _, X in list(out)]
    return out


def _one_electron(types, xyz, Z, nao, omega):
    dev = xyz.device
    S, T, V = (torch.zeros(nao, nao, dtype=torch.float64, device=dev) for _ in range(3))
    for ta in types:
        for tb in types:
            ia = torch.arange(ta.n, device=dev).repeat_interleave(tb.n)
            ib = torch.arange(tb.n, device=dev).repeat(ta.n)
            put = lambda M, x: M.index_put_((ta.ao[:, None], tb.ao[None]), x.reshape(ta.n, tb.n, ta.w, tb.w).permute(
                0, 2, 1, 3).reshape(ta.n * ta.w, tb.n * tb.w))
            p, P, E = _pair_data(ta, tb, ia, ib, xyz)
            put(S, torch.einsum("nxk,nk->nx", E[..., 0], (math.pi / p) ** 1.5))
            # T = -1/2 d^2/dr^2 of shell b: overlaps with the exponents of b raised and lowered by two
            put(T, _kinetic(ta, tb, ia, ib, xyz))
            acc = 0.0
            for C, z in zip(xyz, Z):
                s = omega * omega / (p + omega * omega) if omega > 0 else torch.ones_like(p)
                R = _hermite_coulomb(ta.L + tb.L, p * s, P - C, -z * 2.0 * math.pi / p * torch.sqrt(s))
                acc = acc + torch.einsum("nxkt,nkt->nx", E, torch.stack([R[t] for t in _herm(ta.L + tb.L)], -1))
            put(V, acc)
    return S, T, V


def _kinetic(a, b, ia, ib, xyz):
    e1, e2 = a.e[ia][:, :, None], b.e[ib][:, None, :]
    p = e1 + e2
    A, B = xyz[a.atom[ia]], xyz[b.atom[ib]]
    kab = a.c[ia][:, :, None] * b.c[ib][:, None, :] * torch.exp(-e1 * e2 / p * ((A - B) ** 2).sum(-1)[:, None, None])
    s1 = []
    for d in range(3):
        Pd = (e1 * A[:, None, None, d] + e2 * B[:, None, None, d]) / p
        XA, XB, h = Pd - A[:, None, None, d], Pd - B[:, None, None, d], 0.5 / p
        z = torch.zeros_like(p)
        s = {(0, 0): torch.sqrt(math.pi / p)}
        for i in range(a.L + 1):
            for j in range(b.L + 3):
                if i + j == 0:
                    continue
                if j:
                    s[(i, j)] = XB * s[(i, j - 1)] + h * (i * s.get((i - 1, j - 1), z) + (j - 1) * s.get((i, j - 2), z))
                else:
                    s[(i, j)] = XA * s[(i - 1, j)] + h * ((i - 1) * s.get((i - 2, j), z))
        t = {}
        for i in range(a.L + 1):
            for j in range(b.L + 1):
                v = 4.0 * e2 * e2 * s[(i, j + 2)] - 2.0 * e2 * (2 * j + 1) * s[(i, j)]
                t[(i, j)] = -0.5 * (v + (j * (j - 1) * s[(i, j - 2)] if j > 1 else 0.0))
        s1.append((s, t))
    rows = []
    for x in _cart(a.L):
        for y in _cart(b.L):
            k = [(x[d], y[d]) for d in range(3)]
            (sx, tx), (sy, ty), (sz, tz) = s1
            v = tx[k[0]] * sy[k[1]] * sz[k[2]] + sx[k[0]] * ty[k[1]] * sz[k[2]] + sx[k[0]] * sy[k[1]] * tz[k[2]]
            rows.append((kab * v).sum((1, 2)))
    M = torch.stack(rows, -1).reshape(-1, _ncart(a.L), _ncart(b.L))
    return torch.einsum("nab,xa,yb->nxy", M, a.T, b.T).reshape(M.shape[0], -1)


def _exact_seconds(case, bas):
    """Roughly how long the exact result of one system takes on the GPU: a fixed time per
    block of shell types, and the integrals over all primitive quartets."""
    deriv = int(case["kind"] == "grad")
    types = len({(p.L, n) for p, n in _contractions(bas)})
    elements = float(sum(_nherm(p.L + 1 + deriv) for p in bas.primitives)) ** 4
    fixed = (types * (types + 1) / 2) ** 2 * 0.005 * (4.0 if bas.max_L > 2 else 1.0) * (3.5 if deriv else 1.0)
    return fixed + 1.2e-12 * elements * (6.0 if deriv else 1.0) * (1.0 + case["ndens"] / 8.0)


def _contractions(bas):
    n = {}
    for p in bas.primitives:
        n[p.shellIdx] = n.get(p.shellIdx, 0) + 1
    return [(p, n[p.shellIdx]) for p in bas.primitives]


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    systems = _inputs(case, seed)
    kind, omega = case["kind"], case["omega"]
    if kind != "setup" and sum(_exact_seconds(case, b) for _, b, _ in systems) > 19.5:
        return None
    out = []
    for mol, bas, arrays in systems:
        types = _shell_types(bas, dev)
        xyz = torch.tensor(mol.xyz, device=dev, requires_grad=kind == "grad")
        if kind == "setup":
            return [x.cpu().numpy() for x in _one_electron(types, xyz, mol.Z, bas.nao, omega)]
        Ds = [torch.tensor(a, device=dev) for a in arrays]
        if kind == "eri":
            C, n = Ds[0], Ds[0].shape[1]
            I4 = torch.zeros(n, n, n, n, dtype=torch.float64, device=dev)
            for block in _blocks(types, xyz, omega):
                for a1, a2, a3, a4, I in _orders(block):
                    x = torch.einsum("abcd,ai,bj->ijcd", I, C[a1], C[a2])
                    I4 += torch.einsum("ijcd,ck,dl->ijkl", x, C[a3], C[a4])
            return I4.cpu().numpy()
        if kind == "grad":
            D = Ds[0]
            GJ, GK = torch.zeros_like(xyz), torch.zeros_like(xyz)
            for block in _blocks(types, xyz, omega, limit=1.0e7):
                EJ = EK = 0.0
                for a1, a2, a3, a4, I in _orders(block):
                    EJ = EJ + torch.einsum("abcd,ab,cd->", I, D[a1][:, a2], D[a3][:, a4])
                    EK = EK + torch.einsum("abcd,ac,bd->", I, D[a1][:, a3], D[a2][:, a4])
                GJ += torch.autograd.grad(EJ, xyz, retain_graph=True)[0]
                GK += torch.autograd.grad(EK, xyz)[0]
            return [GJ.detach().cpu().numpy(), GK.detach().cpu().numpy()]
        J = [torch.zeros_like(D) for D in Ds]
        K = [torch.zeros_like(D) for D in Ds]
        for block in _blocks(types, xyz, omega):
            for a1, a2, a3, a4, I in _orders(block):
                for D, j, k in zip(Ds, J, K):
                    j[a1[:, None], a2[None]] += torch.einsum("abcd,cd->ab", I, D[a3][:, a4])
                    k[a1[:, None], a3[None]] += torch.einsum("abcd,bd->ac", I, D[a2][:, a4])
        if kind == "lockstep":
            out.append(torch.stack([J[0], K[0]]))
        else:
            out += [x.cpu().numpy() for x in J + K]
    return out
