"""Performance cases of the two-electron engine.

Each case is one call (or one short sequence of calls) that a program using
this package makes in earnest: a J/K build of an SCF iteration, a nuclear
gradient, a captured build of a batch of molecules, one geometry from scratch,
and the two kernel-level sweeps (Boys function, primitive blocks).  Inputs are
seeded; densities are block-dominant like those of a water cluster (occupied
orbitals localised on their molecule), so screening meets realistic values.

``exact`` restates the quantities in plain torch FP64: McMurchie-Davidson
integrals over all primitives, unscreened, with Boys values from a table
computed in extended precision.
"""

from __future__ import annotations

import math
from functools import lru_cache
from itertools import product
from types import SimpleNamespace

import numpy as np
import torch

import jax_examples_b200 as jqc
from jax_examples_b200 import flops as model
from jax_examples_b200.batch import BatchedERI, MoleculeBatch

DEV = "cuda:0"
BOHR = 1.0 / 0.529177210903
ORBITALS = 5  # occupied orbitals of one water
# (precision, density-screening threshold, size of the density) of the builds
# an SCF makes: a full plain build, the incremental FP64 builds near
# convergence, the full and the incremental builds of the mixed phase.
MODES = {
    "full": ("fp64", 0.0, 1.0),
    "tail": ("fp64", 1e-10, 1e-5),
    "mixed": ("mixed", 1e-8, 1.0),
    "mixed-inc": ("mixed", 2e-8, 1e-3),
}
MIXED_TAU = 1e-4


def listed():
    return [
        # one SCF iteration of the smallest molecule anybody runs: launch and latency bound
        dict(name="jk_water_sto3g", kind="jk", waters=1, basis="sto-3g", spherical=False, spins=1, mode="full"),
        # an open-shell (UHF) iteration in the spherical layout of the reference's default
        dict(name="jk_uhf_w3_631gss", kind="jk", waters=3, basis="6-31g**", spherical=True, spins=2, mode="full"),
        # a full build of a mid-size molecule
        dict(name="jk_w8_631gs", kind="jk", waters=8, basis="6-31g*", spherical=False, spins=1, mode="full"),
        # the headline build: (H2O)16, 304 functions
        dict(name="jk_w16_631gs", kind="jk", waters=16, basis="6-31g*", spherical=False, spins=1, mode="full"),
        # what most iterations of a mixed-precision SCF on it are
        dict(name="jk_w16_mixed_inc", kind="jk", waters=16, basis="6-31g*", spherical=False, spins=1,
             mode="mixed-inc"),
        # one build of a sweep over molecules of uneven size, replayed from its graph
        dict(name="batch_24_mixed_inc", kind="batch", molecules=24, most=12, mode="mixed-inc"),
        # the gradient of one step of a geometry optimisation, plain and screened
        dict(name="grad_w5_631gs", kind="grad", waters=5, basis="6-31g*", spherical=False, spins=1, tau=0.0),
        dict(name="grad_w16_screened", kind="grad", waters=16, basis="6-31g*", spherical=False, spins=1, tau=1e-9),
        # energy and gradient of a new geometry from scratch, as an optimiser asks for them
        dict(name="geometry_water_631gs", kind="geometry", waters=1, basis="6-31g*"),
        # kernel-level sweeps
        dict(name="boys_m8", kind="boys", n=(1 << 22) + 3, m=8, fp32=False),
        dict(name="prim_pppp", kind="prim", cls="1111", n=1 << 20),
        dict(name="prim_dddd", kind="prim", cls="2222", n=(1 << 16) + 5),
    ]


def draw(rng):
    def size(lo, hi):  # log-uniform
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))

    kind = rng.choice(["jk", "jk", "jk", "grad", "grad", "batch", "geometry", "boys", "prim"])
    basis = rng.choice(["sto-3g", "6-31g", "6-31g*", "6-31g*", "6-31g**"])
    if kind == "jk":
        spins = rng.choice([1, 1, 2])
        return dict(kind=kind, waters=size(1, 15 if spins == 1 else 8), basis=basis, spherical=rng.random() < 0.3,
                    spins=spins, mode=rng.choice(sorted(MODES)))
    if kind == "grad":
        spins = rng.choice([1, 1, 2])
        return dict(kind=kind, waters=size(1, 9 if spins == 1 else 5), basis=basis, spherical=rng.random() < 0.3,
                    spins=spins, tau=rng.choice([0.0, 1e-9]) if spins == 1 else 0.0)
    if kind == "batch":
        return dict(kind=kind, molecules=size(2, 23), most=rng.randint(2, 12), mode=rng.choice(sorted(MODES)))
    if kind == "geometry":
        return dict(kind=kind, waters=1, basis=rng.choice(["sto-3g", "6-31g", "6-31g**"]))
    if kind == "boys":
        return dict(kind=kind, n=size(1 << 10, 1 << 22), m=rng.randint(0, 8), fp32=rng.random() < 0.3)
    cls = rng.choice(["0000", "1000", "1010", "1111", "2010", "2110", "2111", "2121", "2200", "2211", "2222"])
    values = math.prod(jqc.core.n_cartesian(int(c)) for c in cls)
    return dict(kind=kind, cls=cls, n=size(1 << 10, min(1 << 20, (1 << 26) // values)))


# ------------------------------------------------------------------- inputs
def _cluster(waters, seed, charge=0, spin=0):
    return jqc.water_cluster(waters, seed=seed, noise_angstrom=0.05, charge=charge, spin=spin)


def _orbitals(mol, basis, seed):
    """Seeded occupied orbitals (n, n_occ), each localised on one water."""
    rng = np.random.default_rng(seed + 7919)
    xyz = np.asarray(mol.coords)
    centre = xyz[np.asarray(basis.basis_to_atom)]
    oxygen = np.repeat(xyz[::3], ORBITALS, axis=0)
    far = np.linalg.norm(centre[:, None] - oxygen[None], axis=-1)
    C = rng.standard_normal((basis.n_basis, len(oxygen))) * np.exp(-far / 1.2)
    return C / np.linalg.norm(C, axis=0)


def _densities(mol, basis, spins, size, seed):
    C = _orbitals(mol, basis, seed)
    if spins == 1:
        D = [2.0 * C @ C.T]
    else:
        D = [C @ C.T, C[:, :-1] @ C[:, :-1].T]  # one electron less in the second spin
    return [torch.tensor(size * d, dtype=torch.float64, device=DEV) for d in D]


def _molecule(case, seed):
    spins = case.get("spins", 1)
    mol = _cluster(case["waters"], seed, charge=spins - 1, spin=spins - 1)
    return mol, jqc.build_basis_set(mol, case["basis"], spherical=case.get("spherical", False))


def _batch_molecules(case, seed):
    """Water clusters of uneven size; the sizes belong to the case, not to the seed."""
    sizes = np.random.default_rng(case["molecules"]).integers(1, case["most"] + 1, case["molecules"])
    return [_cluster(int(n), 1000 * seed + i) for i, n in enumerate(sizes)]


def _batch_density(mols, bases, size, seed):
    n = sum(b.n_basis for b in bases)
    D = torch.zeros((1, n, n), dtype=torch.float64, device=DEV)
    o = 0
    for i, (m, b) in enumerate(zip(mols, bases)):
        D[0, o:o + b.n_basis, o:o + b.n_basis] = _densities(m, b, 1, size, 1000 * seed + i)[0]
        o += b.n_basis
    return D


def _scf_state(case, seed):
    """A converged state as the gradient takes it: density, orbitals and their energies."""
    mol, basis = _molecule(case, seed)
    C = _orbitals(mol, basis, seed)
    eps = np.sort(np.random.default_rng(seed + 104729).uniform(-2.0, -0.4, C.shape[1]))
    dens = _densities(mol, basis, case["spins"], 1.0, seed)
    dev = lambda x: torch.tensor(x, dtype=torch.float64, device=DEV)  # noqa: E731
    state = SimpleNamespace(density=sum(dens), coefficients=dev(C), orbital_energies=dev(eps))
    extra = None
    if case["spins"] == 2:
        extra = dict(density_alpha=dens[0], density_beta=dens[1], coefficients_beta=dev(C[:, :-1]),
                     orbital_energies_beta=dev(eps[:-1]))
    return mol, basis, SimpleNamespace(state=state, precision=extra)


def _boys_arguments(case, seed):
    """Half uniform in [0, 30], half log-uniform in [1e-8, 1e3]."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    u = torch.rand(case["n"], dtype=torch.float64, device=DEV, generator=g)
    wide = torch.exp(math.log(1e-8) + u * math.log(1e11))
    return torch.where(torch.arange(case["n"], device=DEV) % 2 == 0, 30.0 * u, wide)


def _prim_arguments(case, seed):
    """Exponents log-uniform in [0.1, 100], centres uniform in a 4 A cube."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    e = torch.exp(math.log(0.1) + torch.rand(case["n"], 4, dtype=torch.float64, device=DEV, generator=g) * math.log(1e3))
    return e, 4.0 * BOHR * torch.rand(case["n"], 4, 3, dtype=torch.float64, device=DEV, generator=g)


def prepare(case, seed):
    kind = case["kind"]
    s = SimpleNamespace(case=case, kind=kind)
    if kind == "jk":
        mol, basis = _molecule(case, seed)
        s.precision, s.tau, size = MODES[case["mode"]]
        dens = _densities(mol, basis, case["spins"], size, seed)
        s.D = dens[0] if case["spins"] == 1 else torch.stack(dens)
        s.engine = jqc.DirectERI(basis, mol, device=0, schwarz_tau=1e-12)
    elif kind == "batch":
        s.precision, s.tau, size = MODES[case["mode"]]
        batch = MoleculeBatch(_batch_molecules(case, seed), "6-31g*")
        s.engine = BatchedERI(batch, device=0)
        s.D, s.J, s.K = s.engine.buffers()
        s.D.copy_(_batch_density(batch.mols, batch.bases, size, seed))
        s.graph = s.engine.capture_jk(s.D, s.J, s.K, s.precision, MIXED_TAU, max(s.tau, 1e-30))
    elif kind == "grad":
        s.mol, basis, s.result = _scf_state(case, seed)
        s.engine = jqc.DirectERI(basis, s.mol, device=0, schwarz_tau=1e-12)
    elif kind == "geometry":
        s.mol = jqc.water_cluster(case["waters"], seed=seed)
        noise = np.random.default_rng(seed).standard_normal(s.mol.coords.shape)
        s.mol = s.mol.replace(coords=s.mol.coords + 0.03 * noise)
        s.basis = jqc.build_basis_set(s.mol, case["basis"])
    elif kind == "boys":
        s.T = _boys_arguments(case, seed)
    else:
        s.exps, s.centres = _prim_arguments(case, seed)
    return s


def run(s):
    if s.kind == "jk":
        return s.engine.jk(s.D, precision=s.precision, mixed_tau=MIXED_TAU, dens_tau=s.tau)
    if s.kind == "batch":
        s.engine.launch(s.graph)
        return s.J, s.K
    if s.kind == "grad":
        if s.case["spins"] == 2:
            return jqc.uhf_gradient(s.mol, s.result, engine=s.engine)
        return jqc.rhf_gradient(s.mol, s.result, engine=s.engine, dens_tau=s.case["tau"])
    if s.kind == "geometry":
        ints = jqc.compute_integrals(s.mol, s.basis, device=0)
        res = jqc.run_scf(s.mol, ints)
        return res.energy, res.state.density, res.state.fock, jqc.rhf_gradient(s.mol, res)
    if s.kind == "boys":
        return jqc.boys(s.T, s.case["m"], fp32=s.case["fp32"])
    return jqc.eri_prim_quartets([int(c) for c in s.case["cls"]], s.exps, s.centres)


# --------------------------------------------------------------------- work
@lru_cache(maxsize=None)
def _quartet_work(waters, basis, thr):
    """{pair-class pair: (shell quartets, primitive quartets)} with Q_ab Q_cd >= thr
    on the seed-0 cluster, the Schwarz bounds estimated from s functions."""
    mol = _cluster(waters, 0)
    shells = jqc.build_basis_set(mol, basis).shells
    by = {}
    for i, a in enumerate(shells):
        for b in shells[: i + 1]:
            x, y = (a, b) if a.angular_momentum >= b.angular_momentum else (b, a)
            p = np.add.outer(x.exponents, y.exponents)
            k = np.exp(-np.multiply.outer(x.exponents, y.exponents) / p * float(np.sum((x.center - y.center) ** 2)))
            mag = np.abs(np.multiply.outer(x.coefficients, y.coefficients)) * k * 4.16 * p ** -1.25
            l = int(x.angular_momentum), int(y.angular_momentum)
            by.setdefault(l, []).append((float(mag.max()), int((mag > 1e-20).sum())))
    out = {}
    classes = sorted(by)
    arr = {c: np.array(sorted(v)) for c, v in by.items()}
    for ib, cb in enumerate(classes):
        for ck in classes[: ib + 1]:
            q, n = arr[ck][:, 0], arr[ck][:, 1]
            tail = np.concatenate([np.cumsum(n[::-1])[::-1], [0.0]])
            first = np.searchsorted(q, thr / np.maximum(arr[cb][:, 0], 1e-300))
            quartets, prims = float((len(q) - first).sum()), float((arr[cb][:, 1] * tail[first]).sum())
            half = 0.5 if ib == classes.index(ck) else 1.0
            out[cb + ck] = (half * quartets, half * prims)
    return out


def _build_flops(waters, basis, thr, spins, gradient=False):
    total = 0.0
    for cls, (quartets, prims) in _quartet_work(waters, basis, thr).items():
        each = model.grad_prim_quartet_flops(*cls) if gradient else model.prim_quartet_flops(*cls)
        total += prims * each + quartets * model.digestion_flops(*cls, n_dens=spins)
    return total


def work(case):
    kind = case["kind"]
    if kind == "boys":
        size = 4 if case["fp32"] else 8
        return dict(bytes=case["n"] * (8 + size * (case["m"] + 1)), flops=case["n"] * (20 + 3 * case["m"]))
    if kind == "prim":
        cls = [int(c) for c in case["cls"]]
        values = math.prod(jqc.core.n_cartesian(c) for c in cls)
        return dict(bytes=8 * case["n"] * (16 + values), flops=case["n"] * model.prim_quartet_flops(*cls))
    if kind == "batch":
        _, tau, size = MODES[case["mode"]]
        sizes = [(len(m.coords) // 3) for m in _batch_molecules(case, 0)]
        n = 19 * sum(sizes)
        return dict(bytes=8 * 3 * sum((19 * k) ** 2 for k in sizes) + 16 * n,
                    flops=sum(_build_flops(k, "6-31g*", max(1e-12, tau / size), 1) for k in sizes))
    n = jqc.build_basis_set(_cluster(case["waters"], 0), case["basis"], spherical=case.get("spherical", False)).n_basis
    if kind == "jk":
        _, tau, size = MODES[case["mode"]]
        return dict(bytes=24 * case["spins"] * n * n,
                    flops=_build_flops(case["waters"], case["basis"], max(1e-12, tau / size), case["spins"]))
    if kind == "grad":
        return dict(bytes=16 * case["spins"] * n * n + 72 * case["waters"],
                    flops=_build_flops(case["waters"], case["basis"], max(1e-12, case["tau"]), case["spins"], True))
    # one geometry: about a dozen builds and one gradient
    return dict(bytes=8 * n * n * 40, flops=12 * _build_flops(case["waters"], case["basis"], 1e-13, 1)
                + _build_flops(case["waters"], case["basis"], 1e-13, 1, True))


# -------------------------------------------------------------------- exact
def _cart(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _herm(L):
    return [(t, u, v) for s in range(L + 1) for t, u, v in _cart(s)]


GRID = 32  # Boys table: T = i / GRID up to T_ASYMPTOTIC
T_ASYMPTOTIC = 44.0
TAYLOR = 8


@lru_cache(maxsize=None)
def _boys_table(top):
    """F_m(T_i), m = 0 .. top, summed and recurred down in extended precision."""
    t = np.arange(int(T_ASYMPTOTIC * GRID) + 1, dtype=np.longdouble) / GRID
    term = np.ones_like(t) / (2 * top + 1)
    total = term.copy()
    for k in range(1, 400):
        term = term * (2 * t / (2 * top + 2 * k + 1))
        total += term
    e = np.exp(-t)
    F = [e * total]
    for m in range(top - 1, -1, -1):
        F.append((2 * t * F[-1] + e) / (2 * m + 1))
    return torch.tensor(np.array(F[::-1], dtype=np.float64).T.copy(), device=DEV)


def _boys(T, M):
    """F_0 .. F_M of a tensor, as a list."""
    tab = _boys_table(M + TAYLOR)
    small = T.clamp(max=T_ASYMPTOTIC)
    i = torch.round(small * GRID)
    d = i / GRID - small
    i = i.long()
    f = torch.zeros_like(T)
    for k in range(TAYLOR, -1, -1):
        f = tab[i, M + k] + f * d / (k + 1)
    low = [f]
    for m in range(M - 1, -1, -1):
        low.append((2 * small * low[-1] + torch.exp(-small)) / (2 * m + 1))
    low = low[::-1]
    big = T.clamp(min=T_ASYMPTOTIC)
    high = [0.5 * torch.sqrt(math.pi / big)]
    for m in range(M):
        high.append(((2 * m + 1) * high[-1] - torch.exp(-big)) / (2 * big))
    return [torch.where(T < T_ASYMPTOTIC, a, b) for a, b in zip(low, high)]


class _BoysStack(torch.autograd.Function):
    """F_0 .. F_M stacked, with dF_m/dT = -F_{m+1}."""

    @staticmethod
    def forward(ctx, T, M):
        F = _boys(T, M + 1)
        ctx.save_for_backward(*F[1:])
        return torch.stack(F[:-1])

    @staticmethod
    def backward(ctx, g):
        return -sum(gm * f for gm, f in zip(g, ctx.saved_tensors)), None


def _r_tensors(alpha, X, Y, Z, L):
    """{(t, u, v): R_tuv} of total order <= L at exponent alpha and distance (X, Y, Z)."""
    F = _BoysStack.apply(alpha * (X * X + Y * Y + Z * Z), L)
    level = {(0, 0, 0): (-2 * alpha) ** L * F[L]}
    for n in range(L - 1, -1, -1):
        up, level = level, {(0, 0, 0): (-2 * alpha) ** n * F[n]}
        for t, u, v in _herm(L - n)[1:]:
            if t:
                a, k, x = (t - 1, u, v), t - 1, X
                b = (t - 2, u, v)
            elif u:
                a, k, x = (t, u - 1, v), u - 1, Y
                b = (t, u - 2, v)
            else:
                a, k, x = (t, u, v - 1), v - 1, Z
                b = (t, u, v - 2)
            level[t, u, v] = x * up[a] + (k * up[b] if k else 0.0)
    return level


def _e_axis(la, lb, PA, PB, p):
    """{(i, j, t): E^{ij}_t} of one axis."""
    E = {(0, 0, 0): torch.ones_like(p)}

    def get(i, j, t):
        return E.get((i, j, t), 0.0)

    for i, j in product(range(la + 1), range(lb + 1)):
        if i == j == 0:
            continue
        k, l, X = (i - 1, j, PA) if i else (i, j - 1, PB)
        for t in range(i + j + 1):
            E[i, j, t] = get(k, l, t - 1) / (2 * p) + X * get(k, l, t) + (t + 1) * get(k, l, t + 1)
    return E


def _pair_e(la, lb, A, B, P, p, K):
    """(pairs, Cartesian pairs, Hermite) products E^x E^y E^z K, and the axis tables."""
    ax = [_e_axis(la, lb, P[:, k] - A[:, k], P[:, k] - B[:, k], p) for k in range(3)]
    zero = torch.zeros_like(p)
    rows = []
    for a, b in product(_cart(la), _cart(lb)):
        rows.append(torch.stack([
            K * ax[0][a[0], b[0], t] * ax[1][a[1], b[1], u] * ax[2][a[2], b[2], v]
            if t <= a[0] + b[0] and u <= a[1] + b[1] and v <= a[2] + b[2] else zero
            for t, u, v in _herm(la + lb)], dim=1))
    return torch.stack(rows, dim=1)


class _Pairs:
    """Shell pairs of one angular class with their primitives, centres taken from xyz (atoms, 3)."""

    def __init__(self, shells, la, lb, first, xyz):
        self.la, self.lb = la, lb
        off = np.concatenate([[0], np.cumsum([len(_cart(int(s.angular_momentum))) for s in shells])])
        prims, self.a, self.b = [], [], []
        nb = len(_cart(lb))
        self.nab = len(_cart(la)) * nb
        for i, s in enumerate(shells):
            for j in range(i + 1):
                r = shells[j]
                x, y, ix, iy = (s, r, i, j) if s.angular_momentum >= r.angular_momentum else (r, s, j, i)
                if (int(x.angular_momentum), int(y.angular_momentum)) != (la, lb):
                    continue
                q = len(self.a)
                self.a.append((off[ix], ix))
                self.b.append((off[iy], iy))
                for (e, c), (f, d) in product(zip(x.exponents, x.coefficients), zip(y.exponents, y.coefficients)):
                    prims.append((q, x.atom_index, y.atom_index, e, f, c * d))
        self.n, self.first = len(self.a), first
        t = torch.tensor(np.array(prims, dtype=np.float64).reshape(-1, 6), device=DEV)
        self.pair = t[:, 0].long()
        A, B, al, be = xyz[t[:, 1].long()], xyz[t[:, 2].long()], t[:, 3], t[:, 4]
        self.p = al + be
        self.P = (al[:, None] * A + be[:, None] * B) / self.p[:, None]
        K = t[:, 5] * torch.exp(-al * be / self.p * ((A - B) ** 2).sum(1))
        self.E = _pair_e(la, lb, A, B, self.P, self.p, K)
        self.al, self.be, self.A, self.B, self.K = al, be, A, B, K
        # basis-function indices of every pair function, and whether the shells differ
        ai = np.array([o for o, _ in self.a])[:, None] + np.repeat(np.arange(len(_cart(la))), nb)[None]
        bi = np.array([o for o, _ in self.b])[:, None] + np.tile(np.arange(nb), len(_cart(la)))[None]
        self.fa, self.fb = (torch.tensor(v.reshape(-1), device=DEV) for v in (ai, bi))
        off_diag = np.array([x != y for (_, x), (_, y) in zip(self.a, self.b)])
        self.mult = torch.tensor(np.repeat(1.0 + off_diag, self.nab), device=DEV)


def _all_pairs(shells, xyz):
    out, first = [], 0
    for la, lb in [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2)]:
        g = _Pairs(shells, la, lb, first, xyz)
        if g.n:
            out.append(g)
            first += g.n * g.nab
    return out, first


def _eri_rows(bra, ket, lo, hi):
    """Pair functions of the bra primitives [lo, hi) x all of the ket: (hi - lo, nab, ket pairs, ncd),
    contracted over the ket's primitives."""
    p, q = bra.p[lo:hi, None], ket.p[None, :]
    X, Y, Z = (bra.P[lo:hi, None, k] - ket.P[None, :, k] for k in range(3))
    lab, lcd = bra.la + bra.lb, ket.la + ket.lb
    R = _r_tensors(p * q / (p + q), X, Y, Z, lab + lcd)
    pref = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
    sign = torch.tensor([(-1.0) ** sum(h) for h in _herm(lcd)], device=DEV, dtype=torch.float64)
    Ek = ket.E * sign
    out = 0.0
    for x, h in enumerate(_herm(lab)):
        Rh = torch.stack([pref * R[h[0] + k[0], h[1] + k[1], h[2] + k[2]] for k in _herm(lcd)], dim=-1)
        cd = torch.einsum("bkh,kch->kbc", Rh, Ek)
        acc = torch.zeros((ket.n,) + cd.shape[1:], dtype=torch.float64, device=DEV).index_add(0, ket.pair, cd)
        out = out + torch.einsum("ba,nbc->banc", bra.E[lo:hi, :, x], acc)
    return out


def _chunks(bra, ket, budget=1 << 24):
    size = len(_herm(bra.la + bra.lb + ket.la + ket.lb)) + bra.nab * ket.nab
    step = max(1, budget // max(1, size * len(ket.p)))
    for lo in range(0, len(bra.p), step):
        yield lo, min(len(bra.p), lo + step)


def _exact_jk(basis, mol, dens):
    """J and K (Cartesian) of every density, from all integrals over pair functions."""
    xyz = torch.tensor(np.asarray(mol.coords), dtype=torch.float64, device=DEV)
    groups, N = _all_pairs(basis.shells, xyz)
    M = torch.zeros((N, N), dtype=torch.float64, device=DEV)
    for ib, bra in enumerate(groups):
        for ket in groups[: ib + 1]:
            blk = torch.zeros((bra.n, bra.nab, ket.n * ket.nab), dtype=torch.float64, device=DEV)
            for lo, hi in _chunks(bra, ket):
                blk.index_add_(0, bra.pair[lo:hi], _eri_rows(bra, ket, lo, hi).reshape(hi - lo, bra.nab, -1))
            rows, cols = slice(bra.first, bra.first + bra.n * bra.nab), slice(ket.first, ket.first + ket.n * ket.nab)
            M[rows, cols] = blk.reshape(-1, ket.n * ket.nab)
            if bra is not ket:
                M[cols, rows] = M[rows, cols].T
    n = dens[0].shape[0]
    idx = torch.zeros((n, n), dtype=torch.long, device=DEV)
    for g in groups:
        at = g.first + torch.arange(g.n * g.nab, device=DEV)
        idx[g.fb, g.fa] = at
        idx[g.fa, g.fb] = at
    J, K = [], []
    for D in dens:
        flat = torch.zeros(N, dtype=torch.float64, device=DEV).index_add_(0, idx.reshape(-1), D.reshape(-1))
        J.append((M @ flat)[idx])
        K.append(torch.stack([torch.einsum("bcd,bd->c", M[idx[a]][:, idx], D) for a in range(n)]))
    return J, K


SPHERICAL_D = [[0, 3 ** 0.5, 0, 0, 0, 0], [0, 0, 0, 0, 3 ** 0.5, 0], [-0.5, 0, 0, -0.5, 0, 1],
               [0, 0, 3 ** 0.5, 0, 0, 0], [3 ** 0.5 / 2, 0, 0, -(3 ** 0.5) / 2, 0, 0]]


def _to_cartesian(basis):
    """(n, n_cart) map of the basis onto Cartesian functions; identity for a Cartesian basis."""
    ls = [int(s.angular_momentum) for s in basis.shells]
    return torch.block_diag(*[
        torch.tensor(SPHERICAL_D if basis.spherical and l == 2 else np.eye(len(_cart(l))), dtype=torch.float64)
        for l in ls]).to(DEV)


def _one_electron_lagrangian(groups, xyz, Z, D, W):
    """Tr[D (T + V)] - Tr[W S] over pair functions."""
    total = 0.0
    for g in groups:
        ax = [_e_axis(g.la, g.lb + 2, g.P[:, k] - g.A[:, k], g.P[:, k] - g.B[:, k], g.p) for k in range(3)]
        root = torch.sqrt(math.pi / g.p)

        def s1(k, i, j):
            return ax[k][i, j, 0] * root

        def t1(k, i, j):
            v = -2 * g.be ** 2 * s1(k, i, j + 2) + g.be * (2 * j + 1) * s1(k, i, j)
            return v - 0.5 * j * (j - 1) * s1(k, i, j - 2) if j > 1 else v

        nai = 0.0
        for c, z in zip(xyz, Z):
            R = _r_tensors(g.p, *(g.P[:, k] - c[k] for k in range(3)), g.la + g.lb)
            nai = nai - z * 2 * math.pi / g.p * torch.stack([R[h] for h in _herm(g.la + g.lb)])
        V = torch.einsum("pfh,hp->pf", g.E, nai)
        m = g.mult.reshape(g.n, g.nab)[g.pair]
        Dp, Wp = (m * M[g.fa, g.fb].reshape(g.n, g.nab)[g.pair] for M in (D, W))
        for f, (a, b) in enumerate(product(_cart(g.la), _cart(g.lb))):
            S = g.K * s1(0, a[0], b[0]) * s1(1, a[1], b[1]) * s1(2, a[2], b[2])
            T = g.K * sum(
                t1(k, a[k], b[k]) * s1((k + 1) % 3, a[(k + 1) % 3], b[(k + 1) % 3])
                * s1((k + 2) % 3, a[(k + 2) % 3], b[(k + 2) % 3]) for k in range(3))
            total = total + (Dp[:, f] * (T + V[:, f])).sum() - (Wp[:, f] * S).sum()
    return total


def _exact_gradient(basis, mol, dens, W, kscale):
    """Gradient of E_nuc + Tr[D h] - Tr[W S] + E2 at fixed densities, by autograd."""
    xyz = torch.tensor(np.asarray(mol.coords), dtype=torch.float64, device=DEV, requires_grad=True)
    Z = [float(z) for z in mol.atomic_numbers]
    D = sum(dens)
    i, j = torch.triu_indices(len(Z), len(Z), 1)
    zt = torch.tensor(Z, dtype=torch.float64, device=DEV)
    groups, _ = _all_pairs(basis.shells, xyz)
    L = (zt[i] * zt[j] / torch.linalg.norm(xyz[i] - xyz[j], dim=1)).sum()
    L = L + _one_electron_lagrangian(groups, xyz, Z, D, W)
    # two-electron part: the pair quantities are leaves of each chunk's own small graph
    leaves = [(g.P, g.E) for g in groups]
    for g in groups:
        g.P, g.E = g.P.detach().requires_grad_(), g.E.detach().requires_grad_()
    for ib, bra in enumerate(groups):
        for ket in groups[: ib + 1]:
            weight = 0.5 * (1.0 if bra is ket else 2.0)
            fa, fb, bm = (v.reshape(bra.n, bra.nab) for v in (bra.fa, bra.fb, bra.mult))
            for lo, hi in _chunks(bra, ket, 1 << 22):
                a, b = fa[bra.pair[lo:hi]][:, :, None], fb[bra.pair[lo:hi]][:, :, None]
                gam = D[a, b] * D[ket.fa, ket.fb]
                for d in dens:
                    gam = gam - 0.5 * kscale * (d[a, ket.fa] * d[b, ket.fb] + d[a, ket.fb] * d[b, ket.fa])
                gam = weight * gam * bm[bra.pair[lo:hi]][:, :, None] * ket.mult
                (_eri_rows(bra, ket, lo, hi).reshape(gam.shape) * gam).sum().backward()
    outs = [L] + [v for pair in leaves for v in pair]
    seeds = [torch.ones_like(L)] + [v.grad for g in groups for v in (g.P, g.E)]
    (grad,) = torch.autograd.grad(outs, [xyz], seeds)
    return grad


def _exact_prim(cls, exps, centres):
    la, lb, lc, ld = cls
    out = []
    step = max(1, (1 << 25) // (math.prod(len(_cart(l)) for l in cls) + 200))
    sign = torch.tensor([(-1.0) ** sum(h) for h in _herm(lc + ld)], device=DEV, dtype=torch.float64)
    for lo in range(0, len(exps), step):
        e, c = exps[lo:lo + step], centres[lo:lo + step]
        side = []
        for k, (l, m) in ((0, (la, lb)), (2, (lc, ld))):
            p = e[:, k] + e[:, k + 1]
            P = (e[:, k, None] * c[:, k] + e[:, k + 1, None] * c[:, k + 1]) / p[:, None]
            K = torch.exp(-e[:, k] * e[:, k + 1] / p * ((c[:, k] - c[:, k + 1]) ** 2).sum(1))
            side.append((p, P, _pair_e(l, m, c[:, k], c[:, k + 1], P, p, K)))
        (p, P, E), (q, Q, F) = side
        R = _r_tensors(p * q / (p + q), *(P[:, k] - Q[:, k] for k in range(3)), sum(cls))
        pref = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        F = F * sign * pref[:, None, None]
        blk = 0.0
        for x, h in enumerate(_herm(la + lb)):
            Rh = torch.stack([R[h[0] + k[0], h[1] + k[1], h[2] + k[2]] for k in _herm(lc + ld)], dim=1)
            blk = blk + E[:, :, x, None] * torch.einsum("qch,qh->qc", F, Rh)[:, None, :]
        out.append(blk.reshape(len(e), *(len(_cart(l)) for l in cls)))
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "boys":
        T = _boys_arguments(case, seed)
        return torch.stack(_boys(T, case["m"]), dim=1)
    if kind == "prim":
        return _exact_prim([int(c) for c in case["cls"]], *_prim_arguments(case, seed))
    if kind == "jk":
        if case["waters"] > 8:
            return None  # about a minute
        mol, basis = _molecule(case, seed)
        dens = _densities(mol, basis, case["spins"], MODES[case["mode"]][2], seed)
        C = _to_cartesian(basis)
        J, K = _exact_jk(basis, mol, [C.T @ d @ C for d in dens])
        J, K = torch.stack([C @ j @ C.T for j in J]), torch.stack([C @ k @ C.T for k in K])
        return (J, K) if case["spins"] == 2 else (J[0], K[0])
    if kind == "grad":
        if case["waters"] > 3:
            return None  # the chunks' graphs take too long
        mol, basis, result = _scf_state(case, seed)
        C, st, x = _to_cartesian(basis), result.state, result.precision
        W = (3.0 - case["spins"]) * (st.coefficients * st.orbital_energies) @ st.coefficients.T
        dens = [st.density]
        if x is not None:
            Cb, eb = x["coefficients_beta"], x["orbital_energies_beta"]
            W = W + (Cb * eb) @ Cb.T
            dens = [x["density_alpha"], x["density_beta"]]
        return _exact_gradient(basis, mol, [C.T @ d @ C for d in dens], C.T @ W @ C, 0.5 if x is None else 1.0)
    return None  # batches and whole calculations: no closed form at these sizes
