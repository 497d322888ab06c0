"""Performance cases of the scattering-rate path: what a user has it do, through
the Python binding of the C-ABI, with host arrays in and host arrays out.

Every case is one call (or the two or three calls that a solve always makes
together) of fourphonon_b200.abi.Context on a seeded synthetic solve:

  rta4     RTA_driver_4ph at one or several temperatures
  np4      NP_driver_4ph (the counting stage that every four-phonon run starts with)
  sample4  RTA_driver_4ph with sampled processes
  bte3     the three-phonon BTE from its start to the first iterate: NP_driver,
           Ind_driver, iteration0, one Jacobi sweep and kappa
  iter     one in-order sweep of the iterative BTE, its symmetrisation and kappa

Cells, grids and temperatures are those of the tests, of bench.py and of the
serving stream: 2-atom diamond and zincblende, the 4-atom layered cell and
random many-atom cells.
"""
from __future__ import annotations

import functools
import itertools

import numpy as np
import torch

from fourphonon_b200 import abi
from fourphonon_b200 import crystal as C
from fourphonon_b200 import ifcgen as G
from fourphonon_b200 import system as S

PRECISIONS = {"fp64": abi.FP4_PREC_FP64, "mixed": abi.FP4_PREC_MIXED, "mixed_simt": abi.FP4_PREC_MIXED_SIMT}
TEMPS = (300.0, 700.0, 100.0, 1000.0, 500.0, 200.0, 400.0, 900.0)


def _case(op, cell, grid, nT=1, precision="fp64", samples=0):
    return {"op": op, "cell": cell, "n1": grid[0], "n2": grid[1], "n3": grid[2], "nT": nT, "precision": precision,
            "samples": samples}


def listed():
    named = {
        # a quick look at a new cell, and the unit of a test: the latency of one call
        "rta4_diamond_4": _case("rta4", "diamond", (4, 4, 4)),
        # the small grid of a convergence study in the q grid (the benchmark's smallest cell)
        "rta4_diamond_6": _case("rta4", "diamond", (6, 6, 6)),
        # a grid with three different edges, and four temperatures in one call
        "rta4_zincblende_4x5x6_4T": _case("rta4", "zincblende", (4, 5, 6), nT=4),
        # the production grid, as large as a pass here may be; two temperatures as in the benchmark
        "rta4_diamond_12_2T": _case("rta4", "diamond", (12, 12, 12), nT=2),
        # 12 branches and many displacement classes (LiCoO2-like cell, second-shell cutoff)
        "rta4_layered_5": _case("rta4", "layered", (5, 5, 5)),
        # a request of the serving stream: a random 5-atom cell without symmetry, 15 branches
        "rta4_random5_4": _case("rta4", "random5", (4, 4, 4)),
        # mixed precision with the contraction on the tensor cores, odd grid
        "rta4_mixed_diamond_7_2T": _case("rta4", "diamond", (7, 7, 7), nT=2, precision="mixed"),
        # mixed precision on the CUDA cores
        "rta4_simt_zincblende_8": _case("rta4", "zincblende", (8, 8, 8), precision="mixed_simt"),
        # the counting stage of a four-phonon run
        "np4_diamond_10": _case("np4", "diamond", (10, 10, 10)),
        # the sampled estimator for grids whose full enumeration is too dear
        "sample4_zincblende_12_4T": _case("sample4", "zincblende", (12, 12, 12), nT=4, samples=100000),
        # the three-phonon stage of the iterative BTE: counts, lists, amplitudes and a first sweep
        "bte3_diamond_16": _case("bte3", "diamond", (16, 16, 16)),
        # one step of the BTE loop
        "iter_diamond_12": _case("iter", "diamond", (12, 12, 12)),
    }
    return [dict(c, name=n) for n, c in named.items()]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _crystal(cell):
    if cell == "diamond":
        return C.diamond(5.43, (28.085, 28.085))
    if cell == "zincblende":
        return C.diamond(4.78, (10.81, 74.92))
    if cell == "layered":
        return C.layered_rhombohedral()
    return C.random_cell(np.random.default_rng(20240604), int(cell[6:]))


def _tol(cell):
    return 0.15 if cell.startswith("random") else 0.0


@functools.lru_cache(maxsize=None)
def _geometry(cell, grid):
    """Symmetry tables and wedge: the same for every seed."""
    sym = C.build_symmetry(_crystal(cell), grid)
    return sym, C.wedge(sym)


@functools.lru_cache(maxsize=None)
def _clusters(cell, order):
    """Two symmetric sets of force constants on the same clusters; their
    combinations are as symmetric."""
    cr = _crystal(cell)
    shell = 3 if order == 3 else (2 if cell == "layered" else 1)
    d = G.shell_distances(cr, shell + 1, _tol(cell))
    cut = 0.5 * (d[shell - 1] + d[shell])
    return [G.generate_anharmonic(cr, order, cut, 5.0 if order == 3 else 2.0, 101 + x) for x in range(2)]


def _ifc(cell, order, rng):
    a, b = _clusters(cell, order)
    th = rng.uniform(0.2, 1.3)
    mixed = G.Clusters(order, np.cos(th) * a.phi + np.sin(th) * b.phi, a.cells, a.atoms)
    return S.IFC.from_clusters(mixed, _crystal(cell).lattvec)


def _harmonic(cell, grid, sym, rng):
    """omega, group velocity and eigenvectors of seeded central-force springs, in
    the lattice-periodic gauge."""
    cr = _crystal(cell)
    consts = [rng.uniform(2.5, 3.5), rng.uniform(0.3, 0.6), 0.25 * rng.uniform(0.3, 0.6)]
    if cell in ("diamond", "zincblende"):
        consts = consts[:2]
    blocks = G.bvk_fc2(cr, consts, rel_tol=_tol(cell))
    nat, nb = cr.natoms, cr.nbands
    ijk = C.id2ind(grid).astype(float)
    k = (cr.rlattvec() @ (ijk / np.array(grid)[:, None])).T
    mass = cr.masses[cr.types - 1]
    D = np.zeros((k.shape[0], nb, nb), complex)
    dD = np.zeros((3, k.shape[0], nb, nb), complex)
    for (a, b, n), blk in blocks.items():
        R = cr.lattvec @ np.array(n, float)
        w = np.exp(1j * (k @ R))[:, None, None] * (9648.53336213 * blk / np.sqrt(mass[a] * mass[b]))
        D[:, 3 * a:3 * a + 3, 3 * b:3 * b + 3] += w
        for d in range(3):
            dD[d][:, 3 * a:3 * a + 3, 3 * b:3 * b + 3] += 1j * R[d] * w
    D = 0.5 * (D + np.conj(np.transpose(D, (0, 2, 1))))
    w2, z = np.linalg.eigh(D)
    omega = np.sign(w2) * np.sqrt(np.abs(w2))
    with np.errstate(divide="ignore", invalid="ignore"):
        vel = np.stack([np.einsum("qcb,qce,qeb->qb", np.conj(z), dD[d], z).real for d in range(3)], -1) / (
            2.0 * omega[..., None])
    vel = np.einsum("qab,qnb->qna", sym.symmetrizers, np.where(np.isfinite(vel), vel, 0.0))
    omega[0, :3] = 0.0
    vel[0, :3] = 0.0
    return np.asfortranarray(omega), np.asfortranarray(vel), np.asfortranarray(np.transpose(z, (0, 2, 1)))


def _solve(case, seed):
    grid = (case["n1"], case["n2"], case["n3"])
    rng = np.random.default_rng(seed)
    sym, wd = _geometry(case["cell"], grid)
    omega, vel, eig = _harmonic(case["cell"], grid, sym, rng)
    op = case["op"]
    ifc3 = _ifc(case["cell"], 3, rng) if op in ("bte3", "iter") else None
    ifc4 = _ifc(case["cell"], 4, rng) if op in ("rta4", "sample4") else None
    temps = [T + float(rng.uniform(-20.0, 20.0)) for T in TEMPS[:case["nT"]]]
    return S.Solve(_crystal(case["cell"]), grid, omega, vel, eig, sym, wd, temps, ifc3=ifc3, ifc4=ifc4)


def _tau(rate):
    return np.where(rate != 0.0, 1.0 / np.where(rate != 0.0, rate, 1.0), 0.0)


def prepare(case, seed):
    s = _solve(case, seed)
    ctx = abi.Context(0, PRECISIONS[case["precision"]])
    state = {"case": case, "solve": s, "ctx": ctx, "seed": seed}
    if case["op"] == "iter":  # what the loop has in hand: lists, amplitudes, tau and the RTA iterate
        n_p, n_m, _, _ = ctx.np_driver(s)
        lists = ctx.ind_driver(s, n_p, n_m)
        tau = _tau(lists["rate"])
        state.update(n_p=n_p, n_m=n_m, lists=lists, tau=tau, F0=ctx.iteration0(s, tau))
    return state


def run(state):
    c, s, ctx = state["case"], state["solve"], state["ctx"]
    if c["op"] == "rta4":
        return ctx.rta_driver_4ph(s)
    if c["op"] == "np4":
        return ctx.np_driver_4ph(s)
    if c["op"] == "sample4":
        return ctx.rta_driver_4ph_sample(s, c["samples"], state["seed"])
    if c["op"] == "bte3":
        n_p, n_m, p_p, p_m = ctx.np_driver(s)
        lists = ctx.ind_driver(s, n_p, n_m)
        tau = _tau(lists["rate"])
        F = ctx.iteration_jacobi(s, ctx.iteration0(s, tau), tau, n_p, n_m, lists)
        out = {k: v for k, v in lists.items() if k.startswith(("rate", "wp3"))}
        return dict(out, n_plus=n_p, n_minus=n_m, p_plus=p_p, p_minus=p_m, F=F, kappa=ctx.tconduct(s, F))
    F = ctx.iteration(s, state["F0"].copy(), state["tau"], state["n_p"], state["n_m"], state["lists"])
    F = ctx.symmetrize_fn(s, F)
    return {"F": F, "kappa": ctx.tconduct(s, F)}


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------

def _sizes(case):
    grid = (case["n1"], case["n2"], case["n3"])
    nb = _crystal(case["cell"]).nbands
    return int(np.prod(grid)), nb, _geometry(case["cell"], grid)[1].nlist


def _processes4(case):
    """Surviving four-phonon processes: a share of about 0.33/N (2 atoms; less in larger
    cells) of the (i,j,k,l) of each (q',q'')."""
    nptk, nb, nlist = _sizes(case)
    share = {6: 0.33, 12: 0.25}.get(nb, 0.17)
    return min(0.2, share / nptk ** (1.0 / 3.0)) * nlist * float(nptk) ** 2 * nb ** 4


def work(case):
    nptk, nb, nlist = _sizes(case)
    modes = nb * nlist
    harmonic = nptk * nb * (8 + 24 + 16 * nb)
    sigmas = 27.0 * 1.5 * nlist * float(nptk) ** 2 * nb ** 2  # one per (channel, q', q'', k, l) that the channel keeps
    per_v = 8.0 * (nb * nb + nb) + 60.0 + 12.0 * case["nT"]  # u T v, the Gaussian and the weights
    if case["op"] == "rta4":
        return {"bytes": harmonic + 48 * modes * case["nT"], "flops": sigmas + per_v * _processes4(case)}
    if case["op"] == "np4":
        return {"bytes": nptk * nb * 32 + 48 * modes, "flops": sigmas + 40.0 * _processes4(case)}
    if case["op"] == "sample4":
        draws = 3.0 * modes * case["samples"]
        return {"bytes": harmonic + 48 * modes * case["nT"], "flops": 30.0 * draws + per_v * 0.01 * draws}
    n3 = min(0.3, 0.6 / nptk ** (1.0 / 3.0)) * 1.5 * modes * nptk * nb ** 2
    if case["op"] == "bte3":
        return {"bytes": harmonic + 16 * n3, "flops": 27.0 * 2 * modes * nptk * nb ** 2 + per_v * n3}
    return {"bytes": 16 * n3 + nptk * nb * 80, "flops": 9.0 * n3 * nptk / nlist}


def draw(rng):
    largest = _processes4(_case("rta4", "diamond", (12, 12, 12)))
    while True:
        op = rng.choice(("rta4", "rta4", "rta4", "rta4", "np4", "sample4", "bte3", "iter"))
        cell = rng.choice(("diamond", "zincblende", "diamond", "layered", "random3", "random4", "random5"))
        if op in ("np4", "sample4", "bte3", "iter"):
            cell = rng.choice(("diamond", "zincblende"))
        top = {"bte3": 16, "iter": 12, "sample4": 14}.get(op, 12)
        n = int(round(4.0 * (top / 4.0) ** rng.random()))
        grid = (n, n, n)
        if rng.random() < 0.25 and op in ("rta4", "np4"):
            grid = tuple(max(2, n + rng.randint(-2, 2)) for _ in range(3))
        nT = rng.choice((1, 1, 2, 3, 4, 6)) if op in ("rta4", "sample4") else 1
        precision = rng.choice(("fp64", "fp64", "fp64", "mixed", "mixed_simt")) if op == "rta4" else "fp64"
        samples = int(10 ** rng.uniform(3.0, 5.3)) if op == "sample4" else 0
        case = _case(op, cell, grid, nT, precision, samples)
        if op in ("rta4", "np4") and _processes4(case) * (2.0 if cell != "diamond" else 1.0) > 0.5 * largest:
            continue
        if op == "sample4" and 3 * _sizes(case)[1] * _sizes(case)[2] * samples > 3e8:
            continue
        return case


# ---------------------------------------------------------------------------
# the same outputs in plain torch, in 64 bits
# ---------------------------------------------------------------------------

HBAR, KB = 1.05457172647e-22, 1.380648813e-23
HBARP = HBAR * float(np.float32(1e22))
DEV = "cuda" if torch.cuda.is_available() else "cpu"


class _T:
    """A solve's arrays in torch."""

    def __init__(self, s):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV)  # noqa: E731
        self.s, self.n, self.nb, self.nptk = s, s.ngrid, s.nb, s.nptk
        self.w, self.v, self.e = t(s.energy), t(s.velocity), t(s.eig)
        q = np.arange(s.nptk)
        self.ijk = t(np.stack([q % self.n[0], q // self.n[0] % self.n[1], q // (self.n[0] * self.n[1])], 1))
        self.rl = s.rlattvec

    def wrap(self, c):
        c = [torch.remainder(c[..., d], self.n[d]) for d in range(3)]
        return (c[2] * self.n[1] + c[1]) * self.n[0] + c[0]

    def sigma(self, dv):
        """base_sigma of velocity differences (...,3)."""
        m = None
        for d in range(3):
            r = self.rl[:, d]
            x = (dv[..., 0] * r[0] + dv[..., 1] * r[1] + dv[..., 2] * r[2]) / float(self.n[d])
            m = x * x if m is None else torch.maximum(m, x * x)
        return torch.sqrt(m / 2.0) * self.s.scalebroad

    def phase(self, q, cells):
        """exp(2 pi i n(q).m/N), q (...), cells (K,3) -> (...,K)."""
        out = 1.0
        for d in range(3):
            x = torch.remainder(self.ijk[q][..., d, None] * cells[:, d], self.n[d]).double() * (2.0 * np.pi / self.n[d])
            out = out * torch.complex(torch.cos(x), torch.sin(x))
        return out

    def bose(self, T):
        return 1.0 / (torch.exp(HBAR * self.w / KB / T) - 1.0)


def _classes(s, ifc):
    """Clusters grouped by the lattice vector between, and the atoms of, their last two sites."""
    cells, at = np.asarray(ifc.cells), np.asarray(ifc.atoms) - 1
    keys = [tuple(cells[-2, c] - cells[-1, c]) + (at[-2, c], at[-1, c]) for c in range(ifc.ntri)]
    uniq = sorted(set(keys))
    cls = np.array([uniq.index(k) for k in keys])
    mass = np.asarray(s.crystal.masses)[np.asarray(s.crystal.types) - 1]
    mu = 1.0 / np.sqrt(np.prod(mass[at], axis=0))
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV)  # noqa: E731
    u = np.array(uniq, np.int64).reshape(-1, 5)
    shape = (ifc.ntri,) + (3,) * ifc.order
    phi = np.transpose(np.asarray(ifc.phi).reshape(shape), (0,) + tuple(range(ifc.order, 0, -1)))
    return dict(cls=t(cls), D=t(u[:, :3]), a=u[:, 3], b=u[:, 4], mu=t(mu), cells=t(cells.astype(np.int64)),
                at=at, phi=t(phi), n=len(uniq))


def _tabs4(X, K, q0, qs, ch):
    """Sum over the clusters of each class for first mode q0 and second points qs: (ii,i,j,p,s,r)."""
    conj = (lambda z: z.conj()) if ch == 2 else (lambda z: z)
    sj = -1 if ch == 2 else 1
    mj, ml = K["cells"][0], K["cells"][2]
    kap = X.phase(torch.tensor(q0, device=DEV), -ml) * K["mu"] * X.phase(qs, sj * (mj - ml))
    e0, e1 = X.e[q0], conj(X.e[qs])
    Z = torch.zeros((len(qs), X.nb, X.nb, K["n"], 3, 3), dtype=torch.complex128, device=DEV)
    for c in range(K["phi"].shape[0]):
        a, b = 3 * K["at"][0, c], 3 * K["at"][1, c]
        t = torch.einsum("iu,xjt,utsr->xijsr", e0[:, a:a + 3], e1[:, :, b:b + 3], K["phi"][c].to(torch.complex128))
        Z[:, :, :, int(K["cls"][c])] += kap[:, c][:, None, None, None, None] * t
    return Z


def _enum4(X, q0, qs, ch):
    """Surviving processes of (q0, the points qs, ch): (x, i, j, q'', k, l, q''', sigma, delta) with x indexing qs."""
    nb, w = X.nb, X.w
    ar = torch.arange(X.nptk, device=DEV)
    sj, sk = (-1 if ch == 2 else 1), (1 if ch == 0 else -1)
    ss = X.wrap(X.ijk[q0] + sj * X.ijk[qs][:, None] + sk * X.ijk[ar][None])  # (x, jj)
    keep = torch.ones_like(ss, dtype=torch.bool)
    if ch != 1:
        keep &= ar[None] >= qs[:, None]
    if ch != 0:
        keep &= ss >= ar[None]
    x, jj = keep.nonzero(as_tuple=True)
    ss = ss[x, jj]
    sig = X.sigma(X.v[jj][:, :, None] - X.v[ss][:, None, :])  # (P, k, l)
    w2, w3, wi, wj = w[jj][:, :, None], w[ss][:, None, :], w[q0], w[qs[x]]
    sv = wi[None, :, None] - wj[:, None] if ch == 2 else wi[None, :, None] + wj[:, None]  # (P, i, j)
    sv = sv[..., None, None]
    d = (sv + w2[:, None, None] if ch == 0 else sv - w2[:, None, None]) - w3[:, None, None]
    ok = (d.abs() <= sig[:, None, None]) & ((w2 != 0) & (w3 != 0))[:, None, None]
    ok &= ((wi != 0) & (wi <= X.s.omega_max))[None, :, None, None, None] & (wj != 0)[:, None, :, None, None]
    p, i, j, k, l = ok.nonzero(as_tuple=True)
    x, jj, ss, ii = x[p], jj[p], ss[p], qs[x[p]]
    good = torch.ones_like(p, dtype=torch.bool)
    if ch != 1:
        good &= (jj != ii) | (k >= j)
    if ch != 0:
        good &= (ss != jj) | (l >= k)
    if ch == 1:
        good &= ((jj != q0) | (i != k)) & ((ss != q0) | (i != l)) & ((ii != jj) | (j != k)) & ((ii != ss) | (j != l))
    out = [a[good] for a in (x, i, j, jj, k, l, ss)]
    p = p[good]
    return out + [sig[p, out[4], out[5]], d[p, out[1], out[2], out[4], out[5]]]


def _weights4(X, bose, q0, ii, ch, i, j, jj, k, l, ss, sig, dl):
    """Gaussian and Bose weight of each process at each temperature, (nT, n)."""
    sp = np.sqrt(np.pi)
    sg = torch.where(sig <= float(np.float32(0.001)), torch.full_like(sig, 1.0 / sp), sig)
    w0, w1, w2, w3 = X.w[q0, i], X.w[ii, j], X.w[jj, k], X.w[ss, l]
    base = torch.exp(-(dl * dl) / (sg * sg)) / sg / sp / (w0 * w1 * w2 * w3)
    base = torch.where((w1 <= 1.25) | (w2 <= 1.25) | (w3 <= 1.25), torch.zeros_like(base), base)
    out = []
    for b in bose:
        f1, f2, f3 = b[ii, j], b[jj, k], b[ss, l]
        if ch == 0:
            bc = f1 * f2 * (1 + f3) - (1 + f1) * (1 + f2) * f3
        elif ch == 1:
            bc = f1 * (1 + f2) * (1 + f3) - (1 + f1) * f2 * f3
        else:
            bc = (1 + f1) * (1 + f2) * (1 + f3) - f1 * f2 * f3
        out.append(bc * base)
    return torch.stack(out)


def _v4sq(X, K, W, Z, ch, x, i, j, jj, k, l, ss):
    """|V|^2 of each process from the class tables Z and phases W(q'', p)."""
    out = []
    step = max(1, 20_000_000 // (9 * K["n"]))
    a, b = torch.as_tensor(K["a"] * 3, device=DEV), torch.as_tensor(K["b"] * 3, device=DEV)
    r3 = torch.arange(3, device=DEV)
    for o in range(0, len(i), step):
        z = slice(o, o + step)
        u, v = X.e[jj[z], k[z]], X.e[ss[z], l[z]].conj()
        u = u if ch == 0 else u.conj()
        T = Z[x[z], i[z], j[z]] * W[jj[z]][:, :, None, None]
        T = (T * v[:, b[:, None] + r3][:, :, None]).sum(-1)
        V = (T * u[:, a[:, None] + r3]).sum((1, 2))
        out.append(V.real ** 2 + V.imag ** 2)
    return torch.cat(out) if out else X.w.new_zeros(0)


def _exact4(case, s):
    X = _T(s)
    nb, nptk, nT = s.nb, s.nptk, len(s.temperatures)
    rates = case["op"] == "rta4"
    K = _classes(s, s.ifc4) if rates else None
    bose = [X.bose(T) for T in s.temperatures]
    N = torch.zeros((3, s.nmodes), dtype=torch.int64, device=DEV)
    P = torch.zeros((3, s.nmodes), dtype=torch.float64, device=DEV)
    R, Wt = (torch.zeros((3, nT, s.nmodes), dtype=torch.float64, device=DEV) for _ in range(2))
    batch = max(1, 20_000_000 // (nptk * nb ** 4))
    for ch in range(3):
        W = X.phase(torch.arange(nptk, device=DEV), (1 if ch == 0 else -1) * K["D"]) if rates else None
        for ll, q in enumerate(s.wedge.list):
            q0 = int(q) - 1
            for o in range(0, nptk, batch):
                qs = torch.arange(o, min(nptk, o + batch), device=DEV)
                x, i, j, jj, k, l, ss, sig, dl = _enum4(X, q0, qs, ch)
                m = ll * nb + i
                if rates:
                    wp = _weights4(X, bose, q0, qs[x], ch, i, j, jj, k, l, ss, sig, dl)
                    v2 = _v4sq(X, K, W, _tabs4(X, K, q0, qs, ch), ch, x, i, j, jj, k, l, ss)
                    R[ch].index_add_(1, m, wp * v2)
                    Wt[ch].index_add_(1, m, wp)
                else:
                    N[ch].index_add_(0, m, torch.ones_like(m))
                    sg = torch.where(sig <= float(np.float32(0.001)), torch.full_like(sig, np.pi ** -0.5), sig)
                    P[ch].index_add_(0, m, torch.exp(-(dl * dl) / (sg * sg)) / (sg * np.sqrt(np.pi)))
    if not rates:
        return [N[c] for c in range(3)], [P[c] / (float(nptk) ** 3 * nb ** 4) for c in range(3)]
    return _rates4(R / nptk / nptk, Wt / nptk / nptk)


def _rates4(R, Wt):
    R = R * (HBARP ** 2 * np.pi / 8.0 * float(np.float32(3.37617087)) * 1e9)
    names = ("plusplus", "plusminus", "minusminus")
    out = {"rate_" + n: R[c] for c, n in enumerate(names)}
    out.update({"wp4_" + n: Wt[c] for c, n in enumerate(names)})
    out["rate_4ph"] = R.sum(0)
    return out


M64 = (1 << 64) - 1


def _signed(x):
    x &= M64
    return x - (1 << 64) if x >> 63 else x


def _mix(z):
    """splitmix64's output function on int64 tensors holding 64-bit words."""
    lsr = lambda a, n: (a >> n) & ((1 << (64 - n)) - 1)  # noqa: E731
    z = z + _signed(0x9E3779B97F4A7C15)
    z = (z ^ lsr(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ lsr(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ lsr(z, 31)


def _pick(base, k, rng):
    """High 64 bits of the k-th word times rng."""
    z = _mix(base + k)
    hi, lo = (z >> 32) & 0xFFFFFFFF, z & 0xFFFFFFFF
    return (hi * rng + ((lo * rng) >> 32)) >> 32


def _exact_sample4(case, s, seed):
    """The sampled rates from the same stream of draws."""
    X, K = _T(s), _classes(s, s.ifc4)
    nb, nptk, ns, nT = s.nb, s.nptk, case["samples"], len(s.temperatures)
    bose = [X.bose(T) for T in s.temperatures]
    R, Wt = (torch.zeros((3, nT, s.nmodes), dtype=torch.float64, device=DEV) for _ in range(2))
    it = torch.arange(ns, device=DEV)
    allq = torch.arange(nptk, device=DEV)
    for ch in range(3):
        sj, sk = (-1 if ch == 2 else 1), (1 if ch == 0 else -1)
        W = X.phase(allq, sk * K["D"])
        for ll, q in enumerate(s.wedge.list):
            q0 = int(q) - 1
            found = []
            for i in range(nb):
                m = ll * nb + i
                w0 = float(s.energy[q0, i])
                if w0 == 0.0 or w0 > s.omega_max:
                    continue
                base = _mix(_mix(it + ((m * 3 + ch) << 32)) ^ seed)
                ii, j = _pick(base, 0, nptk), _pick(base, 1, nb)
                jj, k, l = _pick(base, 2, nptk), _pick(base, 3, nb), _pick(base, 4, nb)
                ss = X.wrap(X.ijk[q0] + sj * X.ijk[ii] + sk * X.ijk[jj])
                ok = torch.ones_like(ii, dtype=torch.bool)
                if ch != 1:
                    ok &= (jj >= ii) & ((jj != ii) | (k >= j))
                if ch != 0:
                    ok &= (ss >= jj) & ((ss != jj) | (l >= k))
                if ch == 1:
                    ok &= ((jj != q0) | (i != k)) & ((ss != q0) | (i != l)) & ((ii != jj) | (j != k)) & (
                        (ii != ss) | (j != l))
                w1, w2, w3 = X.w[ii, j], X.w[jj, k], X.w[ss, l]
                ok &= (w1 != 0) & (w2 != 0) & (w3 != 0)
                sig = X.sigma(X.v[jj, k] - X.v[ss, l])
                sv = w0 - w1 if ch == 2 else w0 + w1
                dl = (sv + w2 if ch == 0 else sv - w2) - w3
                ok &= dl.abs() <= sig
                o = ok.nonzero(as_tuple=True)[0]
                found.append([torch.full_like(o, i)] + [a[o] for a in (ii, j, jj, k, l, ss, sig, dl)])
            if not found:
                continue
            i, ii, j, jj, k, l, ss, sig, dl = (torch.cat(a) for a in zip(*found))
            wp = _weights4(X, bose, q0, ii, ch, i, j, jj, k, l, ss, sig, dl)
            v2 = torch.zeros_like(sig)
            order = torch.argsort(ii)
            step = max(1, 100_000_000 // (nb * nb * 9 * K["n"]))
            for o in range(0, nptk, step):  # class tables of a range of second points at a time
                sel = order[(ii[order] >= o) & (ii[order] < o + step)]
                if len(sel) == 0:
                    continue
                Z = _tabs4(X, K, q0, torch.arange(o, min(nptk, o + step), device=DEV), ch)
                v2[sel] = _v4sq(X, K, W, Z, ch, ii[sel] - o, i[sel], j[sel], jj[sel], k[sel], l[sel], ss[sel])
            R[ch].index_add_(1, ll * nb + i, wp * v2)
            Wt[ch].index_add_(1, ll * nb + i, wp)
    total = float(nb) ** 3 * float(nptk) ** 2
    return _rates4(R / nptk / nptk / ns * total, Wt / nptk / nptk / ns * total)


def _kappa(s, F):
    """TConduct from F (3,nptk,nb)."""
    T = s.temperatures[0]
    with np.errstate(divide="ignore", invalid="ignore"):
        f = 1.0 / (np.exp(HBAR * s.energy / KB / T) - 1.0)
        c = (f * (f + 1.0) * s.energy)[1:]
    kap = np.einsum("qn,qna,bqn->ban", c, s.velocity[1:], F[:, 1:])
    return (float(np.float32(1e21)) * HBAR ** 2 / (KB * T * T * s.volume * s.nptk) * kap).ravel()


def _exact_bte3(s):
    X, K = _T(s), _classes(s, s.ifc3)
    nb, nptk, T = s.nb, s.nptk, s.temperatures[0]
    bose, sp = X.bose(T), np.sqrt(np.pi)
    ar = torch.arange(nptk, device=DEV)
    unit = float(np.float32(5.60626442)) * 1e8
    out = {k + c: [] for k in ("rate_", "wp3_", "n_", "p_") for c in ("plus", "minus")}
    proc = {"plus": [], "minus": []}
    a, b = torch.as_tensor(K["a"] * 3, device=DEV), torch.as_tensor(K["b"] * 3, device=DEV)
    r3 = torch.arange(3, device=DEV)
    for c, sg in (("plus", 1), ("minus", -1)):
        W = X.phase(ar, sg * K["D"])
        for q in s.wedge.list:
            q0 = int(q) - 1
            ss = X.wrap(X.ijk[q0] + sg * X.ijk)
            kap = X.phase(torch.tensor(q0, device=DEV), -K["cells"][1]) * K["mu"]
            sig = X.sigma(X.v[:, :, None] - X.v[ss][:, None, :])  # (q', j, k)
            w1, w2 = X.w[:, :, None], X.w[ss][:, None, :]
            for i in range(nb):
                w0 = X.w[q0, i]
                d = (w0 + w1 if sg > 0 else w0 - w1) - w2
                ok = (d.abs() <= 2.0 * sig) & (w1 != 0) & (w2 != 0) & (w0 != 0) & (w0 <= s.omega_max)
                j, ii, k = ok.permute(1, 0, 2).nonzero(as_tuple=True)
                qq, sgm, dl = ss[ii], sig[ii, j, k], d[ii, j, k]
                g = torch.exp(-(dl * dl) / (sgm * sgm))
                f1, f2 = bose[ii, j], bose[qq, k]
                wp = (f1 - f2 if sg > 0 else f1 + f2 + 1.0) * g / sgm / sp / (w0 * X.w[ii, j] * X.w[qq, k])
                Z = torch.zeros((K["n"], 3, 3), dtype=torch.complex128, device=DEV)
                e0 = X.e[q0, i][torch.as_tensor(3 * K["at"][0], device=DEV)[:, None] + r3]
                Z.index_add_(0, K["cls"], kap[:, None, None] * torch.einsum("ct,ctsr->csr", e0, K["phi"].to(e0.dtype)))
                u, v = X.e[ii, j], X.e[qq, k].conj()
                u = u if sg > 0 else u.conj()
                v2 = []
                for o in range(0, len(j), 20000):
                    z = slice(o, o + 20000)
                    t = torch.einsum("npr,psr->nps", v[z][:, b[:, None] + r3], Z) * u[z][:, a[:, None] + r3]
                    V = (t.sum(-1) * W[ii[z]]).sum(-1)
                    v2.append(V.real ** 2 + V.imag ** 2)
                v2 = torch.cat(v2) if v2 else dl
                gam = HBARP * np.pi / 4.0 * wp * v2 * unit / nptk
                proc[c].append((ii, j, qq, k, gam))
                out["rate_" + c].append(gam.sum() * (1.0 if sg > 0 else 0.5))
                out["wp3_" + c].append(wp.sum() / nptk * (1.0 if sg > 0 else 0.5))
                out["n_" + c].append(torch.tensor(len(j), dtype=torch.int32))
                out["p_" + c].append((g / sgm / sp).sum() / float(nptk) ** 2 / nb ** 3)
    out = {key: torch.stack(v) for key, v in out.items()}
    out["rate"] = out["rate_plus"] + out["rate_minus"]
    # one Jacobi sweep from the RTA iterate, the site symmetrizers, TConduct
    w, tau = s.wedge, torch.where(out["rate"] != 0, 1.0 / out["rate"], torch.zeros_like(out["rate"]))
    F0 = torch.zeros((3, nptk, nb), dtype=torch.float64, device=DEV)
    eq = torch.as_tensor(np.asarray(w.id_equi) - 1, device=DEV).long()
    star = [(torch.as_tensor(w.allequi[ll, :w.nequi[ll]] - 1, device=DEV).long(),
             torch.as_tensor(w.typeofsym[ll, :w.nequi[ll]] - 1, device=DEV).long()) for ll in range(s.nlist)]
    for m in range(s.nmodes):
        qs, i = star[m // nb][0], m % nb
        F0[:, qs, i] = tau[m] * (X.v[qs, i] * X.w[qs, i][:, None]).T
    F = F0.clone()
    for m in range(s.nmodes):
        (qs, op), i = star[m // nb], m % nb
        for c, f, sgn in (("plus", 1.0, -1.0), ("minus", 0.5, 1.0)):
            y, j, x, k, g = proc[c][m]
            d = F0[:, eq[op[:, None], x[None]], k] + sgn * F0[:, eq[op[:, None], y[None]], j]
            F[:, qs, i] += tau[m] * f * (d * g).sum(-1)
    F = torch.einsum("qab,bqn->aqn", torch.as_tensor(s.sym.symmetrizers, device=DEV), F)
    out["F"], out["kappa"] = F.reshape(-1), _kappa(s, F.cpu().numpy())
    return out


def _exact_iter(state):
    """The in-order sweep, its symmetrisation and TConduct in numpy."""
    s, nb, nptk = state["solve"], state["solve"].nb, state["solve"].nptk
    L, w, sym = state["lists"], s.wedge, s.sym.symmetrizers
    F = state["F0"].reshape(3, nptk, nb).copy()
    off = {"plus": np.concatenate([[0], np.cumsum(state["n_p"], dtype=np.int64)]),
           "minus": np.concatenate([[0], np.cumsum(state["n_m"], dtype=np.int64)])}
    for ll, i in itertools.product(range(s.nlist), range(nb)):
        m = ll * nb + i
        parts = []
        for c, f in (("plus", 1.0), ("minus", 0.5)):
            z = slice(off[c][m], off[c][m + 1])
            y, x = L["ind2_" + c][z] - 1, L["ind3_" + c][z] - 1
            parts.append((y // nb, y % nb, x // nb, x % nb, f * L["gamma_" + c][z], -1.0 if c == "plus" else 1.0))
        for kk in range(w.nequi[ll]):
            qq, op = w.allequi[ll, kk] - 1, w.typeofsym[ll, kk] - 1
            acc = np.zeros(3)
            for qy, by, qx, bx, g, sgn in parts:
                acc += ((F[:, w.id_equi[op, qx] - 1, bx] + sgn * F[:, w.id_equi[op, qy] - 1, by]) * g).sum(1)
            F[:, qq, i] = state["tau"][m] * (s.velocity[qq, i] * s.energy[qq, i] + acc)
            F[:, qq, :] = sym[qq] @ F[:, qq, :]
    F = np.einsum("qab,bqn->aqn", sym, F)
    return {"F": F.ravel(), "kappa": _kappa(s, F)}


def exact(case, seed):
    nptk, nb, nlist = _sizes(case)
    if case["op"] in ("rta4", "np4"):  # candidates that plain torch can look through in a few seconds
        if nlist * float(nptk) ** 2 * nb ** 4 > (2.5e10 if case["op"] == "np4" else 1.2e10):
            return None
        return _exact4(case, _solve(case, seed))
    if case["op"] == "sample4":
        return _exact_sample4(case, _solve(case, seed), seed) if nb * nlist * case["samples"] < 1e8 else None
    if case["op"] == "bte3":
        return _exact_bte3(_solve(case, seed))
    return _exact_iter(prepare(case, seed))
