"""The calls that a user of the impurity solver makes, at the sizes they are made.

Every case goes through the package's public entry points (`Solver`, `Server`,
`serve`).  Sizes are those of the repository's workloads (configs.py, bench.py,
tests): 5 to 16 sites, all sectors or the ones near half filling, up to 300
Lanczos steps, 2048 Matsubara frequencies; one and two orbitals.

  hx       y = H x (or y += H x) of one sector on device vectors: what a
           caller with its own eigensolver applies, the unit of every path
  solve    a DMFT iteration's impurity solve: a new bath (set_model), the
           ground state over the sectors, G_cl on the Matsubara grid
  ground   the ground-state energies of one or more sectors of a new bath
  batch    many independent instances in one call (parameter sweeps,
           inequivalent sites of a lattice)
  serve    requests of mixed sizes, all queued at once, through the served form
  arpack   the lowest eigenpairs by the restarted Lanczos (diag_solver 2)

A program holds one solver for its run and gives it a new model per DMFT
iteration, so the whole calls share one solver and set the model inside the
pass; hx and arpack hold the model set, as a caller's iteration does.
"""

from __future__ import annotations

import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_DIR = os.path.join(ROOT, "dmft-ed-zt_b200")


def _pkg():
    name = "dmft_ed_zt_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(PKG_DIR, "__init__.py"),
                                                      submodule_search_locations=[PKG_DIR])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


_shared = None


def _solver():
    """The program's one solver."""
    global _shared
    if _shared is None:
        _shared = _pkg().Solver(0)
    return _shared


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
# Lanczos steps at which the ground state of a sector has converged, by sites:
# a solve takes these.  Further steps only add copies of converged states to
# the tridiagonal matrix, and rounding then sets the digits of the ground
# state, and of G, beyond the ninth; energies alone hold at any step count.
STEPS = {1: {5: 30, 6: 40, 7: 45, 8: 60, 9: 70, 10: 85, 11: 100, 12: 130, 13: 150}, 2: {6: 30, 8: 40, 10: 55}}


def listed():
    return [
        # one H.v of a small sector (4,900 states): launches and host path
        dict(name="hx_n8", kind="hx", norb=1, nsite=8, nu=4, nd=4, acc=0),
        # an odd, unequal sector with the accumulating form (2.2 M states)
        dict(name="hx_n13_add", kind="hx", norb=1, nsite=13, nu=7, nd=5, acc=1),
        # two orbitals with spin-flip and pair-hopping terms (853,776 states)
        dict(name="hx_2orb_n12", kind="hx", norb=2, nsite=12, nu=6, nd=6, acc=0),
        # the largest sector one solver takes (165.6 M states)
        dict(name="hx_n16", kind="hx", norb=1, nsite=16, nu=8, nd=8, acc=0),
        # the small single-orbital solve, every sector: latency of a whole DMFT iteration
        dict(name="solve_n6", kind="solve", norb=1, nsite=6, every=1, steps=40, nw=2048, nspin=1),
        # the two-orbital Kanamori solve
        dict(name="solve_2orb_n10", kind="solve", norb=2, nsite=10, every=0, steps=55, nw=2048, nspin=1),
        # the headline model's solve: 12 sites, 9 sectors
        dict(name="solve_n12", kind="solve", norb=1, nsite=12, every=0, steps=130, nw=2048, nspin=1),
        # an odd number of sites, both spins
        dict(name="solve_n13", kind="solve", norb=1, nsite=13, every=0, steps=150, nw=2048, nspin=2),
        # the headline scan: 9 sectors of 12 sites, 300 steps
        dict(name="ground_n12", kind="ground", norb=1, nsite=12, nu=0, nd=0, steps=300),
        # the largest eigenvalue problem of a few tenths of a second (41.4 M states)
        dict(name="ground_n15", kind="ground", norb=1, nsite=15, nu=7, nd=8, steps=300),
        # a sweep of 16 instances of 8 to 11 sites
        dict(name="batch_16", kind="batch", count=16, lo=8, hi=11, steps=60, nw=2048, nspin=2),
        # 8 queued requests of 8 to 12 sites
        dict(name="serve_8", kind="serve", count=8, lo=8, hi=12, steps=60, nw=2048, nspin=2),
    ]


def draw(rng):
    kind = rng.choice(["hx", "hx", "hx", "solve", "solve", "ground", "batch", "serve", "arpack"])
    nw = int(round(math.exp(rng.uniform(math.log(200), math.log(4000)))))
    if kind == "hx":
        norb = rng.choice([1, 1, 2])
        ns = rng.randint(5, 16 if norb == 1 else 13)
        spread = 2 if ns >= 8 else 1
        return dict(kind=kind, norb=norb, nsite=ns, nu=ns // 2 + rng.randint(-spread, spread),
                    nd=ns // 2 + rng.randint(-spread, spread), acc=rng.randint(0, 1))
    if kind == "solve":
        norb = rng.choice([1, 1, 2])
        ns = rng.choice(sorted(STEPS[norb]))
        steps = rng.randint(STEPS[norb][ns] * 2 // 3, STEPS[norb][ns])
        return dict(kind=kind, norb=norb, nsite=ns, every=1 if ns <= 7 and norb == 1 else 0, steps=steps, nw=nw,
                    nspin=rng.randint(1, 2))
    if kind == "ground":     # nu = nd = 0: every sector near half filling
        ns = rng.randint(8, 14)
        scan = ns <= 12 and rng.randint(0, 1)
        return dict(kind=kind, norb=1, nsite=ns, nu=0 if scan else ns // 2 + rng.randint(-1, 1),
                    nd=0 if scan else ns // 2 + rng.randint(-1, 1), steps=rng.randint(100, 300))
    if kind == "arpack":
        ns = rng.randint(7, 10)
        return dict(kind=kind, norb=1, nsite=ns, nu=ns // 2, nd=ns // 2 + rng.randint(0, 1))
    lo = rng.randint(6, 9)
    return dict(kind=kind, count=rng.randint(3, 16), lo=lo, hi=rng.randint(lo + 1, 11),
                steps=rng.randint(STEPS[1][lo] * 2 // 3, STEPS[1][lo]), nw=nw, nspin=rng.randint(1, 2))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
BETA = 100.0


def _params(norb, nsite, rng):
    """A random impurity model: bath levels U(-2, 2), couplings U(0.1, 1),
    the same for both spins; two orbitals with their own baths and Hund's
    coupling J = U / 4 (Kanamori)."""
    nbath = nsite - norb
    U = float(rng.uniform(2.0, 3.0))
    ek = rng.uniform(-2.0, 2.0, nbath)
    v = rng.uniform(0.1, 1.0, nbath)
    vmk = np.zeros((norb, nbath, 2))
    for l in range(nbath):
        vmk[l * norb // nbath, l, :] = v[l]
    J = U / 4 if norb > 1 else 0.0
    mu = U / 2 + (norb - 1) * (2 * (U - 2 * J) - J) / 2
    return dict(norb=norb, nbath=nbath, em=np.zeros((norb, 2)), ek=np.stack([ek, ek], 1), vmk=vmk, U=U, J=J, mu=mu)


def _model(p):
    return _pkg().Model(p["norb"], p["nbath"], p["em"], p["ek"], p["vmk"], U=p["U"], Jex=p["J"], mu=p["mu"])


def _sectors(norb, nsite, every):
    if every:
        return [(u, d) for u in range(nsite + 1) for d in range(nsite + 1)]
    if norb > 1:     # fixed total filling, all spin projections near zero
        return [(u, nsite - u) for u in range(nsite // 2 - 2, nsite // 2 + 3)]
    half = [nsite // 2 - 1, nsite // 2, nsite // 2 + 1] if nsite % 2 == 0 else [nsite // 2, nsite // 2 + 1]
    return [(u, d) for u in half for d in half]


def _case_sectors(case):
    if case["kind"] == "solve":
        return _sectors(case["norb"], case["nsite"], case["every"])
    return [(case["nu"], case["nd"])] if case["nu"] else _sectors(1, case["nsite"], 0)


def _omega(nw):
    return (2.0 * np.arange(nw, dtype=np.float64) + 1.0) * np.pi / BETA


def _instances(case, rng):
    out = []
    for _ in range(case["count"]):
        ns = int(rng.integers(case["lo"], case["hi"] + 1))
        out.append(dict(p=_params(1, ns, rng), nsite=ns, sectors=_sectors(1, ns, 0), nspin=case["nspin"],
                        seed=int(rng.integers(1 << 30))))
    return out


def _vectors(case, seed):
    n = math.comb(case["nsite"], case["nu"]) * math.comb(case["nsite"], case["nd"])
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    x /= x.norm()
    y = torch.randn(n, dtype=torch.float64, device="cuda", generator=g) / math.sqrt(n) if case["acc"] else None
    return x, y


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("batch", "serve"):
        inst = [dict(model=_model(i["p"]), sectors=i["sectors"], nspin=i["nspin"], seed=i["seed"])
                for i in _instances(case, rng)]
        st = dict(case=case, solver=_solver(), instances=inst, omega=_omega(case["nw"]))
        if kind == "serve":
            st["server"] = _pkg().Server(st["solver"], case["steps"], st["omega"])
        return st
    p = _params(case["norb"], case["nsite"], rng)
    st = dict(case=case, model=_model(p), seed=int(rng.integers(1 << 30)))
    if kind == "hx":
        st["solver"] = _pkg().Solver(0)
        st["solver"].set_model(st["model"])
        st["x"], y = _vectors(case, seed)
        st["y"] = torch.empty_like(st["x"]) if y is None else y    # y += H x: the caller's running sum
    elif kind == "arpack":
        st["solver"] = _pkg().Solver(0)
        st["solver"].set_model(st["model"])
    else:
        st["solver"] = _solver()
        st["sectors"] = _case_sectors(case)
        if kind == "solve":
            st["omega"] = _omega(case["nw"])
    return st


def run(st):
    case, s = st["case"], st["solver"]
    kind = case["kind"]
    if kind == "hx":
        return s.hx(case["nu"], case["nd"], st["x"], st["y"], py=bool(case["acc"]))
    if kind == "solve":
        s.set_model(st["model"])
        return s.solve(st["sectors"], case["steps"], st["omega"], nspin=case["nspin"], seed=st["seed"])
    if kind == "ground":
        s.set_model(st["model"])
        r = s.ground_state(st["sectors"], case["steps"], seed=st["seed"], want_vec=False)
        return dict(isector=r["isector"], e0=r["e0"], e_sector=r["e_sector"])
    if kind == "batch":
        return s.solve_batch(st["instances"], case["steps"], st["omega"])
    if kind == "serve":
        done, _, _ = _pkg().serve(st["server"], st["instances"], [0.0] * len(st["instances"]))
        return dict(isector=[r["isector"] for r in done], e0=np.array([r["e0"] for r in done]),
                    G_cl=np.concatenate([r["G_cl"].ravel() for r in done]))
    r = s.diag_arpack(case["nu"], case["nd"], seed=st["seed"], want_resid=False)
    return dict(e0=r["e0"], ritz=r["ritz"], vec=r["vec"])


# ---------------------------------------------------------------------------
# work: a Lanczos step reads the last two vectors and writes the next one
# (24 bytes a state); H x reads x and writes y (16, and y again when it adds);
# a multiplication and an addition per hop, and about ten operations more
# ---------------------------------------------------------------------------
def _dim(nsite, nu, nd):
    if not (0 <= nu <= nsite and 0 <= nd <= nsite):
        return 0
    return math.comb(nsite, nu) * math.comb(nsite, nd)


def _solve_work(norb, nsite, sectors, steps, nspin):
    states = sum(_dim(nsite, u, d) * min(steps, _dim(nsite, u, d)) for u, d in sectors)
    u, d = max(sectors, key=lambda s: _dim(nsite, *s))
    per_spin = [(u + 1, d), (u - 1, d)], [(u, d + 1), (u, d - 1)]
    runs = per_spin[0] + (per_spin[1] if nspin == 2 else [])
    states += norb * sum(_dim(nsite, *r) * min(steps, _dim(nsite, *r)) for r in runs)
    return states


def work(case):
    kind = case["kind"]
    if kind == "hx":
        n = _dim(case["nsite"], case["nu"], case["nd"])
        return dict(bytes=(24.0 if case["acc"] else 16.0) * n, flops=(2.0 * case["nsite"] + 4) * n)
    if kind == "arpack":   # restarts depend on the spectrum: at least 100 of 3 products, 7 vectors read each
        n = _dim(case["nsite"], case["nu"], case["nd"])
        return dict(bytes=300.0 * 72.0 * n, flops=300.0 * (2.0 * case["nsite"] + 20) * n)
    if kind == "solve":
        n = _solve_work(case["norb"], case["nsite"], _case_sectors(case), case["steps"], case["nspin"])
        return dict(bytes=24.0 * n, flops=(2.0 * case["nsite"] + 10) * n)
    if kind == "ground":
        n = sum(_dim(case["nsite"], u, d) for u, d in _case_sectors(case)) * case["steps"]
        return dict(bytes=24.0 * n, flops=(2.0 * case["nsite"] + 10) * n)
    mid = (case["lo"] + case["hi"]) / 2
    sizes = range(case["lo"], case["hi"] + 1)
    n = case["count"] / len(sizes) * sum(_solve_work(1, q, _sectors(1, q, 0), case["steps"], case["nspin"])
                                         for q in sizes)
    return dict(bytes=24.0 * n, flops=(2.0 * mid + 10) * n)


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Sector:
    """H of one sector as gathers over the strings of each spin."""

    def __init__(self, p, nu, nd):
        self.p, self.nu, self.nd = p, nu, nd
        self.norb, self.ns = p["norb"], p["norb"] + p["nbath"]
        self.up, self.dn = self._spin(nu, 0), self._spin(nd, 1)
        self.n = self.up["count"] * self.dn["count"]
        P = 1 << self.norb
        U, J = p["U"], p["J"]
        Up = U - 2 * J
        w = np.zeros((P, P))
        occ = lambda q, a: (q >> a) & 1  # noqa: E731
        for pu in range(P):
            for pd in range(P):
                for a in range(self.norb):
                    w[pd, pu] += U * occ(pu, a) * occ(pd, a)
                    for b in range(a + 1, self.norb):
                        w[pd, pu] += (Up - J) * (occ(pu, a) * occ(pu, b) + occ(pd, a) * occ(pd, b))
                        w[pd, pu] += Up * (occ(pu, a) * occ(pd, b) + occ(pd, a) * occ(pu, b))
        w = torch.from_numpy(w).cuda()
        self.w = w
        self.exchange = []
        if J != 0.0:
            for pu in range(P):
                for pd in range(P):
                    for i in range(self.norb):
                        for j in range(self.norb):
                            if i == j:
                                continue
                            par = sum(occ(pu, k) + occ(pd, k) for k in range(min(i, j), max(i, j)))
                            s = -1.0 if par & 1 else 1.0
                            if not occ(pu, i) and occ(pu, j) and not occ(pd, j) and occ(pd, i):
                                self._exchange(pu, pd, pu ^ (1 << i) ^ (1 << j), pd ^ (1 << i) ^ (1 << j), -s * J)
                            if not occ(pu, i) and not occ(pd, i) and occ(pu, j) and occ(pd, j):
                                self._exchange(pu, pd, pu ^ (1 << i) ^ (1 << j), pd ^ (1 << i) ^ (1 << j), s * J)

    def _spin(self, n, s):
        p, ns, norb = self.p, self.ns, self.norb
        t = np.arange(1 << ns, dtype=np.int64)
        bits = ((t[:, None] >> np.arange(ns)) & 1).astype(np.int8)
        t = t[bits.sum(1) == n]
        rank = np.full(1 << ns, -1, dtype=np.int64)
        rank[t] = np.arange(t.size)
        lv = np.concatenate([p["em"][:, s] - p["mu"], p["ek"][:, s]])
        e1 = (((t[:, None] >> np.arange(ns)) & 1) * lv).sum(1)
        hops = []
        for a in range(norb):
            for l in range(p["nbath"]):
                v, j = p["vmk"][a, l, s], norb + l
                if v == 0.0:
                    continue
                ok = ((t >> a) & 1) != ((t >> j) & 1)
                between = t & (((1 << j) - 1) & ~((2 << a) - 1))
                sign = np.where(sum((between >> q) & 1 for q in range(ns)) & 1, -1.0, 1.0)
                tgt = np.where(ok, rank[np.where(ok, t ^ (1 << a) ^ (1 << j), t)], 0)
                hops.append((torch.from_numpy(tgt).cuda(), torch.from_numpy(np.where(ok, sign * v, 0.0)).cuda()))
        return dict(count=t.size, str=t, rank=rank, e1=torch.from_numpy(e1).cuda(), hops=hops,
                    imp=torch.from_numpy(t & ((1 << norb) - 1)).cuda())

    def _exchange(self, pu, pd, pu2, pd2, c):
        P1 = (1 << self.norb) - 1
        cols = [(i, self.up["rank"][(q & ~P1) | pu2]) for i, q in enumerate(self.up["str"]) if q & P1 == pu]
        rows = [(i, self.dn["rank"][(q & ~P1) | pd2]) for i, q in enumerate(self.dn["str"]) if q & P1 == pd]
        if cols and rows:
            c1, c2 = (torch.tensor([v[k] for v in cols], device="cuda") for k in (0, 1))
            r1, r2 = (torch.tensor([v[k] for v in rows], device="cuda") for k in (0, 1))
            self.exchange.append((r1, c1, r2, c2, c))

    def hx(self, x):
        x = x.view(self.dn["count"], self.up["count"])
        y = self.w[self.dn["imp"]][:, self.up["imp"]]
        y += self.up["e1"][None, :]
        y += self.dn["e1"][:, None]
        y *= x
        for tgt, v in self.up["hops"]:
            y += x.index_select(1, tgt).mul_(v[None, :])
        for tgt, v in self.dn["hops"]:
            y += x.index_select(0, tgt).mul_(v[:, None])
        for r1, c1, r2, c2, c in self.exchange:
            y[r1[:, None], c1[None, :]] += c * x[r2[:, None], c2[None, :]]
        return y.reshape(-1)

    def dense(self):
        eye = torch.eye(self.n, dtype=torch.float64, device="cuda")
        return torch.stack([self.hx(eye[i].contiguous()) for i in range(self.n)])

    def lanczos(self, v, steps, keep):
        """alpha, beta (and the basis, fully reorthogonalised, when kept)."""
        a, b, V = [], [], []
        w, prev, bk = v / v.norm(), None, 0.0
        for k in range(min(steps, self.n)):
            if keep:
                V.append(w)
            y = self.hx(w)
            if prev is not None:
                y -= bk * prev
            a.append(float(w @ y))
            y -= a[-1] * w
            if keep:
                for _ in range(2):
                    for q in V:
                        y -= (q @ y) * q
            bk = float(y.norm())
            if bk < 1e-10 or k + 1 == min(steps, self.n):
                break
            b.append(bk)
            prev, w = w, y / bk
        T = np.diag(a) + np.diag(b[: len(a) - 1], 1) + np.diag(b[: len(a) - 1], -1)
        th, z = np.linalg.eigh(T)
        return th, z, V

    def ground(self, steps, want_vec=True):
        if self.n <= 1000:
            e, z = np.linalg.eigh(self.dense().cpu().numpy())
            return float(e[0]), torch.from_numpy(np.ascontiguousarray(z[:, 0])).cuda()
        v = torch.rand(self.n, dtype=torch.float64, device="cuda",
                       generator=torch.Generator(device="cuda").manual_seed(1))
        keep = want_vec and self.n * steps * 8 <= 20e9
        th, z, V = self.lanczos(v, steps, keep)
        vec = None
        if keep:
            vec = sum(float(c) * q for c, q in zip(z[:, 0], V))
            vec /= vec.norm()
        return float(th[0]), vec

    def excited(self, vec, create, orb, spin):
        """c^+ or c of an orbital on a vector, and the sector it is in (None: empty)."""
        d = 1 if create else -1
        nu, nd = self.nu + (d if spin == 0 else 0), self.nd + (d if spin == 1 else 0)
        if not (0 <= nu <= self.ns and 0 <= nd <= self.ns):
            return None, None
        out = _Sector(self.p, nu, nd)
        side, mine = (out.up, self.up) if spin == 0 else (out.dn, self.dn)
        t = side["str"]
        ok = ((t >> orb) & 1) == (1 if create else 0)
        below = t & ((1 << orb) - 1)
        sign = np.where(sum((below >> q) & 1 for q in range(self.ns)) & 1, -1.0, 1.0)
        src = torch.from_numpy(np.where(ok, mine["rank"][np.where(ok, t ^ (1 << orb), mine["str"][0])], 0)).cuda()
        cf = torch.from_numpy(np.where(ok, sign, 0.0)).cuda()
        x = vec.view(self.dn["count"], self.up["count"])
        y = x.index_select(1, src) * cf[None, :] if spin == 0 else x.index_select(0, src) * cf[:, None]
        if spin == 1:      # the down operator passes every up electron
            y = y * (-1.0 if self.nu & 1 else 1.0)
        return out, y.reshape(-1).contiguous()


def _exact_solve(p, nsite, sectors, steps, omega, nspin):
    best, e0, vec, sec = -1, math.inf, None, None
    for i, (u, d) in enumerate(sectors):
        S = _Sector(p, u, d)
        e, v = S.ground(steps)
        if best < 0 or e < e0 - 1e-10 * max(1.0, abs(e0)):
            best, e0, vec, sec = i, e, v, S
    even = nspin == 1 and sec.nu == sec.nd
    G = np.zeros((2, p["norb"], omega.size), dtype=complex)
    for orb in range(p["norb"]):
        for spin in range(1 if even else 2):
            for create in (True, False):
                out, phi = sec.excited(vec, create, orb, spin)
                if out is None or float(phi.norm()) == 0.0:
                    continue
                th, z, _ = out.lanczos(phi, steps, out.n * steps * 8 <= 20e9)
                wt = float(phi @ phi) * z[0] ** 2
                pole = (e0 - th) if create else (th - e0)
                G[spin, orb] += (wt[None, :] / (1j * omega[:, None] + pole[None, :])).sum(1)
    if nspin == 1:
        G = G[:1] if even else 0.5 * (G[:1] + G[1:])
    return best, e0, G


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve", "arpack"):     # instances of other sizes stop short of convergence at one step count
        return None
    rng = np.random.default_rng(seed)
    p = _params(case["norb"], case["nsite"], rng)
    if kind == "hx":
        x, y = _vectors(case, seed)
        h = _Sector(p, case["nu"], case["nd"]).hx(x)
        return h if y is None else h.add_(y)
    if kind == "solve":
        _, e0, G = _exact_solve(p, case["nsite"], _case_sectors(case), case["steps"], _omega(case["nw"]),
                                case["nspin"])
        return dict(isector=None, e0=e0, G_cl=G)
    e = np.array([_Sector(p, u, d).ground(case["steps"], want_vec=False)[0] for u, d in _case_sectors(case)])
    return dict(isector=None, e0=float(e.min()), e_sector=e)
