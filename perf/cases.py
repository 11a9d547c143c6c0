"""Timed cases of the solver: what a user of the library runs, through its
public entry points.

A case is a dict of plain values; ``prepare`` builds the solver and the flow
a program has in hand, ``run`` makes one pass, ``work`` counts what the pass
cannot do without, ``exact`` restates the Roe iteration in plain float64
torch.  Kinds of case:

  march     n pseudo-time iterations from a given flow (``CodeNS.atsch_num``):
            boxes, bump channels and batches of independent boxes; Euler and
            Navier-Stokes; the flux families; FP64 and mixed precision
  rans      the same on a flat plate with the Spalart-Allmaras step
  host      one iteration on a pinned host state (copy in, advance, copy out)
  routines  one iteration of a driver that calls the reference's routines
            itself, block by block, on device arrays
  adjoint   the transposed residual and the transposed implicit phase of one
            adjoint iteration
"""
import math

import numpy as np
import torch

from codens_b200 import CodeNS, cases

LMAX = 10


def listed():
    return [
        # the smallest grids (a deck being set up, a unit check): launch latency
        _march("box", (16, 12, 8), 0, 0, 10, name="tiny box Euler FP64"),
        # the 64x32x32 box as its three sub-runs: Roe, Jameson, limited viscous
        _march("box", (64, 32, 32), 0, 0, 10, name="box 64x32x32 Euler Roe FP64"),
        _march("box", (64, 32, 32), 0, 1, 10, flux=1, name="box 64x32x32 Euler Jameson mixed"),
        _march("box", (64, 32, 32), 1, 0, 10, ilim=1, name="box 64x32x32 NS minmod FP64"),
        # a few uneven blocks, odd sizes, limited: an ordinary parity run
        _march("channel", (97, 59, 61), 1, 0, 5, nblk=3, ilim=1, name="channel 1M ragged NS minmod FP64"),
        # a medium run with another flux family
        _march("channel", (83, 57, 45), 1, 1, 5, nblk=2, flux=14, name="channel 0.4M NS HLLC mixed"),
        # production: the eight-block 4.4M-cell bump channel
        _march("channel", (97, 62, 91), 1, 1, 5, nblk=8, name="channel 4.4M NS mixed"),
        # many independent small cases in one layout
        _march("batch", (16, 64, 24), 0, 1, 5, name="batch of 24 boxes Euler mixed"),
        {"name": "flat plate 2.1M SA mixed", "kind": "rans", "n0": 256, "n1": 128, "n2": 64,
         "prec": 1, "steps": 3},
        {"name": "host arrays channel 0.9M NS mixed", "kind": "host", "n0": 96, "n1": 56, "n2": 58,
         "nblk": 3, "prec": 1, "ns": 1, "ilim": 0, "steps": 1},
        {"name": "routine by routine channel 0.5M NS FP64", "kind": "routines", "n0": 75, "n1": 51,
         "n2": 65, "nblk": 2, "prec": 0, "ns": 1, "ilim": 0, "steps": 1},
        {"name": "adjoint products 512x256x4 Euler FP64", "kind": "adjoint", "n0": 512, "n1": 256,
         "n2": 4, "prec": 0, "steps": 1},
    ]


def _march(shape, n, ns, prec, steps, nblk=1, flux=7, ilim=0, name=None):
    c = {"kind": "march", "shape": shape, "n0": n[0], "n1": n[1], "n2": n[2], "nblk": nblk, "ns": ns,
         "prec": prec, "flux": flux, "ilim": ilim, "steps": steps}
    return dict(c, name=name) if name else c


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(cells, lo=8, hi=160):
        """three sides, each over its range in logarithm, of at most `cells` cells"""
        while True:
            n = [log_int(lo, hi) for _ in range(3)]
            if n[0] * n[1] * n[2] <= cells:
                return n

    kind = rng.choice(["box", "box", "channel", "channel", "batch", "rans", "host", "routines", "adjoint"])
    prec, ns = rng.randint(0, 1), rng.randint(0, 1)
    if kind == "box":
        flux = rng.choice([7, 7, 7, 14, 9, 1] if ns else [7, 7, 14, 1])
        return _march("box", box(1_000_000), ns, prec, rng.choice([5, 10]), flux=flux,
                      ilim=ns * rng.randint(0, 1) if flux in (7, 14) else 0)
    if kind == "channel":
        nblk = rng.randint(1, 6)
        return _march("channel", box(1_800_000 // nblk, 12, 140), 1, prec, 5, nblk=nblk,
                      flux=rng.choice([7, 7, 7, 14, 5]), ilim=rng.randint(0, 1))
    if kind == "batch":
        return _march("batch", (rng.randint(10, 20), rng.randint(24, 56), rng.randint(4, 28)), 0, prec, 5)
    if kind == "rans":
        return {"kind": "rans", "n0": log_int(48, 224), "n1": log_int(48, 128), "n2": log_int(4, 64),
                "prec": prec, "steps": 3}
    if kind == "adjoint":
        return {"kind": "adjoint", "n0": log_int(64, 512), "n1": log_int(32, 256), "n2": rng.randint(2, 4),
                "prec": prec, "steps": 1}
    nblk = rng.randint(1, 4)
    n = box((900_000 if kind == "host" else 500_000) // nblk, 12, 120)
    return {"kind": kind, "n0": n[0], "n1": n[1], "n2": n[2], "nblk": nblk, "prec": prec * (kind == "host"),
            "ns": 1, "ilim": rng.randint(0, 1), "steps": 1}


# ---------------------------------------------------------------------------
# the flow of a case
# ---------------------------------------------------------------------------
def _case(c, seed):
    n = (c["n0"], c["n1"], c["n2"])
    if c["kind"] == "rans":
        # a uniform start (the wall spacing takes no noise): the seed is the inflow's
        k = cases.flat_plate_case(n, mach=0.25 + 0.1 * np.random.default_rng(seed).random(), lmax=LMAX)
    elif c["kind"] == "adjoint":
        k = cases.channel_case([n[0]], n[1], n[2], seed=seed, reynz=1.0e12, lmax=LMAX, ilim=0)
        k.scheme.ns, k.scheme.muscl, k.scheme.qfix_dfez = 0, 0, 1
    elif c["kind"] != "march" or c["shape"] == "channel":
        # uneven blocks around n0 cells along the channel
        ni = [max(4, n[0] + (-1) ** b * (b * n[0] // 20)) for b in range(c["nblk"])]
        k = cases.channel_case(ni, n[1], n[2], seed=seed, ilim=c["ilim"], lmax=LMAX)
    elif c["shape"] == "batch":
        # n0..n1: the sides' range, n2: the number of boxes; sides, Mach
        # numbers and angles belong to the case, the noise to the seed
        k = cases.batch_case(n[2], (n[0], n[1]), seed=4, lmax=LMAX, qfix_dfez=1)
        noise = np.random.default_rng(seed).uniform(-0.01, 0.01, k.layout.ld)
        k.v0 *= 1.0 + noise
    else:
        k = cases.box_case(n, seed=seed, ns=bool(c["ns"]), ilim=c["ilim"], lmax=LMAX, skew=0.01,
                           reynz=1.0e4, qfix_dfez=0 if c["ns"] else 1)
    k.scheme.precision = c["prec"]
    k.scheme.ischema = c.get("flux", 7)
    return k


def _tiles(layout, prec):
    """the sweep tiling a program gives instead of having one timed, so that
    every run of a grid takes the same: wide patches of the deepest plane
    count that still leaves a patch for each of 300 resident CTAs"""
    ti, tj = (32, 8) if prec else (16, 8)
    for kc in (16, 8, 4, 2):
        if sum(-(-(b.ni - 1) // ti) * -(-(b.nj - 1) // tj) * -(-(b.nk - 1) // kc) for b in layout.blocks) >= 300:
            break
    return ti, tj, kc


def prepare(case, seed):
    k = _case(case, seed)
    s = CodeNS(k)
    s.metric()
    st = {"kind": case["kind"], "steps": case["steps"], "solver": s, "v0": s.v.clone()}
    if case["kind"] in ("march", "rans", "host"):
        s.set_sweep_tiles(case["prec"], *_tiles(k.layout, case["prec"]))
    if case["kind"] == "rans":
        s.set_sa(s.atcaldis3(), rokinf=k.meta["rokinf"], stilde_fix=1)
    elif case["kind"] == "host":
        st["v_host"] = torch.from_numpy(np.ascontiguousarray(k.v0.reshape(-1))).pin_memory()
    elif case["kind"] == "adjoint":
        s.adjoint_prepare()
        g = torch.Generator(device="cuda").manual_seed(seed)
        real = torch.zeros(s.ld, dtype=torch.float64, device="cuda")
        real[torch.as_tensor(k.layout.real_cells(), device="cuda")] = 1.0
        for a in ("lam", "y"):
            st[a] = (torch.randn(5, s.ld, dtype=torch.float64, device="cuda", generator=g) * real).reshape(-1)
        st["wbar"], st["sbar"], st["out"] = (torch.zeros(m * s.ld, dtype=torch.float64, device="cuda")
                                             for m in (6, 9, 5))
    torch.cuda.synchronize()
    return st


def run(state):
    s = state["solver"]
    if state["kind"] == "host":
        s.atsch_num_host(state["v_host"], state["steps"])
        return {"v": state["v_host"]}
    if state["kind"] == "adjoint":
        s.adjoint_rt(state["lam"], state["wbar"], state["sbar"])
        s.adjoint_lt(state["y"], state["out"])
        return {a: state[a] for a in ("wbar", "sbar", "out")}
    with torch.cuda.stream(s.stream):  # the given flow: the start of a run
        s.v.copy_(state["v0"])
        if state["kind"] == "rans":
            s.mut.zero_()
    if state["kind"] == "routines":
        return _routines(s, state["v0"])
    s.set_cycle(0, 0)
    norms = s.atsch_num(state["steps"])
    # the reduced-precision forms are asked for a state, the FP64 one for its norms too
    return {"v": s.v} if s.case.scheme.precision else {"v": s.v, "norms": norms}


def _routines(s, v0):
    """one iteration as the reference's atsch_num.f90 makes it"""
    lmx = s.case.scheme.lmax
    blocks = range(1, s.case.layout.nblk + 1)
    for l in blocks:
        s.zpres(l, s.v, s.pression, s.ztemp, s.cson)
        s.zvismo(l, s.mu, s.v, s.ztemp)
        s.chronos(l, s.mu, s.mut, s.v, s.dt, s.sn, s.vol, s.cson)
    s.rbord(s.v, s.pression, s.ztemp, s.cson)
    s.zvisqc(s.v, s.mu, s.mut, s.tau, s.sn, s.vol, s.ztemp)
    for l in blocks:
        s.sch_roe(l, s.u, s.v, s.tau, s.sn, s.pression)
        s.implimf_3d(l, s.u, s.dt, s.v, s.d, s.mu, s.mut, s.sn, s.vol, s.pression, s.cson, lmx)
    norms = s.rscpsv(v0, s.v, s.dt)
    return {"v": s.v, "u": s.u, "norms": norms}


def work(case):
    """per iteration and cell: the state read and written, the face areas and
    the volume read (FP64), the turbulent viscosity where there is one; the
    operations of the scheme's own expressions (a Roe face about 650, the
    viscous gradients 250, a Jacobi sweep 450, the rest of an iteration 200)"""
    c = case
    n = c["n0"] * c["n1"] * c["n2"] * c.get("nblk", 1)
    if c.get("shape") == "batch":
        k = cases.batch_case(c["n2"], (c["n0"], c["n1"]), seed=4, noise=0.0)
        n = k.layout.nreal
    if c["kind"] == "adjoint":
        # the Jacobian of the three faces (24 + 3 columns of 5), lambda, y and
        # the products; the transposed sweeps
        return {"bytes": n * 8.0 * (3 * 27 * 5 + 5 + 6 + 9 + 5 + 5 + 9 + 9), "flops": n * (2.0 * 3 * 27 * 5 + LMAX * 250)}
    ns = c.get("ns", 1)
    b = 40 + 40 + 72 + 8 + 8 * ns
    f = 3 * 650 + 250 * ns + 450 * LMAX + 200
    if c["kind"] == "rans":
        b, f = b + 4 * 8 + 8, f + 6 * 100 + 3 * 150 + 600
    if c["kind"] == "host":
        b += 80
    return {"bytes": float(b) * n * c["steps"], "flops": float(f) * n * c["steps"]}


# ---------------------------------------------------------------------------
# the Roe iteration in plain float64
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] in ("rans", "adjoint") or case.get("flux", 7) != 7:
        return None
    with torch.no_grad():
        m = _Exact(_case(case, seed))
        for _ in range(case["steps"]):
            m.step()
    if case["kind"] == "routines":
        return {"v": m.v.reshape(-1), "u": m.u.reshape(-1), "norms": m.norms}
    if case["kind"] == "host" or case["prec"]:
        return {"v": m.v.reshape(-1)}
    return {"v": m.v.reshape(-1), "norms": m.norms}


class _Exact:
    """State of one case as views (comp, k, j, i) of flat arrays per block."""

    def __init__(self, k):
        self.k, lay = k, k.layout
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.gam, self.pinfl = k.phys.gam, k.phys.pinfl
        self.ns, self.ilim = k.scheme.ns, k.scheme.ilim
        self.v, self.u = (torch.zeros(5, lay.ld, dtype=torch.float64, device=self.dev) for _ in range(2))
        self.v.copy_(torch.as_tensor(k.v0))
        self.blk = [self._block(b) for b in lay.blocks]
        self.norms = None

    def _block(self, b):
        o = {"b": b, "real": (slice(1, b.nk), slice(1, b.nj), slice(1, b.ni))}
        sl, shape = slice(b.npc, b.npc + b.nnn), (b.nkd, b.njd, b.nid)
        o["v"], o["u"] = self.v[:, sl].view(5, *shape), self.u[:, sl].view(5, *shape)
        for a, m in (("p", 1), ("T", 1), ("c", 1), ("mu", 1), ("vel", 3), ("tau", 9)):
            o[a] = torch.zeros(m, *shape, dtype=torch.float64, device=self.dev)
        # nodes with the ghost layer (each ghost node repeats its neighbour)
        P = torch.stack([torch.as_tensor(a[sl]).view(shape) for a in (self.k.x, self.k.y, self.k.z)]).to(self.dev)
        for ax, n in ((1, b.nk), (2, b.nj), (3, b.ni)):
            at = torch.arange(P.shape[ax], device=self.dev).clamp(1, n)
            P = P.index_select(ax, at)
        P = torch.nn.functional.pad(P, (0, 1, 0, 1, 0, 1))

        def at(di, dj, dk):
            return P[:, dk:dk + b.nkd, dj:dj + b.njd, di:di + b.nid]

        S, sums = [], []
        for e, f, axis in (((0, 1, 0), (0, 0, 1), 0), ((1, 0, 0), (0, 0, 1), 1), ((1, 0, 0), (0, 1, 0), 2)):
            ef = tuple(p + q for p, q in zip(e, f))
            n = 0.5 * torch.linalg.cross(at(*ef) - at(0, 0, 0), at(*f) - at(*e), dim=0)
            edge = [0, 0, 0]
            edge[axis] = 1
            mid = (slice(None), *o["real"])
            if float((n * (at(*edge) - at(0, 0, 0)))[mid].sum()) < 0:
                n = -n
            S.append(n)
            sums.append(((at(0, 0, 0) + at(*e) + at(*f) + at(*ef)) * n).sum(0))
        vol = torch.zeros(shape, dtype=torch.float64, device=self.dev)
        r = o["real"]
        for d in range(3):
            vol[r] += self.up(sums[d], d)[r] - sums[d][r]
        o["S"], o["vol"] = S, vol / 12.0
        return o

    @staticmethod
    def up(x, d):
        """the value one cell further along direction d"""
        return torch.roll(x, -1, dims=x.dim() - 1 - d)

    # -- boundary faces ------------------------------------------------------
    def ends(self, x, face):
        """(ghost, interior) slices of the component array x at a face"""
        d, hi = "ijk".index(face[0]), face[1] == "2"
        b = x["b"]
        nd = (b.ni, b.nj, b.nk)[d]
        g, n = (nd, nd - 1) if hi else (0, 1)
        sl = list(x["real"])
        sg, si = list(sl), list(sl)
        sg[2 - d], si[2 - d] = g, n
        return (slice(None), *sg), (slice(None), *si), d, hi

    def boundaries(self):
        gam, g1 = self.gam, self.gam - 1.0
        for q in self.k.boundaries:
            o = self.blk[q.block]
            g, n, d, hi = self.ends(o, q.face)
            W, p = o["v"][n], o["p"][n][0]
            nrm = o["S"][d][g if hi else n] * (-1.0 if hi else 1.0)
            nrm = nrm / nrm.square().sum(0).sqrt()
            if q.kind == cases.BC_RC:
                t = self.k.boundaries[q.partner]
                to = self.blk[t.block]
                tn = self.ends(to, t.face)[1]
                for a in ("v", "p", "T", "c"):
                    o[a][g] = 0.5 * (o[a][n] + to[a][tn])
                o["vol"][g[1:]] = to["vol"][tn[1:]]
                continue
            if q.kind == cases.BC_IDD:
                G, pg = self.injection(W, nrm, q.values)
            elif q.kind == cases.BC_PRD:
                pg = torch.full_like(p, q.values[0])
                vel = W[1:4] / W[0]
                pi = g1 * (W[4] - 0.5 * W[0] * vel.square().sum(0) - self.pinfl)
                rho = W[0] + (pg - pi) / (gam * pi / W[0])
                vel = vel + (pg - pi) / torch.sqrt(gam * pi * W[0]) * nrm
                G = torch.cat([rho[None], rho * vel, (pg / g1 + self.pinfl + 0.5 * rho * vel.square().sum(0))[None]])
            else:
                G, pg = W.clone(), p
                if q.kind == cases.BC_PARA:
                    G[1:4] = 0.0
                    G[4] = W[4] - 0.5 * W[1:4].square().sum(0) / W[0]
            o["v"][g], o["p"][g] = G, pg
            if q.kind in (cases.BC_IDD, cases.BC_PRD):
                o["T"][g] = gam * pg / G[0]
                o["c"][g] = o["T"][g].sqrt()
            else:
                o["T"][g], o["c"][g] = o["T"][n], o["c"][n]

    def injection(self, W, nrm, val):
        gam, g1 = self.gam, self.gam - 1.0
        rpi, rti = val[:2]
        d0 = torch.tensor(val[2:], dtype=torch.float64, device=self.dev).view(3, 1, 1)
        usdn = 1.0 / (d0 * nrm).sum(0)
        qn = (W[1:4] * nrm).sum(0) / W[0]
        p = g1 * (W[4] - 0.5 * W[1:4].square().sum(0) / W[0] - self.pinfl)
        roc0 = -torch.sqrt(gam * p * W[0])
        am0 = p + roc0 * qn
        for it in range(21):
            b = 1.0 / (1.0 + 0.5 * g1 / rti * (usdn * qn).square())
            pp = self.k.phys.pa1 * rpi * b ** (gam / g1)
            ro = gam * pp / (b * rti)
            if it and res <= 1e-7 or it == 20:
                break
            dq = -(pp + roc0 * qn - am0) / (roc0 - ro * qn * usdn.square())
            res = float((dq.abs() / qn).max())
            qn = qn + dq
        m = ro * (qn * usdn * d0)
        E = pp / g1 + self.pinfl + 0.5 * m.square().sum(0) / ro
        return torch.cat([ro[None], m, E[None]]), pp

    # -- one iteration ---------------------------------------------------------
    def step(self):
        gam, g1, ph = self.gam, self.gam - 1.0, self.k.phys
        for o in self.blk:
            r = (slice(None), *o["real"])
            W = o["v"][r]
            p = g1 * (W[4] - 0.5 * W[1:4].square().sum(0) / W[0] - self.pinfl)
            T = gam * p / W[0]
            o["p"][r], o["T"][r], o["c"][r] = p, T, T.sqrt()
            if self.ns:
                a = ph.suth_a
                o["mu"][r] = T * T.sqrt() * (1.0 + a) / (T + a) / ph.reynz
            s2 = [torch.maximum(x := S.square().sum(0), self.up(x, d))[r[1:]] for d, S in enumerate(o["S"])]
            dism = o["vol"][r[1:]] / (s2[0] + s2[1] + s2[2]).sqrt()
            o["dt"] = self.k.scheme.eta * dism / (W[1:4].square().sum(0).sqrt() / W[0] + T.sqrt())
            if self.ns:
                mu = o["mu"][r][0]
                rv = torch.maximum(gam * mu / ph.pr / W[0], 4.0 / 3.0 * mu / W[0])
                o["dt"] = torch.minimum(o["dt"], self.k.scheme.eta * 0.25 * dism.square() / rv)
        self.boundaries()
        for o in self.blk:
            o["vel"][:] = o["v"][1:4] / o["v"][:1]
            if self.ns:
                self.stresses(o)
        if self.ns:
            for q in self.k.boundaries:
                o = self.blk[q.block]
                g, n = self.ends(o, q.face)[:2]
                t = o["tau"][n]
                if q.kind == cases.BC_RC:
                    z = self.k.boundaries[q.partner]
                    zo = self.blk[z.block]
                    t = 0.5 * (t + zo["tau"][self.ends(zo, z.face)[1]])
                o["tau"][g] = t
        for o in self.blk:
            r = (slice(None), *o["real"])
            o["u"][r] = sum(self.residual(o, d) for d in range(3))
            d = self.implicit(o)
            o["res"] = d / o["dt"]
            o["v"][r] += d
        res = torch.cat([o["res"].reshape(5, -1) for o in self.blk], 1)
        self.norms = torch.stack([res.abs().mean(1), res.square().mean(1).sqrt(), res.abs().amax(1)])

    def stresses(self, o):
        r = (slice(None), *o["real"])
        f = torch.cat([o["vel"], o["T"]])
        g = torch.zeros(4, 3, *o["dt"].shape, dtype=torch.float64, device=self.dev)
        for d in range(3):
            fl, S = torch.roll(f, 1, dims=f.dim() - 1 - d), o["S"][d]
            s = f + fl
            first, last = [slice(None)] * 4, [slice(None)] * 4
            nd = (o["b"].ni, o["b"].nj, o["b"].nk)[d]
            first[3 - d], last[3 - d] = 1, nd
            s[tuple(first)] = 2 * fl[tuple(first)]
            s[tuple(last)] = 2 * f[tuple(last)]
            m = s[:, None] * S[None]
            g += (self.up(m, d) - m)[(slice(None), *r)]
        g = g * (0.5 / o["vol"][r[1:]])
        mu = o["mu"][r][0]
        div = g[0, 0] + g[1, 1] + g[2, 2]
        t = o["tau"]
        for q, (a, b) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
            t[q][r[1:]] = mu * (g[a, b] + g[b, a]) - (2.0 / 3.0 * mu * div if a == b else 0.0)
        k = mu / self.k.phys.pr / (self.gam - 1.0)
        for a in range(3):
            t[6 + a][r[1:]] = k * g[3, a]

    def lines(self, o, x, d):
        """x (comp, k, j, i) as lines of direction d over the other two
        directions' real cells: (comp, ., ., 0..nd)"""
        sl = [slice(None), *o["real"]]
        nd = (o["b"].ni, o["b"].nj, o["b"].nk)[d]
        sl[3 - d] = slice(0, nd + 1)
        return x[tuple(sl)].movedim(3 - d, 3)

    @staticmethod
    def dot(a, S):
        return a[0] * S[0] + a[1] * S[1] + a[2] * S[2]

    def tensor_flux(self, t, vel, S):
        """the stresses' part of a flux through S: (4, ...)"""
        row = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
        f = [self.dot([t[q] for q in row[a]], S) for a in range(3)]
        return torch.stack(f + [self.dot(f, vel) + self.dot(t[6:9], S)])

    def residual(self, o, d):
        W, vel, p, S = (self.lines(o, x, d) for x in (o["v"], o["vel"], o["p"], o["S"][d]))
        tau = self.lines(o, o["tau"], d) if self.ns else None
        nd = W.shape[3] - 1
        G = torch.zeros(5, *W.shape[1:3], nd + 1, dtype=torch.float64, device=self.dev)  # faces 1..nd
        for face, gh in ((1, 0), (nd, nd)):
            w, q, s, pg = W[..., gh], vel[..., gh], S[..., face], p[0, ..., gh] - self.pinfl
            m = self.dot(w[1:4], s)
            rho = W[0, ..., 1] if not self.ns and face == 1 and d > 0 else w[0]
            G[..., face] = torch.cat([m[None], w[1:4] * self.dot(q, s) + pg * s, ((w[4] + pg) * m / rho)[None]])
            if self.ns:
                G[1:, ..., face] -= self.tensor_flux(tau[..., gh], q, s)
        if nd > 2:
            c = torch.cat([W[:1], vel, p])
            L, R = self.muscl(c, nd)
            G[..., 2:nd] = self.roe(L, R, S[..., 2:nd])
            if self.ns:
                tl, tr = tau[..., 1:nd - 1], tau[..., 2:nd]
                s = S[..., 2:nd]
                G[1:, ..., 2:nd] -= 0.5 * (self.tensor_flux(tl, L[1:4], s) + self.tensor_flux(tr, R[1:4], s))
        return (G[..., 2:] - G[..., 1:-1]).movedim(3, 3 - d)

    def muscl(self, c, nd):
        xk = self.k.scheme.xk
        dc = c[..., 1:] - c[..., :-1]  # dc[f - 1]: across face f
        a, b, e = dc[..., :nd - 2], dc[..., 1:nd - 1], dc[..., 2:nd]
        c4 = 0.25 * self.k.scheme.muscl
        k1, k2, k3, k4 = (torch.ones_like(b) for _ in range(4))
        if self.ns and self.ilim == 1:
            # the slope ratios, each over the already updated one below it
            r = torch.ones_like(c)
            prev = dc[..., 0]
            for f in range(2, nd):
                cur, nxt = dc[..., f - 1], dc[..., f]
                prev = torch.where((prev * cur * nxt).abs() <= torch.finfo(torch.float64).tiny,
                                   torch.ones_like(cur), cur / prev)
                r[..., f] = prev

            def phi(x):
                return x.clamp(max=1.0).clamp(min=0.0)
            rm, rp = r[..., 2:nd - 1], r[..., 3:nd]
            lim = slice(0, nd - 3)
            for k, x in ((k1, rm), (k2, 1.0 / rm), (k3, rp), (k4, 1.0 / rp)):
                k[..., lim] = phi(x)
        L = c[..., 1:nd - 1] + c4 * ((1 - xk) * k1 * a + (1 + xk) * k2 * b)
        R = c[..., 2:nd] - c4 * ((1 + xk) * k3 * b + (1 - xk) * k4 * e)
        return L, R

    def roe(self, L, R, S):
        gam, g1, pi = self.gam, self.gam - 1.0, self.pinfl
        area = S.square().sum(0).sqrt()
        n = S / area
        E = [x[4] / g1 + pi + 0.5 * x[0] * x[1:4].square().sum(0) for x in (L, R)]
        H = [gam * x[4] / x[0] / g1 + 0.5 * x[1:4].square().sum(0) for x in (L, R)]
        F = 0.0
        for x, e in zip((L, R), E):
            m = x[0] * self.dot(x[1:4], S)
            F = F + torch.cat([m[None], m * x[1:4] + (x[4] - pi) * S, (m / x[0] * (e + x[4] - pi))[None]])
        w = (R[0] / L[0]).sqrt()
        q = (L[1:4] + w * R[1:4]) / (1 + w)
        h = (H[0] + w * H[1]) / (1 + w)
        rho = (L[0] * R[0]).sqrt()
        q2 = 0.5 * q.square().sum(0)
        a2 = (g1 * (h - q2)).abs()
        a, vn = a2.sqrt(), self.dot(q, n)
        dW = torch.cat([(R[0] - L[0])[None], R[0] * R[1:4] - L[0] * L[1:4], (E[1] - E[0])[None]])
        # wave strengths of the conserved jump
        dm = dW[1:4]
        dp = g1 * (dW[4] - self.dot(q, dm) + q2 * dW[0])
        dvn = (self.dot(dm, n) - vn * dW[0]) / rho
        l1, l4, l5 = (area * x.abs() for x in (vn, vn + a, vn - a))
        ent = l1 * (dW[0] - dp / a2)
        w4, w5 = l4 * (dp + rho * a * dvn) / (2 * a2), l5 * (dp - rho * a * dvn) / (2 * a2)
        shear = l1 * (dm - q * dW[0] - rho * dvn * n)
        D0 = ent + w4 + w5
        Dm = ent * q + shear + w4 * (q + a * n) + w5 * (q - a * n)
        DE = ent * q2 + self.dot(q, shear) + w4 * (h + a * vn) + w5 * (h - a * vn)
        return 0.5 * (F - torch.cat([D0[None], Dm, DE[None]]))

    def implicit(self, o):
        r = (slice(None), *o["real"])
        ph, W, vol = self.k.phys, o["v"], o["vol"]
        rv = torch.zeros_like(vol)
        if self.ns:
            rv[r[1:]] = (self.gam * o["mu"][0] / ph.pr / W[0])[r[1:]]
        ce, cd = [], vol[r[1:]] / o["dt"]
        for d in range(3):
            def lo(x):
                return torch.roll(x, 1, dims=x.dim() - 1 - d)
            S = o["S"][d]
            s2 = S.square().sum(0)
            vn = self.dot(0.5 * (o["vel"] + lo(o["vel"])), S).abs()
            ca = s2.sqrt() * 0.5 * (o["c"][0] + lo(o["c"][0]))
            e = 0.5 * (vn + ca) + (rv + lo(rv)) * s2 / (vol + lo(vol)) if self.ns else 0.5 * vn + ca
            ce.append((e[r[1:]], self.up(e, d)[r[1:]]))
            cd = cd + ce[d][0] + ce[d][1]
        w, p = W[r], o["p"][r][0]
        pi, g1, u = self.pinfl, self.gam - 1.0, o["u"][r]
        d = -u / cd

        def flux(w, p):
            q = w[1:4] / w[0]
            f = [torch.cat([w[1 + a][None], w[1:4] * q[a], ((w[4] + p - pi) * q[a])[None]]) for a in range(3)]
            for a in range(3):
                f[a][1 + a] += p
            return f
        f0 = flux(w, p)
        S = [x[r] for x in o["S"]]
        Su = [self.up(x, a)[r] for a, x in enumerate(o["S"])]
        for _ in range(self.k.scheme.lmax - 1):
            x = w + d
            f1 = flux(x, g1 * (x[4] - 0.5 * x[1:4].square().sum(0) / x[0] - pi))
            f = [a - b for a, b in zip(f1, f0)]
            acc = -u
            for a in range(3):
                ax = 3 - a

                def shift(y, s):
                    y = torch.roll(y, s, dims=ax)
                    y.select(ax, 0 if s == 1 else -1).zero_()
                    return y
                dn, up = [shift(y, 1) for y in f], [shift(y, -1) for y in f]
                tl = 0.5 * sum((f[q] + dn[q]) * S[a][q] for q in range(3))
                tu = 0.5 * sum((f[q] + up[q]) * Su[a][q] for q in range(3))
                acc = acc + tl - tu + ce[a][0] * shift(d, 1) + ce[a][1] * shift(d, -1)
            d = acc / cd
        return d
