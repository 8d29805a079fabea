"""The workloads a user of this framework runs, as cases with inputs, one pass and its outputs.

The systems are closed-shell electron gases of the sizes the serving stream and the batched
twist average use: N electrons (N/2 occupied), the `basis` * N/2 plane waves of lowest
|n + k_s|^2, r_s in [0.5, 5], every twist k_s drawn from the seed in [-0.5, 0.5)^3.

Kinds of case, and what each stands for:
  mp2          a host program's DrvMBPT on one system: E(2) and the three amplitude arrays back
  drpa         DrvMBPT then DrvdRPA on one system, the reference's own iteration
  ccd          DrvMBPT then DrvCCD on one system with Pulay DIIS
  residual     one CCD residual for a host that keeps its own iteration loop
  two_channel  DrvCCD with Do Rings and without Do XRings (T2abab and T2abba iterated apart)
  flags        one two-channel residual with per-term range flags
  twists       a twist average: a batch that differs by twist, solved and downloaded
  scan         an r_s scan at one size: a batch that differs by r_s, solved and downloaded
  stream       a mixed cohort of the serving loop: incremental solve, results as they stop
  pipeline     a new twist batch made, solved (CCD or dRPA), downloaded and released, as each
               step of a twist-averaging program with fresh twists does

A drawn case is one of these kinds with its sizes spread over the same ranges.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from uegccd_b200 import Batch, Context, heg
from uegccd_b200.solver import SystemSet

REPLAY = dict(scheme=0)                              # the reference's iteration, tol 1e-8
DIIS = dict(scheme=1, ndiis=6, denom_factor=1.0)     # Pulay over six vectors, undamped steps
STREAM_N = (14, 54, 66, 114)                         # the serving stream's sizes
# per-term range flags whose direct and exchange integrals differ (Safe ERI)
FLAGS = dict(ring=1, mosaic=1, driver_direct=1, quad_rings=1, lin_ladders=1, energy=1)


def listed():
    return [
        # the smallest call: one N=14 system (57 orbitals), latency of the launches and copies
        dict(name="mp2_n14", kind="mp2", electrons=14, basis=8.15, rs=1.0),
        # the reference's dRPA benchmark size
        dict(name="drpa_n14", kind="drpa", electrons=14, basis=8.15, rs=1.0),
        # the reference's own twist average: 100 twists of a small system, its own iteration
        dict(name="ccd_n14_twists100", kind="twists", electrons=14, basis=8.0, rs=1.0, count=100,
             scheme="replay", precision=0),
        # one mid-size system solved by a host program
        dict(name="ccd_n54", kind="ccd", electrons=54, basis=17.963, rs=5.0),
        # the batched twist average, FP64 and mixed precision
        dict(name="ccd_n54_twists100", kind="twists", electrons=54, basis=17.963, rs=1.0, count=100,
             scheme="diis", precision=0),
        dict(name="ccd_n54_twists100_mixed", kind="twists", electrons=54, basis=17.963, rs=1.0,
             count=100, scheme="diis", precision=1),
        # the twist average of the other method, a fresh batch per step
        dict(name="drpa_n54_twists30", kind="pipeline", method="drpa", electrons=54, basis=17.963, rs=1.0, count=30),
        # the largest system, over r_s
        dict(name="ccd_n114_scan4", kind="scan", electrons=114, basis=18.333, count=4),
        # one residual for a host's own loop, ragged sizes
        dict(name="residual_n38", kind="residual", electrons=38, basis=13.0, rs=2.0),
        # rings without crossed rings: both channels
        dict(name="two_channel_n54", kind="two_channel", electrons=54, basis=17.963, rs=1.0),
        # a serving cohort of mixed sizes
        dict(name="stream_12", kind="stream", count=12, pick=3),
        # a fresh batch per step
        dict(name="ccd_n54_pipeline25", kind="pipeline", method="ccd", electrons=54, basis=12.0, rs=1.0, count=25),
    ]


def draw(rng):
    def rs(hi=5.0):
        return round(math.exp(rng.uniform(math.log(0.5), math.log(hi))), 3)

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["mp2", "drpa", "ccd", "residual", "two_channel", "flags", "twists", "twists", "twists",
                       "scan", "stream", "pipeline"])
    basis = round(rng.uniform(4.0, 20.0), 2)
    if kind == "mp2":
        return dict(kind=kind, electrons=2 * rng.randint(7, 57), basis=basis, rs=rs())
    if kind in ("drpa", "ccd", "residual"):
        return dict(kind=kind, electrons=2 * rng.randint(7, 57), basis=basis, rs=rs())
    if kind in ("two_channel", "flags"):
        return dict(kind=kind, electrons=2 * rng.randint(7, 27), basis=round(rng.uniform(4.0, 16.0), 2), rs=rs(2.0))
    if kind == "twists":
        n = rng.choice([14, 24, 38, 54, 66])
        most = {14: 100, 24: 100, 38: 100, 54: 60, 66: 30}[n]
        precision = rng.choice([0, 0, 0, 1])
        return dict(kind=kind, electrons=n, basis=round(rng.uniform(4.0, 17.0), 2), rs=rs(2.0),
                    count=log_int(3, most), scheme="diis" if precision else rng.choice(["diis", "replay"]),
                    precision=precision)
    if kind == "scan":
        return dict(kind=kind, electrons=rng.choice([54, 66, 114]), basis=round(rng.uniform(4.0, 18.0), 2),
                    count=rng.randint(2, 4))
    if kind == "stream":
        return dict(kind=kind, count=rng.randint(2, 12), pick=rng.randint(1, 999))
    return dict(kind=kind, method=rng.choice(["ccd", "drpa"]), electrons=2 * rng.randint(7, 33),
                basis=round(rng.uniform(4.0, 16.0), 2), rs=rs(2.0), count=log_int(3, 25))


# ------------------------------------------------------------------------------ inputs
def _nbasis(nocc, basis):
    return max(nocc + 1, int(round(basis * nocc)))


@functools.lru_cache(maxsize=None)
def _lattice(nbasis):
    """Integer |n|^2 cutoff whose lattice holds 1.6 times the basis: room for the twisted sort."""
    g = np.arange(-16, 17)
    n2 = (g[:, None, None] ** 2 + g[None, :, None] ** 2 + g[None, None, :] ** 2).ravel()
    return max(2, int(np.searchsorted(np.cumsum(np.bincount(n2)), int(1.6 * nbasis) + 8)))


def _set_up(electrons, basis, rs):
    nocc = electrons // 2
    nb = _nbasis(nocc, basis)
    return heg.Heg(heg.default_input(nelectron=electrons, maxkpoint=_lattice(nb), rsmin=rs, rsmax=rs,
                                     fcut=(nb / nocc) ** (2.0 / 3.0)))


def _one_system(case, seed):
    h = _set_up(case["electrons"], case["basis"], case["rs"])
    h.change_twist(np.random.default_rng(seed).random(3) - 0.5)
    return h.system()


def _batch_systems(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "stream":
        out = []
        pick = np.random.default_rng(case["pick"])   # the sizes are the case's, the twists the seed's
        for _ in range(case["count"]):
            h = _set_up(int(pick.choice(STREAM_N)), float(pick.choice((4, 8, 12, 16))),
                        float(np.exp(pick.uniform(math.log(0.5), math.log(5.0)))))
            h.change_twist(rng.random(3) - 0.5)
            out.append(h.system())
        return out
    if case["kind"] == "scan":
        twist = rng.random(3) - 0.5   # one twist, several r_s
        out = []
        for rs in (0.5, 1.0, 2.0, 5.0)[: case["count"]]:
            h = _set_up(case["electrons"], case["basis"], rs)
            h.change_twist(twist)
            out.append(h.system())
        return out
    h = _set_up(case["electrons"], case["basis"], case["rs"])
    return h.twist_systems(rng.random((case["count"], 3)) - 0.5)[0]


def _screening(nocc, length):
    kf = (3.0 * math.pi ** 2 * 2 * nocc / length ** 3) ** (1.0 / 3.0)
    return (4.0 / math.pi * kf) ** 0.5


def _options(case):
    if case.get("method") == "drpa":
        return dict(REPLAY)
    if case["kind"] in ("scan", "pipeline"):
        return dict(DIIS, tol=1e-9)
    if case["kind"] == "stream":
        return dict(DIIS, tol=1e-8, max_iter=200)
    if case["scheme"] == "replay":
        return dict(REPLAY)
    return dict(DIIS, tol=1e-9, precision=case["precision"])


def prepare(case, seed):
    """One system in a context, or a batch and the page-locked buffer its amplitudes go to."""
    kind = case["kind"]
    if kind in ("mp2", "drpa", "ccd", "residual", "two_channel", "flags"):
        system = _one_system(case, seed)
        state = dict(case=case, ctx=Context(*system))
        if kind == "residual":
            state["t"] = state["ctx"].mp2()[2]
        if kind == "flags":
            state["t2"] = state["ctx"].mp2()[2:4]
            state["ctx"].set_eri(FLAGS, safe_eri=True, screening=_screening(system[0], system[1]))
        return state
    systems = _batch_systems(case, seed)
    total = sum(s[0] * s[0] * (len(s[3]) - s[0]) for s in systems)
    state = dict(case=case, options=_options(case),
                 out=torch.empty(total, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy())
    if kind == "pipeline":
        state["systems"] = SystemSet(systems)
    else:
        state["batch"] = Batch(systems)
    return state


# ------------------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mp2":
        return state["ctx"].mp2()
    if kind == "drpa":
        e2, t, _, _ = state["ctx"].mp2()
        _, r, _, _ = state["ctx"].drpa(t)
        return e2, r["ecorr"], r["ecorr_sosex"], t
    if kind == "ccd":
        e2, *t = state["ctx"].mp2()
        _, r, _, _ = state["ctx"].ccd(*t, tol=1e-9, **DIIS)
        return e2, r["ecorr"], t
    if kind == "two_channel":
        e2, *t = state["ctx"].mp2()
        _, r, _, _ = state["ctx"].ccd(*t, do_ring=1, do_xring=0, **REPLAY)
        return e2, r["ecorr"], t
    if kind == "residual":
        return state["ctx"].ccd_g2(state["t"])
    if kind == "flags":
        return state["ctx"].ccd_g2_2ch(*state["t2"])
    if kind == "stream":
        b = state["batch"]
        e2 = b.start(**state["options"])
        ecorr = np.zeros(b.n)
        active = b.n
        while active > 0:
            active, done = b.advance()
            for s, r in done:
                ecorr[s] = r["ecorr"]
        b.all_amplitudes(out=state["out"])
        return e2, ecorr, state["out"]
    b = Batch(state["systems"]) if kind == "pipeline" else state["batch"]
    _, e2, results = b.solve(drpa=case.get("method") == "drpa", **state["options"])
    b.all_amplitudes(out=state["out"])
    ecorr = np.array([r["ecorr"] for r in results])
    sosex = np.array([r["ecorr_sosex"] for r in results])
    if kind == "pipeline":
        b.close()
    return e2, ecorr, sosex, state["out"]


# ------------------------------------------------------------------------------ the work of a pass
@functools.lru_cache(maxsize=None)
def _shape(electrons, basis):
    """Counts of a twisted system: (occupied O, virtuals V, allowed amplitudes with i <= j,
    ladder multiply-adds, ring multiply-adds)."""
    O = electrons // 2
    M = _nbasis(O, basis)
    g = np.arange(-9, 10)
    n = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    key = ((n + np.array([0.137, 0.211, 0.318])) ** 2).sum(1)
    n = n[np.argsort(key, kind="stable")[:M]]
    index = {tuple(v): p for p, v in enumerate(n)}
    pairs = {}
    for i in range(O):
        for j in range(i, O):
            k = tuple(n[i] + n[j])
            pairs[k] = pairs.get(k, 0) + 1
    amps = ladder = 0
    for k, o in pairs.items():
        v = sum(1 for a in n[O:] if index.get(tuple(np.array(k) - a), -1) >= O)
        amps += o * v
        ladder += o * v * v
    groups = {}
    for i in range(O):
        for x in range(O, M):
            q = tuple(n[x] - n[i])
            groups[q] = groups.get(q, 0) + 1
    rings = 0
    for q, n1 in groups.items():
        n2 = groups.get(tuple(-c for c in q), 0)
        if n1 < n2 or (n1 == n2 and q < tuple(-c for c in q)):
            rings += 5 * n1 * n1 * n2 + 2 * n1 * n2 * n2
    return O, M - O, amps, ladder, rings


def work(case):
    kind = case["kind"]
    if kind == "stream":
        pick = np.random.default_rng(case["pick"])
        sizes = []
        for _ in range(case["count"]):
            sizes.append((int(pick.choice(STREAM_N)), float(pick.choice((4, 8, 12, 16)))))
            pick.uniform()
    else:
        sizes = [(case["electrons"], case["basis"])] * case.get("count", 1)
    # iterations a solve of each scheme takes at these sizes
    iterations = {"mp2": 0, "residual": 1, "flags": 1, "drpa": 22, "ccd": 14, "two_channel": 33, "scan": 13,
                  "stream": 12, "pipeline": 22 if case.get("method") == "drpa" else 12}.get(kind)
    drpa = kind == "drpa" or case.get("method") == "drpa"
    if iterations is None:
        iterations = 12 if case["scheme"] == "diis" else 33
    nbytes = flops = 0
    for electrons, basis in sizes:
        O, V, amps, ladder, rings = _shape(electrons, basis)
        channels = 2 if kind in ("two_channel", "flags") else 1
        dense = 8 * O * O * V
        arrays = {"mp2": 3, "drpa": 1, "ccd": 3, "residual": 2, "two_channel": 3, "flags": 4}.get(kind, 1)
        nbytes += arrays * dense + 32 * (O + V) + iterations * channels * 16 * amps
        flops += 8 * amps + iterations * (20 * amps if drpa else channels * channels * 2 * (ladder + rings))
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------ 64-bit values
class _Exact:
    """MP2, the CCD residual of both channels and the dRPA residual of one system with plain
    dense tensors T[i, j, a]; integrals V(|n_p - n_q|^2) from one table per range flag."""

    def __init__(self, system, flags=None):
        O, L, madelung, eigen, nvec = system
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        n = torch.as_tensor(np.array(nvec), dtype=torch.int64, device=dev)
        M = n.shape[0]
        R = int(n.abs().max())
        S = 6 * R + 3   # holds every n_p + n_q - n_r
        cube = torch.full((S, S, S), -1, dtype=torch.int64, device=dev)
        cube[tuple((n + 3 * R + 1).T)] = torch.arange(M, device=dev)

        def orbital(v):
            return cube[tuple((v + 3 * R + 1).unbind(-1))]

        self.O, self.V, self.dev = O, M - O, dev
        occ, vir = n[:O], n[O:]
        b = orbital(occ[:, None, None] + occ[None, :, None] - vir[None, None, :])
        self.ok = b >= O
        self.b = torch.where(self.ok, b - O, 0)
        # d of (i, l, a): n_d = n_l + n_a - n_i
        d = orbital(occ[None, :, None] + vir[None, None, :] - occ[:, None, None])
        self.d_ok = d >= O
        self.d = torch.where(self.d_ok, d - O, 0)
        l = orbital(occ[:, None, None] + occ[None, :, None] - occ[None, None, :])
        self.l_ok = (l >= 0) & (l < O)
        self.l = torch.where(self.l_ok, l, 0)
        e = torch.as_tensor(np.array(eigen), dtype=torch.float64, device=dev)
        eo, ev = e[:O], e[O:]
        self.denom = eo[:, None, None] + eo[None, :, None] - ev[None, None, :] - ev[self.b]

        def q2(x, y):
            return ((x[:, None] - y[None, :]) ** 2).sum(-1)

        top = 12 * R * R + 1
        q = torch.arange(top, dtype=torch.float64, device=dev)
        sd = _screening(O, L)
        plain = 1.0 / (L * math.pi * q)
        plain[0] = -madelung
        short = (1.0 / L ** 3) * 4.0 * math.pi / (sd ** 2 + q * (2.0 * math.pi / L) ** 2)
        table = {0: plain, 1: short}
        self.flag = flags or {}

        def values(name):   # name -> V between two orbital lists for a term's flag
            x, y = {"oo": (occ, occ), "ov": (occ, vir), "vv": (vir, vir)}[name]
            idx = q2(x, y)
            return {f: table[f][idx] for f in table}

        self.oo, self.ov, self.vv = values("oo"), values("ov"), values("vv")
        # v(n_i + n_k - n_a - n_l) as [i, a, k, l]
        w = occ[:, None, None, None] + occ[None, None, :, None] - vir[None, :, None, None] - occ[None, None, None, :]
        idx4 = (w ** 2).sum(-1).clamp_(max=top - 1)
        self.w4 = {f: table[f][idx4] for f in ({0, 1} if self.flag else {0})}

    def f(self, *names):
        return max(self.flag.get(k, 0) for k in names)

    def at_b(self, x):
        return torch.where(self.ok, torch.gather(x, 2, self.b), 0.0)

    def mp2(self):
        t = torch.where(self.ok, self.ov[0][:, None, :] / self.denom, 0.0)
        return t, -self.at_b(t)

    def energy(self, ab, ba):
        v1 = self.ov[self.f("energy")]
        x = v1[:, None, :] * (2.0 * ab + ba) - v1[None, :, :] * (ab + 2.0 * ba)
        return 0.5 * float(torch.where(self.ok, x, 0.0).sum())

    def swapped(self, x):   # x[i, j, a] -> x[j, i, b]
        return self.at_b(x.transpose(0, 1))

    def residual(self, p, m, ring=True, xring=True):
        """G of both channels: p = T2abab, m = T2abba (zero where not allowed)."""
        ok, oo, ov, vv = self.ok, self.oo, self.ov, self.vv
        O, V = self.O, self.V
        via, vja = ov[self.f("driver_direct")][:, None, :], ov[self.f("driver_exchange")][None, :, :]
        g1 = (via + 0.0 * p)
        g2 = -self.at_b(ov[self.f("driver_exchange")][:, None, :] + 0.0 * p)
        # mosaics
        vm = ov[self.f("mosaic")]
        s = torch.where(ok, vm[:, None, :] * (2.0 * p + m) - vm[None, :, :] * (p + 2.0 * m), 0.0)
        jv, jo = s.sum((0, 1)), s.sum((1, 2))
        j = 0.5 * (jv[None, None, :] + jv[self.b] + jo[:, None, None] + jo[None, :, None])
        g1 = g1 - j * p
        g2 = g2 - j * m
        # hole-hole ladder
        ld, lx = self.f("ladder", "direct_ladders", "lin_ladders"), self.f("ladder", "exchange_ladders", "lin_ladders")
        qd, qx = self.f("ladder", "direct_ladders", "quad_ladders"), self.f("ladder", "exchange_ladders", "quad_ladders")

        def kth(x, v):   # sum_c v(c - k) x[ij, c]
            return (x.reshape(O * O, V) @ v.T).reshape(O, O, O)

        def at_l(x):
            return torch.gather(x, 2, self.l)

        h2 = oo[ld][:, None, :] + 0.5 * (kth(p, ov[qd]) - at_l(kth(m, ov[qx])))
        h3 = -at_l(oo[lx][:, None, :].expand(O, O, O)) + 0.5 * (kth(m, ov[qd]) - at_l(kth(p, ov[qx])))
        h2, h3 = (torch.where(self.l_ok, h, 0.0) for h in (h2, h3))
        ii = torch.arange(O, device=self.dev)
        for k in range(O):   # t[k, l(i, j, k), a]
            tp, tm = p[k][self.l[:, :, k]], m[k][self.l[:, :, k]]
            g1 = g1 + 0.5 * (h2[:, :, k, None] * tp + h3[:, :, k, None] * tm)
            g2 = g2 + 0.5 * (h2[:, :, k, None] * tm + h3[:, :, k, None] * tp)
        # particle-particle ladder

        def pp(x, v):
            return (x.reshape(O * O, V) @ v).reshape(O, O, V)

        g1 = g1 + 0.5 * (pp(p, vv[ld]) - self.at_b(pp(m, vv[lx])))
        g2 = g2 + 0.5 * (pp(m, vv[ld]) - self.at_b(pp(p, vv[lx])))
        if ring:
            rd, rx = self.f("ring", "direct_rings", "lin_rings"), self.f("ring", "exchange_rings", "lin_rings")
            sp, sm = p.sum(1), m.sum(1)
            d1 = ov[rd] * (2.0 * sp + sm)
            e1 = d1[:, None, :] - torch.einsum("ika,kj->ija", p, oo[rx])
            e2 = -torch.einsum("ika,kj->ija", m, oo[rx])
            g1 = g1 + e1 + self.swapped(e1)
            g2 = g2 + e2 + self.swapped(e2)
            rd, rx = self.f("ring", "direct_rings", "quad_rings"), self.f("ring", "exchange_rings", "quad_rings")
            vd = ov[rd][:, None, :]
            wp, wm = (torch.einsum("ika,iakl->ila", x, self.w4[rx]) for x in (p, m))
            r1 = vd * (2.0 * sp + sm)[:, None, :] - wp - wm
            r2 = vd * (2.0 * sp + sm)[:, None, :] - wp
            r3 = -wm
            dok = self.d_ok
            for i in range(O):   # t[l, j, d(i, l, a)]
                la = torch.arange(O, device=self.dev)[:, None]
                tp = torch.where(dok[i][:, :, None], p.transpose(1, 2)[la, self.d[i]], 0.0)
                tm = torch.where(dok[i][:, :, None], m.transpose(1, 2)[la, self.d[i]], 0.0)
                g1[i] += torch.einsum("la,laj->ja", r2[i], tp + tm) + torch.einsum("la,laj->ja", r1[i], tp)
                g2[i] += torch.einsum("la,laj->ja", r3[i], tm)
        if xring:
            xd, xx = self.f("xring", "direct_rings", "lin_rings"), self.f("xring", "exchange_rings", "lin_rings")
            tp, tm = p.transpose(0, 1), m.transpose(0, 1)   # x[i, k, b] = t[k, i, b]
            c1 = -torch.einsum("ikb,kj->ijb", tp, oo[xx])
            c2 = ov[xd][:, None, :] * (tp.sum(1) + 2.0 * tm.sum(1))[:, None, :] - torch.einsum("ikb,kj->ijb", tm, oo[xx])
            # the (j, a) form at (i, j, a); the (i, b) form through the partner
            g1 = g1 + self.at_b(c1) + c1.transpose(0, 1)
            g2 = g2 + self.at_b(c2) + c2.transpose(0, 1)
            xd, xx = self.f("xring", "direct_rings", "quad_rings"), self.f("xring", "exchange_rings", "quad_rings")
            vd = ov[xd][:, None, :]
            wp, wm = (torch.einsum("ikb,ibkl->ilb", x, self.w4[xx]) for x in (tp, tm))
            base = vd * (tp.sum(1) + 2.0 * tm.sum(1))[:, None, :]
            x1, x2, x3 = base - wp - wm, base - wm, wp
            for i in range(O):   # x[i, l, b(i, j, a)] against t[l, j, a]
                bi = self.b[i].reshape(-1)
                y1, y2, y3 = (x[i][:, bi].reshape(O, O, V) for x in (x1, x2, x3))
                g2[i] -= (y1 * m + y2 * (p + m)).sum(0)
                g1[i] += (y3 * p).sum(0)
        return torch.where(ok, g1, 0.0), torch.where(ok, g2, 0.0)

    def drpa_residual(self, t):
        v = self.ov[0]
        s = torch.where(self.ok, 2.0 * v[:, None, :] * t, 0.0)
        jv, jo = s.sum((0, 1)), s.sum((1, 2))
        g = v[:, None, :] - 0.5 * (jv[None, None, :] + jv[self.b] + jo[:, None, None] + jo[None, :, None]) * t
        e = 2.0 * (v * t.sum(1))[:, None, :] + 0.0 * t
        g = g + e + self.swapped(e)
        for i in range(self.O):
            la = torch.arange(self.O, device=self.dev)[:, None]
            tl = torch.where(self.d_ok[i][:, :, None], t.transpose(1, 2)[la, self.d[i]], 0.0).sum(0)   # [a, j]
            g[i] += 4.0 * (v[i] * t[i].sum(0))[None, :] * tl.T
        return torch.where(self.ok, g, 0.0)

    def iterate(self, t, step, tol, denom_factor, most=200):
        """Damped Jacobi steps from t until max|dT| < tol, as the reference iterates."""
        dt, n = max(float(x.abs().max()) for x in t), 1
        while dt >= tol and n < most:
            g = step(*t)
            new = [torch.where(self.ok, (y / self.denom - (1.0 - denom_factor) * x) / denom_factor, 0.0)
                   for x, y in zip(t, g)]
            dt = max(float((x - y).abs().max()) for x, y in zip(t, new))
            t, n = new, n + 1
        return t

    @staticmethod
    def out(t):   # T[i, j, a] in the framework's (a, j, i) layout
        return t.permute(2, 1, 0).contiguous().cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("scan", "stream", "twists", "pipeline"):
        return None   # many systems, or a solve of minutes in plain tensors
    system = _one_system(case, seed)
    if case["electrons"] > 80 and kind != "mp2":
        return None
    x = _Exact(system, FLAGS if kind == "flags" else None)
    p, m = x.mp2()
    e2 = float(torch.where(x.ok, p * (2.0 * x.ov[0][:, None, :] - x.ov[0][None, :, :]), 0.0).sum())
    if kind == "mp2":
        return e2, x.out(p + m), x.out(p), x.out(m)
    if kind == "residual":
        return x.out(x.residual(p, m)[0])
    if kind == "flags":
        return tuple(x.out(g) for g in x.residual(p, m))
    if kind == "drpa":
        (t,) = x.iterate([p + m], lambda a: (x.drpa_residual(a),), 1e-8, 2.0)
        v = x.ov[0]
        e = [float(torch.where(x.ok, t * (2.0 * v[:, None, :] - c * v[None, :, :]), 0.0).sum()) for c in (0.0, 1.0)]
        return e2, e[0], e[1], x.out(t)
    if kind == "two_channel":
        p, m = x.iterate([p, m], lambda a, c: x.residual(a, c, xring=False), 1e-8, 2.0)
    else:   # ccd: the fixed point the extrapolated solve approaches
        p, m = x.iterate([p, m], x.residual, 1e-13, 2.0)
    return e2, x.energy(p, m), [x.out(p + m), x.out(p), x.out(m)]
