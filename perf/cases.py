"""Timed cases of the chemistry solve: what a climate model's time loop asks of this package, by size and kind.

A case names a kind of call and its sizes; ``prepare`` makes what the caller has in hand, ``run`` is one call through
the public entry points. Settled states come from a plain torch integration of a small column grid (written here, so
the inputs do not depend on the code that is timed), spread over the case's cells with the changes that transport
makes between two chemistry calls. ``exact`` is the same torch integration of the case's own cells.

Kinds: "call" (CudaSolver), "jvp" and "vjp" (ADSolver), "glue" (the mass/mole conversions either side of a call),
"forward" (the surrogate network). ``start`` of a call: "settled" (the call a time loop makes again and again),
"solar" (the first call of a run, from solar gas), "dark" (a single relaxation over dt = 1e10 s without photolysis).
"""

import functools
import math

import numpy as np
import torch

from maxichem_b200 import coupling, synthetic, tables
from maxichem_b200.ad import ADSolver
from maxichem_b200.solver import CudaSolver
from maxichem_b200.surrogate import Surrogate

LEVELS, COLUMNS = 64, 12  # the settled base grid
DT = {"cho41": 300.0, "chno69": 300.0, "sncho91": 600.0}
RTOL, ATOL, MAX_STEPS = 1e-3, 1e-25, 4000


def listed():
    return [
        # one model column: a single-column run, or the last ragged share of a rank; latency decides
        {"name": "one_column", "kind": "call", "network": "chno69", "start": "settled", "cells": 64},
        # a coarse model's share of one GPU, not a multiple of anything
        {"name": "small_grid", "kind": "call", "network": "chno69", "start": "settled", "cells": 3001},
        # the 69-species configuration's whole grid
        {"name": "full_grid", "kind": "call", "network": "chno69", "start": "settled", "cells": 65536},
        # the small C-H-O network of long runs
        {"name": "cho_grid", "kind": "call", "network": "cho41", "start": "settled", "cells": 40000},
        # the sulfur network, its own longer time step
        {"name": "sulfur_grid", "kind": "call", "network": "sncho91", "start": "settled", "cells": 16385},
        # the first call of a run: every cell far from its steady state, some 140 steps
        {"name": "first_call", "kind": "call", "network": "chno69", "start": "solar", "cells": 1500},
        # relaxation to the thermochemical steady state, no light
        {"name": "relaxation", "kind": "call", "network": "cho41", "start": "dark", "cells": 1000},
        # one sensitivity direction through the call
        {"name": "tangent", "kind": "jvp", "network": "chno69", "cells": 4096, "directions": 1, "adapt": True},
        # a few directions that share a call, the step control held fixed
        {"name": "tangents_4", "kind": "jvp", "network": "cho41", "cells": 2500, "directions": 4, "adapt": False},
        # the gradient of a loss on the composition
        {"name": "adjoint", "kind": "vjp", "network": "chno69", "cells": 4096, "adapt": True},
        # a high-resolution grid's conversions before and after a call
        {"name": "glue", "kind": "glue", "network": "chno69", "cells": 262144},
        # the surrogate's forward pass on the 69-species grid
        {"name": "surrogate", "kind": "forward", "network": "chno69", "cells": 65536},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call"] * 6 + ["jvp", "jvp", "vjp", "vjp", "glue", "forward"])
    network = rng.choice(["cho41", "chno69", "chno69", "sncho91"])
    size = {"cho41": 2.0, "chno69": 1.0, "sncho91": 0.4}[network]  # cells for about the same work
    if kind == "call":
        start = rng.choice(["settled"] * 4 + ["solar", "dark"])
        most = {"settled": 40000, "solar": 1500, "dark": 1000}[start]
        return {"kind": kind, "network": network, "start": start, "cells": _between(rng, 16, most * size)}
    if kind == "jvp":
        directions = rng.choice([1, 1, 2, 3, 5, 8])
        return {"kind": kind, "network": network, "cells": _between(rng, 50, 6000 * size / directions),
                "directions": directions, "adapt": rng.random() < 0.7}  # fmt: skip
    if kind == "vjp":
        return {"kind": kind, "network": network, "cells": _between(rng, 50, 5000 * size), "adapt": rng.random() < 0.7}
    if kind == "glue":
        return {"kind": kind, "network": network, "cells": _between(rng, 1000, 190000)}
    return {"kind": kind, "network": network, "cells": _between(rng, 1000, 65536)}


# ---- a plain torch integration of the call: Rodas3 with the exact Jacobian, per-cell adaptive steps ----


class _Chemistry:
    """A network's laws as torch tensors: rates of a cell, S v and its derivative."""

    def __init__(self, net, photo, dev):
        self.dev = dev
        f = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=dev)  # noqa: E731
        ix = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.long, device=dev)  # noqa: E731
        ln = lambda a: math.log(a) if a > 0 else -math.inf  # noqa: E731
        reac, photos = net.reac, (net.photo if photo else [])
        self.ns, self.nrt, self.nr = len(net.species), len(reac), len(reac) + len(photos)
        S = np.asarray(net.S, np.float64)
        self.S = f(np.hstack([S, np.asarray(net.Sp, np.float64)]) if photo else S)
        self.lo, self.hi = f(net.lo), f(net.hi)
        pad = lambda a: list(a) + [self.ns] * (3 - len(a))  # noqa: E731
        self.left = ix([pad(r["re"]) for r in reac] + [pad(r["re"]) for r in photos])
        self.right = ix([pad(r["pr"]) for r in reac] + [[self.ns] * 3 for _ in photos])
        rows, marks, order = [], [], []
        for r in reac:
            two = r["kind"] == 2  # two-body: one Arrhenius law
            k0 = (r["A"], r["B"], r["C"]) if two else (r["A0"], r["B0"], r["C0"])
            k1 = (r["A1"], r["B1"], r["C1"]) if "A1" in r else (0.0, 0.0, 0.0)
            ki = (r["Ai"], r["Bi"], r["Ci"]) if r["kind"] in (3, 6) else (1.0, 0.0, 0.0)
            rows.append([ln(k0[0]), *k0[1:], ln(k1[0]), *k1[1:], ln(ki[0]), *ki[1:],
                         *r.get("troe", (0.0, 1.0, 1.0, 0.0)), r.get("eff", 1.0)])  # fmt: skip
            marks.append([r["kind"] in (3, 6), "A1" in r, r["kind"] in (3, 5, 6), "troe" in r,
                          r.get("width") == "vm11"])  # fmt: skip
            order.append([len(r["re"]), len(r["pr"])])
        self.law = f(rows)
        self.falloff, self.second, self.three, self.troe, self.vm11 = (
            torch.as_tensor(np.array(marks)[:, k], device=dev) for k in range(5))  # fmt: skip
        self.order = f(order)

    def rates(self, T, P, J):
        q, Tc = self.law, T[:, None]
        nd = P[:, None] / (1.380649e-16 * Tc)
        lT, iT = torch.log(Tc), 1.0 / Tc
        arr = lambda k: torch.exp(q[:, k] + q[:, k + 1] * lT - q[:, k + 2] * iT)  # noqa: E731
        k = arr(0)
        k = torch.where(self.second, k + arr(3), k)
        pr = k * nd / arr(6)
        bound = k / (1.0 + pr)
        fc = torch.log10((1.0 - q[:, 9]) * torch.exp(-Tc / q[:, 10]) + q[:, 9] * torch.exp(-Tc / q[:, 11])
                         + torch.exp(-q[:, 12] / Tc))  # fmt: skip
        safe = torch.where(pr > 0, pr, torch.ones_like(pr))
        x = torch.where(self.vm11, torch.log10(safe), torch.log10(safe) - 0.4 - 0.67 * fc)
        y = x / (0.75 - 1.27 * fc - torch.where(self.vm11, torch.zeros_like(x), 0.14 * x))
        wide = bound * 10.0 ** (fc / (1.0 + y * y))
        k = torch.where(self.falloff, torch.where(self.troe, wide, bound), k) * q[:, 13]
        a = torch.where((T < 1000.0)[:, None, None], self.lo, self.hi)
        t = Tc
        h = (-a[..., 0] * iT * iT + a[..., 1] * lT * iT + a[..., 2] + a[..., 3] * t / 2 + a[..., 4] * t**2 / 3
             + a[..., 5] * t**3 / 4 + a[..., 6] * t**4 / 5 + a[..., 7] * iT)  # fmt: skip
        s = (-a[..., 0] * iT * iT / 2 - a[..., 1] * iT + a[..., 2] * lT + a[..., 3] * t + a[..., 4] * t**2 / 2
             + a[..., 5] * t**3 / 3 + a[..., 6] * t**4 / 4 + a[..., 8])  # fmt: skip
        g = torch.cat([h - s, torch.zeros_like(Tc)], 1)
        left, right = self.left[: self.nrt], self.right[: self.nrt]
        dg = g[:, right].sum(2) - g[:, left].sum(2)
        lKT = torch.log(1.380649e-16 * Tc / 1.0e6)
        c3 = torch.where(self.three, nd, torch.ones_like(nd))
        kf = k * c3
        kr = kf * torch.exp(dg + (self.order[:, 1] - self.order[:, 0]) * lKT)
        q2 = torch.maximum(self._two(kf, self.order[:, 0], nd), self._two(kr, self.order[:, 1], nd))
        cc = torch.where(q2 > 1e-9, 1e-9 / q2, torch.ones_like(q2))  # the collision limit
        kf, kr = kf * cc, kr * cc
        if J is not None and self.nr > self.nrt:
            kf, kr = torch.cat([kf, J], 1), torch.cat([kr, torch.zeros_like(J)], 1)
        return kf, kr, nd[:, 0]

    def _two(self, k, m, nd):
        return torch.where(m == 3, k * nd, torch.where(m == 2, k, torch.where(self.three, k / nd, torch.zeros_like(k))))

    def sv(self, kf, kr, n):
        """S v(n) and the factors of each side's product."""
        e = torch.cat([n, torch.ones_like(n[:, :1])], 1)
        l, r = e[:, self.left], e[:, self.right]
        return (kf * l.prod(2) - kr * r.prod(2)) @ self.S.T, l, r

    def jacobian(self, kf, kr, l, r):
        B = kf.shape[0]
        dv = torch.zeros(B, self.nr, self.ns + 1, dtype=torch.float64, device=self.dev)
        for m in range(3):
            o, p = (m + 1) % 3, (m + 2) % 3
            dv = dv.scatter_add(2, self.left[None, :, m, None].expand(B, -1, 1), (kf * l[..., o] * l[..., p])[..., None])
            dv = dv.scatter_add(2, self.right[None, :, m, None].expand(B, -1, 1), (-kr * r[..., o] * r[..., p])[..., None])
        return torch.einsum("pr,brq->bpq", self.S, dv[..., : self.ns])


def _advance(chem, x, T, P, dt, h, J, adapt=True):
    """One call: x, h, steps after dt; a cell's arithmetic does not depend on the others. With adapt False the step
    sizes carry no derivative."""
    B, ns = x.shape
    kf, kr, nd = chem.rates(T, P, J)
    h = torch.minimum(h, dt).clamp_min(1e-12)
    stop = (lambda a: a) if adapt else (lambda a: a.detach())
    h, dtq = stop(h), stop(dt)
    N, t, nok = x, torch.zeros_like(T), torch.zeros_like(T)
    prej = torch.zeros(B, dtype=torch.bool, device=chem.dev)
    pen, pha = torch.zeros_like(T), torch.zeros_like(T)
    eye = torch.eye(ns, dtype=torch.float64, device=chem.dev)
    for _ in range(MAX_STEPS):
        on = t.detach() < dt.detach() * (1.0 - 1e-14)
        idx = on.nonzero().flatten()
        if idx.numel() == 0:
            break
        c = lambda a: a[idx]  # noqa: E731
        n0, ndc, kfc, krc = c(N), c(nd)[:, None], c(kf), c(kr)
        ha = torch.minimum(c(h), c(dtq) - c(t))
        ntot = n0.sum(1, keepdim=True)

        def rhs(Y):
            tot = Y.sum(1, keepdim=True)
            s, l, r = chem.sv(kfc, krc, Y * (ndc / tot))
            return s * (tot / ndc), s, l, r

        F, s, l, r = rhs(n0)
        Jn = chem.jacobian(kfc, krc, l, r)
        w = s / ndc - (Jn @ n0[..., None])[..., 0] / ntot
        igh, ih = (2.0 / ha)[:, None, None], (1.0 / ha)[:, None]
        # W = M0 - w 1^T by Sherman-Morrison; M0 = I / (gamma h) - Jn keeps its diagonal as pivots, which loses less to
        # cancellation than exchanging rows of the full W
        LU, piv = torch.linalg.lu_factor(igh * eye - Jn, pivot=False)
        msolve = lambda b: torch.linalg.lu_solve(LU, piv, b[..., None])[..., 0]  # noqa: E731
        u = msolve(w)
        c0 = 1.0 / (1.0 - u.sum(1, keepdim=True))

        def solve(b):
            y = msolve(b)
            return y + c0 * y.sum(1, keepdim=True) * u

        K1 = solve(F)
        K2 = solve(F + 4.0 * ih * K1)
        K3 = solve(rhs(n0 + 2.0 * K1)[0] + ih * (K1 - K2))
        K4 = solve(rhs(n0 + 2.0 * K1 + K3)[0] + ih * (K1 - K2 - (8.0 / 3.0) * K3))
        Y = n0 + 2.0 * K1 + K3 + K4
        q = K4 / (RTOL * torch.maximum(n0.abs(), Y.abs()) + ATOL)
        er = torch.sqrt((q * q).sum(1) / ns)
        emx = q.abs().amax(1)
        en = torch.where((c(t) == 0) & torch.isfinite(er), torch.maximum(er, emx), er)
        ok = (en <= 1.0) & (Y >= -ATOL).all(1) & torch.isfinite(en)
        good = torch.where(torch.isfinite(en), en, torch.ones_like(en))
        fac = torch.where(torch.isfinite(en), 0.9 * good.clamp_min(1e-10) ** (-1.0 / 3.0), torch.full_like(en, 0.1))
        fac = fac.clamp_min(0.2).clamp_max(20.0)
        sec = ~ok & torch.isfinite(en) & c(prej) & (en > 1) & (c(pen) > 1) & (c(pha) > ha)
        one = torch.ones_like(en)
        pe = torch.log(torch.where(sec, c(pen) / good, 2 * one)) / torch.log(torch.where(sec, c(pha) / ha, 2 * one))
        pes = torch.where(pe > 0.05, pe, one)
        alt = torch.where(pe > 0.05, ((0.5 / good) ** (1.0 / pes.clamp_max(3.0))).clamp_min(1e-4), 1e-4 * one)
        fac = torch.where(sec, alt, fac)
        fac = torch.where(ok, fac, fac.clamp_max(0.5))
        put = lambda a, v: a.index_put((idx,), v)  # noqa: E731
        N = put(N, torch.where(ok[:, None], Y.clamp_min(0.0), n0))
        t = put(t, stop(torch.where(ok, c(t) + ha, c(t))))
        nok = put(nok, c(nok) + ok.double())
        h, prej, pen, pha = put(h, stop(ha * fac)), put(prej, ~ok), put(pen, stop(en)), put(pha, ha)
    return N / N.sum(1, keepdim=True), h, nok


def _in_parts(chem, args, part):
    out = [_advance(chem, *(None if a is None else a[k : k + part] for a in args)) for k in range(0, args[0].shape[0], part)]
    return tuple(torch.cat(v) for v in zip(*out))


# ---- inputs ----


@functools.lru_cache(maxsize=None)
def _net(name):
    return synthetic.network(name)


@functools.lru_cache(maxsize=None)
def _chem(name, photo):
    return _Chemistry(_net(name), photo, torch.device("cuda", torch.cuda.current_device()))


@functools.lru_cache(maxsize=1)  # a program keeps the one solver of its network
def _solver(name, photo, ad):
    dev = torch.device("cuda", torch.cuda.current_device())
    return (ADSolver if ad else CudaSolver)(_net(name), dev, photo=photo)


@functools.lru_cache(maxsize=None)
def _flops(name, photo):
    return tables.build(_net(name), photo).flops


@functools.lru_cache(maxsize=None)
def _base(name):
    """The settled base grid of a network: x, T, P, h, J after four calls from solar gas [LEVELS * COLUMNS]."""
    net, chem = _net(name), _chem(name, True)
    w = synthetic.workload(net, "column", LEVELS * COLUMNS, seed=11)
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=chem.dev)  # noqa: E731
    x, T, P, h, J = t(w.x), t(w.T), t(w.P), t(w.h), t(w.J)
    dt = torch.full_like(T, DT[name])
    with torch.no_grad():
        for _ in range(4):
            x, h, _ = _in_parts(chem, (x, T, P, dt, h, J), 1024)
    return x, T, P, h, J


def _settled(name, cells, seed):
    """`cells` cells of settled columns one model step later: each column a base column mixed 0.1 % with the level
    above, its temperatures up to 0.5 K and its light up to 2 % changed."""
    bx, bT, bP, bh, bJ = _base(name)
    dev = bx.device
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    u = lambda *s: torch.rand(*s, generator=g, device=dev, dtype=torch.float64)  # noqa: E731
    i = torch.arange(cells, device=dev)
    col = torch.randint(0, COLUMNS, (-(-cells // LEVELS),), generator=g, device=dev)[i // LEVELS]
    lev = i % LEVELS
    at = col * LEVELS + lev
    up = col * LEVELS + (lev + 1).clamp_max(LEVELS - 1)
    mix = 1e-3 * u(cells, 1)
    x = (1.0 - mix) * bx[at] + mix * bx[up]
    x = x / x.sum(1, keepdim=True)
    T = bT[at] + (u(cells) - 0.5)
    J = bJ[at] * (1.0 + 0.04 * (u(cells, 1) - 0.5))
    return [x, T, bP[at].clone(), torch.full_like(T, DT[name]), bh[at].clone(), J]


def _cells(case, seed):
    name, start = case["network"], case.get("start", "settled")
    if start == "settled":
        return _settled(name, case["cells"], seed)
    dev = torch.device("cuda", torch.cuda.current_device())
    w = synthetic.workload(_net(name), "column" if start == "solar" else "cfg0", case["cells"], seed=seed)
    a = [torch.as_tensor(v, dtype=torch.float64, device=dev) for v in (w.x, w.T, w.P, w.dt, w.h, w.J)]
    if start == "solar":
        a[3].fill_(DT[name])
        return a
    return a[:5] + [None]


def _directions(case, seed, a):
    """Tangents of the inputs [D, B, ...], as the sensitivity of a run to its state, forcing and light."""
    x, T, P, dt, h, J = a
    g = torch.Generator(device=x.device)
    g.manual_seed(seed + 1)
    r = lambda v: torch.randn(case["directions"], *v.shape, generator=g, device=x.device, dtype=torch.float64)  # noqa: E731
    dx = x * r(x)
    dx = dx - x * dx.sum(2, keepdim=True)
    return [dx, 0.01 * T * r(T), 0.1 * P * r(P), torch.zeros_like(r(T)), torch.zeros_like(r(T))], 0.1 * J * r(J)


def _cotangents(case, seed, a):
    """Of a loss on the abundant species' mole fractions and, with the step control differentiated, on log h."""
    x, h = a[0], a[4]
    g = torch.Generator(device=x.device)
    g.manual_seed(seed + 1)
    gx = torch.randn(*x.shape, generator=g, device=x.device, dtype=torch.float64) / x.clamp_min(1e-6)
    return gx, (torch.randn(*h.shape, generator=g, device=x.device, dtype=torch.float64) / h if case["adapt"] else None)


def _glue(case, seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    net = _net(case["network"])
    mw = coupling.molar_masses(np.asarray(net.atoms), list(net.elements)).to(dev)
    q = 10.0 ** (-20.0 * torch.rand(case["cells"], len(net.species), generator=g, device=dev, dtype=torch.float64))
    return q / q.sum(1, keepdim=True), mw, q.new_ones(case["cells"])


def _features(case, seed, dev):
    """A surrogate in its network's sizes and standardised features."""
    net = _net(case["network"])
    sur = Surrogate(len(net.species), len(net.photo), np.asarray(net.atoms, np.float64), dev, seed=3)
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    feat = torch.randn(case["cells"], sur.kin, generator=g, device=dev)
    feat[:, sur.nf :] = 0.0
    return sur, feat.to(torch.bfloat16)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    kind = case["kind"]
    if kind == "glue":
        q, mw, mass = _glue(case, seed, dev)
        return {"kind": kind, "q": q, "mw": mw, "mass": mass}
    if kind == "forward":
        sur, feat = _features(case, seed, dev)
        return {"kind": kind, "sur": sur, "feat": feat}
    a = _cells(case, seed)
    s = {"kind": kind, "in": a[:5], "J": a[5], "solver": _solver(case["network"], a[5] is not None, kind != "call")}
    if kind == "jvp":
        s["tan"], s["dJ"] = _directions(case, seed, a)
        s["adapt"] = case["adapt"]
    elif kind == "vjp":
        s["gx"], s["gh"] = _cotangents(case, seed, a)
        s["adapt"] = case["adapt"]
    return s


def run(state):
    kind = state["kind"]
    if kind == "call":
        r = state["solver"](*state["in"], J=state["J"])
        return {"x": r.x, "h": r.h, "done": r.done, "steps": r.steps}
    if kind == "jvp":
        r = state["solver"].jvp(*state["in"], *state["tan"], J=state["J"], dJ=state["dJ"], adapt=state["adapt"])
        return {"x": r.x, "h": r.h, "done": r.done, "steps": r.steps, "dx": r.dx, "dh": r.dh}
    if kind == "vjp":
        r = state["solver"].vjp(*state["in"], state["gx"], gh=state["gh"], J=state["J"], adapt=state["adapt"])
        c = r.cotangents
        return {"x": r.x, "h": r.h, "done": r.done, "steps": r.steps,
                "gx": c.x, "gT": c.T, "gP": c.P, "gdt": c.dt, "gh": c.h, "glm": c.lm, "grc": c.rc, "gJ": c.J}  # fmt: skip
    if kind == "glue":
        x = coupling.mass_to_mole(state["q"], state["mw"])
        return {"x": x, "q": coupling.mole_to_mass(x, state["mw"], state["mass"])}
    return state["sur"].forward(state["feat"])


# tries of a cell in one call, measured: what the steps of the inputs above take
TRIES = {"settled": 13.0, "solar": 165.0, "dark": 230.0}


def work(case):
    B, net = case["cells"], _net(case["network"])
    ns, nr, nj = len(net.species), len(net.reac) + len(net.photo), len(net.photo)
    if case["kind"] == "glue":
        return {"bytes": 8.0 * B * (4 * ns + 1), "flops": 6.0 * B * ns}
    if case["kind"] == "forward":
        width = (ns + 4 + nj, 512, 512, 512, 512, 4 * (ns + 1))
        macs = sum(a * b for a, b in zip(width, width[1:]))
        return {"bytes": 2.0 * B * width[0] + 4.0 * B * width[-1] + 2.0 * macs, "flops": 2.0 * B * macs}
    start = case.get("start", "settled")
    f = _flops(case["network"], start != "dark")
    one = f["rates"] + TRIES[start] * f["fresh_try"]
    io = 8.0 * B * (2 * ns + (nj if start != "dark" else 0) + 7)
    if case["kind"] == "jvp":  # a direction: three right-hand sides' and four solves' worth again, twice the rates
        d = case["directions"]
        per = 2 * f["rates"] + TRIES[start] * (4 * (f["solve"] + 2 * f["rhs"]) + 3 * f["rhs"])
        return {"bytes": io + 8.0 * B * d * (2 * ns + 5 + nj), "flops": B * (one + d * per)}
    if case["kind"] == "vjp":
        per = 2 * f["rates"] + TRIES[start] * (4 * (f["solve"] + 2 * f["rhs"]) + 3 * f["rhs"])
        return {"bytes": io + 8.0 * (B * (2 * ns + nr + nj + 5) + 9 * nr), "flops": B * (one + per)}
    return {"bytes": io, "flops": B * one}


def tolerance(case):
    kind = case["kind"]
    if kind == "glue":
        return {"rel": 1e-14, "max": 1e-13}
    if kind == "forward":  # BF16 activations: a sum in another order rounds some of them to the neighbouring value
        return {"rel": 4e-3, "max": 4e-2}
    # x and the steps agree to 1e-10 with the torch integration below; the next step h follows the cube root of an error
    # estimate that is a difference of nearly equal stages: measured 1e-5 (worst cell 2.4e-4), on the 41-species
    # network, whose estimates fall to rounding, 3.2e-3 (3.2e-2); the derivatives 1e-8 to 1e-6
    if case["network"] == "cho41" or case.get("start") == "dark":
        return {"rel": 1.3e-2, "max": 0.13}
    return {"rel": 5e-5, "max": 1e-3}


def exact(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    kind = case["kind"]
    if kind == "glue":
        q, mw, mass = _glue(case, seed, dev)
        n = q / mw
        x = n / n.sum(1, keepdim=True)
        m = x * mw
        return {"x": x, "q": m * (mass / m.sum(1))[:, None]}
    if kind == "forward":
        sur, feat = _features(case, seed, dev)
        a = feat.double()
        for l, (w, b) in enumerate(sur.unpack(sur.params())):
            w = torch.as_tensor(w, device=dev).to(torch.bfloat16).double()
            a = a @ w.T + torch.as_tensor(b, device=dev).double()
            a = torch.nn.functional.silu(a) if l < sur.layers else a
        return a
    a = _cells(case, seed)
    chem = _chem(case["network"], a[5] is not None)
    if kind == "call":
        # h and steps have no such value: the step control compares an error estimate with thresholds, and rounding alone
        # moves some cells across them
        with torch.no_grad():
            x, _, _ = _in_parts(chem, a, 2048)
        return {"x": x, "h": None, "done": None, "steps": None}
    if kind == "jvp":
        return _exact_jvp(chem, case, seed, a)
    return _exact_vjp(chem, case, seed, a)


def _exact_jvp(chem, case, seed, a):
    tan, dJ = _directions(case, seed, a)
    dxs = []
    x = None
    for d in range(case["directions"]):
        parts = []
        for k in range(0, case["cells"], 1024):
            with torch.autograd.forward_ad.dual_level(), torch.no_grad():
                dual = [torch.autograd.forward_ad.make_dual(v[k : k + 1024], t[d][k : k + 1024])
                        for v, t in zip(a, tan + [dJ])]  # fmt: skip
                y, _, _ = _advance(chem, *dual, adapt=case["adapt"])
                parts.append(tuple(torch.autograd.forward_ad.unpack_dual(y)))
        x = torch.cat([p for p, _ in parts])
        dxs.append(torch.cat([t for _, t in parts]))
    return {"x": x, "h": None, "done": None, "steps": None, "dx": torch.stack(dxs), "dh": None}


def _exact_vjp(chem, case, seed, a):
    gx, gh = _cotangents(case, seed, a)
    out = []
    for k in range(0, case["cells"], 256):
        ins = [v[k : k + 256].clone().requires_grad_() for v in a]
        x, h, _ = _advance(chem, *ins, adapt=case["adapt"])
        loss = (x * gx[k : k + 256]).sum() + (0.0 if gh is None else (h * gh[k : k + 256]).sum())
        g = torch.autograd.grad(loss, ins, allow_unused=True)
        out.append([x.detach()] + [torch.zeros_like(v) if q is None else q for v, q in zip(ins, g)])
        del x, h, loss, g
    x, cx, cT, cP, cdt, ch, cJ = (torch.cat(v) for v in zip(*out))
    return {"x": x, "h": None, "done": None, "steps": None, "gx": cx, "gT": cT, "gP": cP, "gdt": cdt, "gh": ch,
            "glm": None, "grc": None, "gJ": cJ}  # fmt: skip
