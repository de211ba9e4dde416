"""The time steps a user of this framework runs, as measurable cases.

A pass is what a host program does with a context it keeps: copy a state from
pinned host memory into it, advance it, copy the result back.  The context
(grid tables, registers, tile variant), the initial state and the pinned
result buffer are in hand before the pass.

Families (sizes from the committed example inputs, tests and benchmark):

* ``tube``     1-D two-fluid (or one-fluid) shock tube
* ``droplet``  2-D air shock on a water droplet, plain FP64, split precision,
               learned gate, with or without the viscous terms and their WENO
               velocity gradients, fixed dt or a constant CFL number
* ``bubble``   3-D air shock on a helium sphere, FP64 or split precision
* ``ensemble`` many independent 2-D droplets advanced together

``exact`` restates the scheme (uniform grid, WENO5-JS, HLLC, TVD-RK3) in
64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from microfc_gb300 import Case, Simulation, cases, gate, preprocess
from microfc_gb300.ensemble import Ensemble

DEV = "cuda"
AIR = cases.stiffened(1.4)
WATER = cases.stiffened(6.12, 3.43e8)
HELIUM = cases.stiffened(1.67)
RE_SHEAR, RE_BULK = (10.0, 500.0), (0.0, 200.0)
CFL = 0.3


def _case(name, family, nx, ny, nz, steps, **kw):
    c = {"name": name, "family": family, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "precision": "fp64",
         "fluids": 2, "bc": -3, "viscous": False, "weno_re_flux": False, "cfl_run": False, "tune": False, "count": 1}
    c.update(kw)
    return c


def listed():
    return [
        # the example shock tubes: a few hundred to a thousand cells, thousands
        # of steps, where the latency of a stage is the whole cost
        _case("tube_1000", "tube", 1000, 1, 1, 50),
        # a small odd 2-D grid in plain FP64 (the size of the example 2-D
        # shock-bubble), stepped as it comes, without autotuning
        _case("droplet_301x101", "droplet", 301, 101, 1, 10),
        # the benchmark grid in plain FP64, autotuned as long runs are
        _case("droplet_1024x512", "droplet", 1024, 512, 1, 4, tune=True),
        # a run at a constant CFL number: the monitor's value sets each next dt
        _case("droplet_cfl_400x200", "droplet", 400, 200, 1, 10, cfl_run=True),
        # split precision, a parameter-study size with partial edge tiles
        _case("droplet_split_333x167", "droplet", 333, 167, 1, 50, precision="split"),
        # split precision on the benchmark grid
        _case("droplet_split_1024x512", "droplet", 1024, 512, 1, 100, precision="split", tune=True),
        # the learned gate on its own configuration's grid
        _case("droplet_gated_2048x1024", "droplet", 2048, 1024, 1, 20, precision="gated", tune=True),
        # viscous terms, finite-difference gradients, symmetry below
        _case("droplet_viscous_320x160", "droplet", 320, 160, 1, 8, viscous=True, bc=-2),
        # viscous terms with WENO velocity gradients in split precision
        _case("droplet_viscous_weno_split_1024x512", "droplet", 1024, 512, 1, 30, precision="split", viscous=True,
              weno_re_flux=True),
        # a 3-D verification run in plain FP64, odd sizes
        _case("bubble_97x80x71", "bubble", 97, 80, 71, 3),
        # the 3-D configuration in split precision: states past every cache
        _case("bubble_split_256", "bubble", 256, 256, 256, 10, precision="split", tune=True),
        # a seeded study of 24 small droplets in one ensemble
        _case("ensemble_gated_24", "ensemble", 512, 256, 1, 150, precision="gated", tune=True, count=24),
    ]


# rough cost of one cell and step in nanoseconds, so that a drawn case takes
# 2 to 30 ms a pass
_COST = {"tube": 8.0, "fp64": 9.0, "split": 0.3, "gated": 0.3, "fp64_3d": 15.0, "split_3d": 0.4}


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def steps(cells, ns, top):
        return max(1, min(top, int(rng.uniform(2e6, 3e7) / (cells * ns))))

    family = rng.choice(["tube", "droplet", "droplet", "droplet", "droplet", "bubble", "ensemble"])
    if family == "tube":
        nx = log(100, 20000)
        return _draw(family, nx, 1, 1, steps(nx, _COST["tube"], 60), fluids=rng.choice([1, 2]),
                     precision=rng.choice(["fp64", "fp64", "split"]), bc=rng.choice([-3, -3, -2, -1]))
    if family == "droplet":
        precision = rng.choice(["fp64", "split", "split", "gated"])
        nx = log(50, 1024 if precision == "fp64" else 2048)
        ny = max(26, int(nx * rng.choice([0.33, 0.5, 0.5, 1.0])) + rng.choice([0, 0, 1, 3]))
        viscous = rng.random() < 0.3
        wrf = viscous and rng.random() < 0.5
        ns = _COST[precision] * (2.0 if wrf else 1.0) * (1.5 if viscous else 1.0)
        return _draw(family, nx, ny, 1, steps(nx * ny, ns, 60), precision=precision, viscous=viscous,
                     weno_re_flux=wrf, bc=rng.choice([-3, -3, -2, -1]),
                     cfl_run=not viscous and rng.random() < 0.25, tune=rng.random() < 0.5)
    if family == "bubble":
        precision = rng.choice(["fp64", "split"])
        hi = 128 if precision == "fp64" else 256
        nx, ny, nz = (log(32, hi) for _ in range(3))
        return _draw(family, nx, ny, nz, steps(nx * ny * nz, _COST[precision + "_3d"], 40), precision=precision,
                     bc=rng.choice([-3, -3, -2, -1]), tune=rng.random() < 0.5)
    nx = rng.choice([128, 256, 384, 512])
    count = rng.randint(4, 32)
    precision = rng.choice(["split", "gated", "gated"])
    return _draw(family, nx, nx // 2, 1, steps(count * nx * nx // 4, _COST[precision], 150), precision=precision,
                 tune=rng.random() < 0.7, count=count)


def _draw(family, nx, ny, nz, steps, **kw):
    c = _case("", family, nx, ny, nz, steps, **kw)
    del c["name"]
    return c


# -- inputs -------------------------------------------------------------------

def _domain(family):
    if family == "tube":
        return ((0.0, 1.0), (0.0, 0.0), (0.0, 0.0))
    if family == "bubble":
        return ((-0.5, 0.5),) * 3
    return ((0.0, 0.02), (0.0, 0.01), (0.0, 0.0))


def _fluids(c):
    if c["family"] == "tube":
        return [AIR] * c["fluids"]
    return [HELIUM, AIR] if c["family"] == "bubble" else [WATER, AIR]


def _initial(c, rng):
    """Conservative state [S, nz, ny, nx] (FP64, on the GPU), the case's cell
    widths and the dt of CFL number 0.3."""
    fam, n = c["family"], (c["nx"], c["ny"], c["nz"])
    nd = 1 + (n[1] > 1) + (n[2] > 1)
    nf = c["fluids"]
    dom = _domain(fam)
    h = [(dom[d][1] - dom[d][0]) / n[d] for d in range(nd)]
    xyz = []
    for d in range(nd):
        s = [1, 1, 1]
        s[2 - d] = n[d]
        xyz.append((dom[d][0] + h[d] * (torch.arange(n[d], dtype=torch.float64, device=DEV) + 0.5)).reshape(s))
    one = torch.ones((n[2], n[1], n[0]), dtype=torch.float64, device=DEV)
    if fam == "tube":
        x0, hot = rng.uniform(0.4, 0.6), rng.uniform(0.8, 1.5)
        left = (xyz[0] < x0) * one
        rho = torch.where(left > 0, one * hot, one * 0.125)
        p = torch.where(left > 0, one * hot, one * 0.1)
        vel = [0.0 * one]
        a1 = torch.where(left > 0, one * (1.0 - 1e-6), one * 1e-6)
        alpha = [one] if nf == 1 else [a1, 1.0 - a1]
        arho = [a * rho for a in alpha]
    else:
        if fam == "bubble":
            mach, r0, amb, rho_in, front = rng.uniform(1.1, 1.5), rng.uniform(0.1, 0.2), (1.0, 1.0), 0.138, -0.3
            centre = [rng.uniform(-0.05, 0.05) for _ in range(3)]
        else:
            mach, r0, amb, rho_in, front = rng.uniform(1.2, 2.5), rng.uniform(1e-3, 3e-3), (1.2, 101325.0), 1000.0, 4e-3
            centre = [rng.uniform(0.0075, 0.0085), rng.uniform(0.0045, 0.0055)]
        rho2, u2, p2 = cases.normal_shock(1.4, amb[0], amb[1], mach)
        hit = (xyz[0] < front) * one > 0
        r = torch.sqrt(sum((xyz[d] - centre[d]) ** 2 for d in range(nd)) + 0.0 * one)
        a1 = 0.5 - 0.5 * torch.tanh(0.5 / min(h) * (r - r0))
        a1 = torch.where(a1 < 1e-12, 0.0 * one, a1)
        alpha = [a1, 1.0 - a1]
        arho = [a1 * rho_in, (1.0 - a1) * torch.where(hit, one * rho2, one * amb[0])]
        p = torch.where(hit, one * p2, one * amb[1])
        vel = [torch.where(hit, one * u2, 0.0 * one)] + [0.0 * one] * (nd - 1)
    fl = _fluids(c)
    rho = sum(arho)
    gam = sum(a * g for a, (g, _) in zip(alpha, fl))
    pinf = sum(a * q for a, (_, q) in zip(alpha, fl))
    q = torch.stack(arho + [rho * u for u in vel]
                    + [gam * p + pinf + 0.5 * rho * sum(u * u for u in vel)] + alpha)
    snd = torch.sqrt(((gam + 1.0) * p + pinf) / (gam * rho))
    dt = CFL * min(float((h[d] / (vel[d].abs() + snd)).min()) for d in range(nd))
    return q, h, dt


def _sizes(c):
    """The member widths of an ensemble, taken in turn (heights are half)."""
    return [n for n in (128, 256, 384, 512) if n <= c["nx"]]


def _members(c, seed):
    """(case, state, widths, dt) of every run of the pass."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(c["count"]):
        m = dict(c)
        if c["family"] == "ensemble":
            nx = _sizes(c)[(3 * i) % len(_sizes(c))]
            m.update(nx=nx, ny=nx // 2)
        out.append((m, *_initial(m, rng)))
    return out


def _config(m, dt):
    nd = 1 + (m["ny"] > 1) + (m["nz"] > 1)
    none = (-100, -100)
    fl = _fluids(m)
    bc = (m["bc"], m["bc"])
    if m["bc"] == -2:  # symmetry along one side, extrapolation elsewhere
        bcs = [(-3, -3), (-2, -3), (-3, -3)] if nd > 1 else [(-2, -3), none, none]
    else:
        bcs = [bc, bc, bc]
    dom = _domain(m["family"])
    return Case(m=m["nx"] - 1, n=m["ny"] - 1, p=m["nz"] - 1, x_domain=dom[0], y_domain=dom[1], z_domain=dom[2], dt=dt,
                t_step_stop=m["steps"], t_step_save=m["steps"], num_fluids=m["fluids"], time_stepper=3, weno_order=5,
                weno_eps=1e-16, bc_x=bcs[0], bc_y=bcs[1] if nd > 1 else none, bc_z=bcs[2] if nd > 2 else none,
                gammas=tuple(f[0] for f in fl), pi_infs=tuple(f[1] for f in fl),
                re_shear=RE_SHEAR if m["viscous"] else (), re_bulk=RE_BULK if m["viscous"] else (),
                weno_re_flux=m["weno_re_flux"], precision=m["precision"])


def _pinned(t):
    h = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def prepare(case, seed):
    runs = _members(case, seed)
    configs = [_config(m, dt) for m, _, _, dt in runs]
    q = [_pinned(s) for _, s, _, _ in runs]
    weights = gate.load() if case["precision"] == "gated" else None
    if case["family"] == "ensemble":
        # the ensemble's constructor lays a state from the patches: a plain
        # background, replaced by each pass's upload
        patches = cases.shock_droplet_2d(32, 32, dt=1.0).patches
        sim = Ensemble([k.replace(patches=patches) for k in configs], ic="device")
        for i, s in enumerate(q):
            sim.upload(i, s)
        result = None
    else:
        sim = Simulation(configs[0], *preprocess.grid(configs[0]), q_cons=q[0])
        result = torch.empty(q[0].shape, dtype=torch.float64, pin_memory=True).numpy()
    if weights is not None:
        sim.set_gate(weights)
    if case["tune"]:
        sim.tune(3)
    return {"case": case, "sim": sim, "q": q, "result": result, "dt": configs[0].dt}


def run(state):
    case, sim = state["case"], state["sim"]
    if case["family"] == "ensemble":
        for i, q in enumerate(state["q"]):
            sim.upload(i, q)
        sim.run(0, case["steps"])
        return [sim.download(i) for i in range(case["count"])]
    sim.upload(state["q"][0])
    if case["cfl_run"]:
        dt, time = sim.run_cfl(case["steps"], CFL, dt=state["dt"])
        return [sim.download(state["result"]), dt, time]
    sim.run(0, case["steps"])
    return [sim.download(state["result"])]


def work(case):
    """Bytes: the state copied in and out, and one read and one write of it per
    step (a step's stages could share one pass over the state; separate steps
    of a state past the caches cannot).  Operations: the counted adds,
    multiplies, divisions and square roots of a 2-D two-fluid RK3 step,
    5325 a cell, scaled by directions and variables; the viscous terms add
    about 400, their WENO gradients about 3000."""
    if case["family"] == "ensemble":
        s = _sizes(case)
        cells = sum(s[(3 * i) % len(s)] ** 2 // 2 for i in range(case["count"]))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    nd = 1 + (case["ny"] > 1) + (case["nz"] > 1)
    S = 2 * case["fluids"] + nd + 1
    per_cell = 5325.0 * nd / 2.0 * S / 7.0 + (400.0 if case["viscous"] else 0.0) \
        + (3000.0 if case["weno_re_flux"] else 0.0)
    return {"bytes": 16.0 * S * cells * (case["steps"] + 1), "flops": per_cell * cells * case["steps"]}


# -- the scheme in 64-bit torch -------------------------------------------------

def _ghosts(t, dim, h, bc, flip=()):
    """t with h ghost cells on both sides along dim; flip: variables whose
    sign changes across a symmetry."""
    n = t.shape[dim]
    i = torch.arange(-h, n + h, device=t.device)
    lo, hi = i < 0, i >= n
    j = i.clone()
    j[lo] = i[lo] + n if bc[0] == -1 else (-i[lo] - 1 if bc[0] == -2 else 0)
    j[hi] = i[hi] - n if bc[1] == -1 else (2 * n - 1 - i[hi] if bc[1] == -2 else n - 1)
    g = t.index_select(dim, j)
    for v in flip:
        for side, b in ((lo, bc[0]), (hi, bc[1])):
            if b == -2:
                s = torch.where(side, -1.0, 1.0).to(t.dtype)
                shape = [1] * (t.dim() - 1)
                shape[dim - 1] = -1
                g[v] = g[v] * s.reshape(shape)
    return g


def _weno5(t, dim, eps=1e-16):
    """Left- and right-face values of the cells 2 .. n-3 of t along dim."""
    n = t.shape[dim] - 4
    v = [t.narrow(dim, k, n) for k in range(5)]
    d = [v[k + 1] - v[k] for k in range(4)]
    b = [4 / 3 * x * x - 11 / 3 * x * y + 10 / 3 * y * y + eps for x, y in ((d[3], d[2]), (d[0], d[1]))]
    mid = 4 / 3 * d[2] * d[2] - 5 / 3 * d[2] * d[1] + 4 / 3 * d[1] * d[1] + eps
    b = (b[0], mid, b[1])
    out = []
    for side in (0, 1):
        if side:
            p0 = v[2] + 2 / 3 * d[2] - 1 / 6 * d[3]
            p1 = v[2] + 1 / 3 * d[2] + 1 / 6 * d[1]
            p2 = v[2] + 5 / 6 * d[1] - 1 / 3 * d[0]
            w = (0.3, 0.6, 0.1)
        else:
            p0 = v[2] - 5 / 6 * d[2] + 1 / 3 * d[3]
            p1 = v[2] - 1 / 6 * d[2] - 1 / 3 * d[1]
            p2 = v[2] - 2 / 3 * d[1] + 1 / 6 * d[0]
            w = (0.1, 0.6, 0.3)
        a = [w[k] / (b[k] * b[k]) for k in range(3)]
        s = a[0] + a[1] + a[2]
        out.append((a[0] * p0 + a[1] * p1 + a[2] * p2) / s)
    return out


class _Scheme:
    def __init__(self, m, h):
        self.h, self.nd = h, len(h)
        cfg = _config(m, 1.0)
        self.bc = [cfg.bc_x, cfg.bc_y, cfg.bc_z][: self.nd]
        self.fl = _fluids(m)
        self.nf = len(self.fl)
        self.mom, self.E, self.adv = self.nf, self.nf + self.nd, self.nf + self.nd + 1
        self.visc, self.wrf = m["viscous"], m["weno_re_flux"]

    def mix(self, w, off):
        return sum(w[self.adv + f] * self.fl[f][off] for f in range(self.nf))

    def prim(self, q):
        w = q.clone()
        rho = sum(q[f] for f in range(self.nf)).clamp_min(1e-16)
        ke = 0.0
        for d in range(self.nd):
            w[self.mom + d] = q[self.mom + d] / rho
            ke = ke + 0.5 * q[self.mom + d] * w[self.mom + d]
        w[self.E] = (q[self.E] - ke - self.mix(q, 1)) / self.mix(q, 0)
        return w

    def hllc(self, L, R, d):
        st = []
        for w in (L, R):
            rho = sum(w[f] for f in range(self.nf))
            u = w[self.mom + d]
            sq = sum(w[self.mom + k] ** 2 for k in range(self.nd))
            g = self.mix(w, 0)
            e = g * w[self.E] + self.mix(w, 1) + 0.5 * rho * sq
            c = torch.sqrt(((e + w[self.E]) / rho - 0.5 * sq) / g)
            st.append((rho, u, w[self.E], e, c))
        (rL, uL, pL, _, cL), (rR, uR, pR, _, cR) = st
        sL, sR = torch.minimum(uL - cL, uR - cR), torch.maximum(uR + cR, uL + cL)
        sS = (pR - pL + rL * uL * (sL - uL) - rR * uR * (sR - uR)) / (rL * (sL - uL) - rR * (sR - uR))
        left = ~torch.signbit(sS)
        rho, u, p, e = (torch.where(left, a, b) for a, b in zip(st[0][:4], st[1][:4]))
        sk = torch.where(left, sL, sR)
        s = torch.where(left, sL.clamp_max(0.0), sR.clamp_min(0.0))
        w = torch.where(left, L, R)
        xi = (sk - u) / (sk - sS)
        us = u + s * (xi - 1.0)
        F = w * us
        for k in range(self.nd):
            v = w[self.mom + k]
            F[self.mom + k] = rho * (u * v + s * (xi * (sS if k == d else v) - v)) + (p if k == d else 0.0)
        F[self.E] = u * (e + p) + s * (xi * (e + (sS - u) * (rho * sS + p / (sk - u))) - e)
        vs = [w[self.mom + k] + (s * (xi - 1.0) if k == d else 0.0) for k in range(self.nd)]
        return F, us, vs

    def velocity_ghosts(self, w, h):
        u = w[self.mom:self.mom + self.nd]
        for d in range(self.nd):
            u = _ghosts(u, u.dim() - 1 - d, h, self.bc[d], (d,))
        return u

    def face_gradients(self, w, d):
        """grad[c][e] = d u_c / d x_e on the faces along d."""
        nd, n = self.nd, w.dim()
        if self.wrf:
            u = self.velocity_ghosts(w, 5)
            grad = []
            for e in range(nd):
                dim = n - 1 - e
                vl, vr = _weno5(u, dim)
                g = (vr - vl) / self.h[e]  # cells -3 .. n+2 along e
                for o in range(nd):
                    if o != e:
                        g = g.narrow(n - 1 - o, 2, g.shape[n - 1 - o] - 4)
                for o in range(nd):  # the interior across the sweep
                    if o != d:
                        g = g.narrow(n - 1 - o, 3, g.shape[n - 1 - o] - 6)
                vl, vr = _weno5(g, n - 1 - d)  # cells -1 .. n
                k = vl.shape[n - 1 - d]
                grad.append(0.5 * (vr.narrow(n - 1 - d, 0, k - 1) + vl.narrow(n - 1 - d, 1, k - 1)))
            return [[grad[e][c] for e in range(nd)] for c in range(nd)]
        u = self.velocity_ghosts(w, 1)
        dim = n - 1 - d

        def inner(t, skip):
            for o in range(nd):
                if o not in skip:
                    t = t.narrow(n - 1 - o, 1, t.shape[n - 1 - o] - 2)
            return t

        grad = [[None] * nd for _ in range(nd)]
        k = u.shape[dim]
        for e in range(nd):
            if e == d:
                g = inner((u.narrow(dim, 1, k - 1) - u.narrow(dim, 0, k - 1)) / self.h[d], (d,))
            else:
                de = n - 1 - e
                ke = u.shape[de]
                c = inner((u.narrow(de, 2, ke - 2) - u.narrow(de, 0, ke - 2)) / (2.0 * self.h[e]), (d, e))
                g = 0.5 * (c.narrow(dim, 0, k - 1) + c.narrow(dim, 1, k - 1))
            for c in range(nd):
                grad[c][e] = g[c]
        return grad

    def viscous(self, w, L, R, vs, d):
        g = self.face_gradients(w, d)
        inv = []
        for re in (RE_SHEAR, RE_BULK):
            side = [sum(q[self.adv + f] / re[f] for f in range(self.nf) if re[f] > 0).clamp_min(1e-16)
                    for q in (L, R)]
            inv.append(0.5 * (side[0] + side[1]))
        div = sum(g[k][k] for k in range(self.nd))
        tau = []
        for k in range(self.nd):
            if k == d:
                t = (2.0 * g[d][d] - 2.0 / 3.0 * div) * inv[0] + div * inv[1]
            else:
                t = (g[k][d] + g[d][k]) * inv[0]
            tau.append(-t)
        return tau, sum(v * t for v, t in zip(vs, tau))

    def rhs(self, q):
        w = self.prim(q)
        out = torch.zeros_like(q)
        for d in range(self.nd):
            dim = w.dim() - 1 - d
            vl, vr = _weno5(_ghosts(w, dim, 3, self.bc[d], (self.mom + d,)), dim)
            k = vl.shape[dim]
            L, R = vr.narrow(dim, 0, k - 1), vl.narrow(dim, 1, k - 1)
            F, us, vs = self.hllc(L, R, d)
            if self.visc:
                tau, fe = self.viscous(w, L, R, vs, d)
                for c in range(self.nd):
                    F[self.mom + c] += tau[c]
                F[self.E] += fe
            n = q.shape[dim]
            out += (F.narrow(dim, 0, n) - F.narrow(dim, 1, n)) / self.h[d]
            du = (us.narrow(dim - 1, 1, n) - us.narrow(dim - 1, 0, n)) / self.h[d]
            for f in range(self.nf):
                out[self.adv + f] += w[self.adv + f] * du
        return out

    def step(self, q, dt):
        q1 = q + dt * self.rhs(q)
        q2 = (3.0 * q + q1 + dt * self.rhs(q1)) / 4.0
        del q1
        return (q + 2.0 * q2 + 2.0 * dt * self.rhs(q2)) / 3.0

    def icfl(self, q, dt):
        w = self.prim(q)
        rho = sum(w[f] for f in range(self.nf))
        g = self.mix(w, 0)
        c = torch.sqrt(((g + 1.0) * w[self.E] + self.mix(w, 1)) / (g * rho))
        return dt * max(float(((w[self.mom + d].abs() + c) / self.h[d]).max()) for d in range(self.nd))


def exact(case, seed):
    out = []
    for i, (m, q, h, dt) in enumerate(_members(case, seed)):
        if i % 6:  # a few members of an ensemble: each takes seconds
            out.append(None)
            continue
        s = _Scheme(m, h)
        if case["cfl_run"]:
            t = 0.0
            for _ in range(case["steps"]):
                q = s.step(q, dt)
                t += dt
                dt *= CFL / s.icfl(q, dt)
            return [q, dt, t]
        t, final = 0.0, case["steps"] * dt
        for _ in range(case["steps"]):
            t += dt
            q = s.step(q, dt)
            if t + dt >= final:
                dt = final - t
        out.append(q)
    return out
