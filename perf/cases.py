"""What a user of this framework has it do, as measurable cases.

Every case is a whole call sequence through the public entry points
(``uq_b200.solver``): fields in, some time steps, fields out.

- ``solver``: one ``Solver`` restarted from a checkpoint (``set_dist``) and
  stepped with ``runOne``/``step`` with the residual read every step, as a
  driver that watches convergence does.
- ``batch``: a ``Batch`` of one or many samples restarted from host fields
  (pinned memory), advanced, and its fields and status read back: a parameter
  study, or one large solve.
- ``server``: requests submitted to a running ``Server``, waited for, and
  their fields collected.

Flows are those of ``uq_b200.workloads``: thermal Couette flow (periodic in x,
solid walls in y), the four-quadrant Riemann problem (open edges) and the
supersonic flat plate (stretched rows, solid wall, fixed inflow).  Fields of
single-precision runs are handed on in single precision, those of
double-precision runs in double precision.

Step counts are short enough that the flows, which amplify rounding by orders
of magnitude over tens of steps, still determine their outputs.
"""
import math
import random

import numpy as np
import torch

from uq_b200 import workloads as W
from uq_b200.solver import Batch, Server, Solver

SIDES = (64, 128, 256, 512)  # the ensemble's grid sides


def listed():
    return [
        # the smallest calls: a 16 x 16 solve watched step by step
        dict(name="watch_16_f64", entry="solver", flow="couette", n=1, mix=0, nx=16, ny=16, prec="f64", rk=1, fm=1,
             steps=8),
        # one 64 x 128 Couette solve, both precisions: launch latency counts
        dict(name="couette_64x128_f64", entry="batch", flow="couette", n=1, mix=0, nx=64, ny=128, prec="f64", rk=1,
             fm=1, steps=16),
        dict(name="couette_64x128_f32", entry="batch", flow="couette", n=1, mix=0, nx=64, ny=128, prec="f32", rk=1,
             fm=1, steps=16),
        # the Riemann setup of the reference (NND, RK1) on a small grid, watched
        dict(name="riemann_256_f64", entry="solver", flow="riemann", n=1, mix=0, nx=256, ny=256, prec="f64", rk=0,
             fm=0, steps=24),
        # the boundary-layer input's grid, 1001 x 101: ragged in both directions
        dict(name="plate_1001x101_f64", entry="batch", flow="plate", n=1, mix=0, nx=1001, ny=101, prec="f64", rk=1,
             fm=1, steps=16),
        # parameter studies: 16 samples of mixed sides, odd sides, both precisions
        dict(name="ensemble_16_f64", entry="batch", flow="couette", n=16, mix=1, nx=0, ny=0, prec="f64", rk=1, fm=1,
             steps=16),
        dict(name="ensemble_16_odd_f32", entry="batch", flow="couette", n=16, mix=-2, nx=0, ny=0, prec="f32", rk=1,
             fm=1, steps=16),
        # the Riemann problem at higher order in double precision
        dict(name="riemann_1024_f64", entry="batch", flow="riemann", n=1, mix=0, nx=1024, ny=1024, prec="f64", rk=1,
             fm=1, steps=12),
        # requests arriving together at the server
        dict(name="serve_12_f32", entry="server", flow="mixed", n=12, mix=3, nx=0, ny=0, prec="f32", rk=0, fm=0,
             steps=48),
        # the large ones: Riemann 2048 x 2048, flat plates 2048 x 512, a 64-sample ensemble
        dict(name="riemann_2048_f32", entry="batch", flow="riemann", n=1, mix=0, nx=2048, ny=2048, prec="f32", rk=0,
             fm=0, steps=16),
        dict(name="plates_3x2048x512_f32", entry="batch", flow="plate", n=3, mix=0, nx=2048, ny=512, prec="f32", rk=1,
             fm=1, steps=6),
        dict(name="ensemble_64_f32", entry="batch", flow="couette", n=64, mix=4, nx=0, ny=0, prec="f32", rk=1, fm=1,
             steps=16),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solver", "one", "one", "study", "study", "server"])
    prec = rng.choice(["f32", "f64"])
    flow = rng.choice(["couette", "riemann", "plate"])
    rk, fm = rng.choice([0, 1, 1]), rng.choice([0, 1, 1])
    base = dict(entry="batch", flow=flow, n=1, mix=0, nx=0, ny=0, prec=prec, rk=rk, fm=fm, steps=16)
    if kind == "solver":
        flow = rng.choice(["couette", "riemann"])
        return dict(base, entry="solver", flow=flow, prec="f64", nx=_logint(rng, 16, 300), ny=_logint(rng, 16, 300),
                    steps=8)
    if kind == "one":
        return dict(base, nx=_logint(rng, 48, 1600), ny=_logint(rng, 48, 1200),
                    steps=6 if flow == "plate" and prec == "f32" else 14)
    if kind == "study":
        mix = rng.randrange(10, 10000)
        if flow == "couette":
            return dict(base, n=_logint(rng, 2, 40), mix=rng.choice([mix, -mix]))
        return dict(base, n=rng.randrange(2, 6), nx=_logint(rng, 64, 700), ny=_logint(rng, 64, 500),
                    steps=6 if flow == "plate" and prec == "f32" else 14)
    return dict(base, entry="server", flow="mixed", n=rng.randrange(4, 13), mix=rng.randrange(10, 10000), prec="f32",
                rk=0, fm=0, steps=rng.randrange(24, 48))


# --------------------------------------------------------------- what a case holds
def _members(case):
    """[(flow, nx, ny, rk, fm, steps, CFL)] of a case's samples, without the
    values that the seed draws; mix seeds the sizes (negative: odd ones)."""
    r = random.Random(abs(case["mix"]))
    out = []
    for _ in range(case["n"]):
        if case["flow"] == "mixed":
            flow = r.choice(["couette", "riemann"])
            side, rk, fm = r.randint(64, 256), r.randrange(2), r.randrange(2)
            if flow == "couette":
                out.append((flow, side, side, rk, fm, 16, 0.3))
            else:
                out.append((flow, side, side, rk, 0, case["steps"], 0.05))
            continue
        nx, ny = case["nx"], case["ny"]
        if not nx:
            nx = ny = r.choice(SIDES)
            if case["mix"] < 0:
                nx, ny = nx + 2 * r.randint(-8, 8) + 1, ny + 2 * r.randint(-8, 8) + 1
        cfl = 0.2 if case["flow"] == "riemann" else 0.5
        out.append((case["flow"], nx, ny, case["rk"], case["fm"], case["steps"], cfl))
    return out


def _samples(case, seed):
    """Per sample: the solver configuration (``uq_b200.workloads``'s keys,
    with every node of a region in one property) and the initial fields
    rho, ux, uy, T as [nx, ny] arrays."""
    g = np.random.default_rng([seed, 20])
    out = []
    for flow, nx, ny, rk, fm, steps, cfl in _members(case):
        bnd = np.zeros((nx, ny), dtype=np.int32)
        cfg = dict(W.BASE, RKMETHOD=rk, FMETHOD=fm, CFL=cfl, steps=steps, Pr=float(g.uniform(0.6, 1.0)))
        uy = np.zeros((nx, ny))
        if flow == "couette":
            u_w, tau = float(g.uniform(0.05, 0.2)), float(g.uniform(0.02, 0.04))
            cfg.update(periodicX=1, mu=tau)
            bnd[:, 0], bnd[:, ny - 1], ct, vx = 1, 2, [0, 2, 2], [0.0, 0.0, u_w]
            rho, T, ux = 1.0 + g.uniform(-1e-4, 1e-4, (nx, ny)), np.ones((nx, ny)), np.zeros((nx, ny))
            rho[:, 0] = rho[:, ny - 1] = 1.0
            ux[:, ny - 1] = u_w
            props = dict(density=[1.0] * 3, temp=[1.0] * 3, velocityX=vx, velocityY=[0.0] * 3)
        elif flow == "riemann":
            q = W.RIEMANN_QUADRANTS
            s = 1.0 + g.uniform(-0.05, 0.05, 4)  # the four states, each a little off
            rq, pq = np.array(q["rho"]) * s, np.array(q["p"])
            cfg.update(mu=float(g.uniform(0.8e-3, 1.2e-3)), Tc_Tref=1.5)
            mx, my = nx // 2, ny // 2
            bnd[mx:, my:], bnd[:mx, my:], bnd[:mx, :my], bnd[mx:, :my], ct = 0, 1, 2, 3, [0] * 4
            rho, T = rq[bnd], (pq / rq)[bnd]
            ux, uy = np.array(q["ux"])[bnd], np.array(q["uy"])[bnd]
            props = dict(density=rq, temp=pq / rq, velocityX=np.array(q["ux"]), velocityY=np.array(q["uy"]))
        else:
            mach, tau = float(g.uniform(1.5, 2.2)), float(g.uniform(1e-3, 2e-3))
            dy = 0.25 * 1.02 ** np.arange(ny)
            cfg.update(mu=tau, Tc_Tref=4.0, dx=1.0, dy=float(dy.min()), dx_array=np.ones(nx), dy_array=dy)
            u_inf = mach * math.sqrt(1.4)
            bnd[0, :], bnd[:, ny - 1] = 1, 1
            bnd[:, 0], ct = 2, [0, 1, 2]
            fluid = bnd == 0
            rho, T = np.ones((nx, ny)), np.ones((nx, ny))
            rho[fluid] += g.uniform(-1e-3, 1e-3, int(fluid.sum()))
            ux = np.where(bnd == 2, 0.0, u_inf)
            props = dict(density=[1.0] * 3, temp=[1.0] * 3, velocityX=[u_inf, u_inf, 0.0], velocityY=[0.0] * 3)
        props.update(pressure=np.zeros(len(ct)), cellType=ct)
        out.append((W._finish(cfg, props, bnd), (rho, ux, uy, T)))
    return out


def prepare(case, seed):
    samples = _samples(case, seed)
    f32 = case["prec"] == "f32"
    if case["entry"] == "server":
        reqs = []
        for cfg, (rho, ux, uy, T) in samples:  # each node its own property, as a request with its own initial fields has
            cfg = dict(cfg)
            ct = np.asarray(cfg["cellType"])[cfg["bnd"]]
            n = rho.size
            cfg.update(density=rho.reshape(-1), temp=T.reshape(-1), velocityX=ux.reshape(-1), velocityY=uy.reshape(-1),
                       pressure=np.zeros(n), cellType=ct.reshape(-1), numProps=n,
                       bnd=np.arange(n, dtype=np.int32).reshape(rho.shape))
            reqs.append(cfg)
        return dict(entry="server", srv=Server(precision=case["prec"], arena_bytes=2 << 30), reqs=reqs, f32=f32)
    if case["entry"] == "solver":
        cfg, fields = samples[0]
        b = Batch([cfg], case["prec"])
        b.set_macro(0, *fields)
        f, h = b.dist(0)
        b.close()
        return dict(entry="solver", solver=Solver(cfg, case["prec"]), f=f, h=h, steps=case["steps"], f32=f32)
    n = sum(a[0].size for _, a in samples)
    fields = torch.empty((4, n), dtype=torch.float64, pin_memory=True)
    for k in range(4):
        fields[k] = torch.from_numpy(np.concatenate([a[k].reshape(-1) for _, a in samples]))
    out = torch.empty((5, n), dtype=torch.float64, pin_memory=True)
    out32 = torch.zeros((5, n), dtype=torch.float32) if f32 else None
    return dict(entry="batch", batch=Batch([c for c, _ in samples], case["prec"]), fields=fields, out=out, out32=out32,
                steps=case["steps"])


def run(state):
    if state["entry"] == "server":
        srv, res = state["srv"], []
        ids = [srv.submit(c) for c in state["reqs"]]
        for rid in ids:
            srv.wait(rid)
            status, m = srv.result(rid)
            srv.release(rid)
            t = np.float32 if state["f32"] else np.float64
            res.append(dict(status=int(status), rho=m["rho"].astype(t), u=np.stack([m["ux"], m["uy"]]).astype(t),
                            T=m["T"].astype(t)))
        return res
    if state["entry"] == "solver":
        s = state["solver"]
        s.set_dist(state["f"], state["h"])
        residuals = []
        for _ in range(state["steps"]):
            status, r = s.step(1, residual=True)
            residuals.append(r)
        m = s.macro()
        return dict(status=int(status), residuals=np.array(residuals), rho=m["rho"], u=np.stack([m["ux"], m["uy"]]),
                    T=m["T"], p=m["p"])
    b, out = state["batch"], state["out"]
    b.set_macro_all_ptr(*[v.data_ptr() for v in state["fields"]])
    b.step(state["steps"])
    b.macro_all_ptr(*[v.data_ptr() for v in out])
    status = b.status()
    if state["out32"] is not None:
        out = state["out32"].copy_(out)
    return dict(status=status, rho=out[0], u=out[1:3], T=out[3], p=out[4])


def work(case):
    """Per node: fields in and out (FP64) once; per step the 26 values read
    and written once, and the arithmetic of the scheme (32 reconstructions
    per stencil phase, the moments, equilibria and updates)."""
    size = 4 if case["prec"] == "f32" else 8
    bytes_, flops = 0.0, 0.0
    for _, nx, ny, rk, fm, steps, _ in _members(case):
        n, phases = nx * ny, 2 if rk == 1 else 1
        bytes_ += n * (9 * 8 + steps * 52.0 * size)
        flops += n * steps * phases * (32.0 * (46 if fm else 8) + 700.0)
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------- the scheme in FP64
EX = (0, 1, 0, -1, 0, 1, -1, -1, 1, 2, 0, -2, 0)
EY = (0, 0, 1, 0, -1, 1, 1, -1, -1, 0, 2, 0, -2)


def _equilibrium(rho, ux, uy, T, K, RTc, Tc):
    """The 13 f and 13 h equilibria as lists of fields."""
    s = math.sqrt(RTc)
    u, v, T = ux / s, uy / s, T / Tc
    a, c = u * u, v * v
    s2, pc, T2 = a + c, a * c, T * T
    T3 = T2 * T
    f, h = [None] * 13, [None] * 13
    f[0] = 1 + 2.5 * T2 + 2.5 * T * (s2 - 1) + 0.25 * (a * a + c * c) + pc - 1.25 * s2
    h[0] = (T3 * (1.25 * K + 20 / 3) + T2 * ((1.25 * K + 11.25) * s2 - 1.25 * K - 5)
            + T * (0.125 * K * (s2 * s2 + 2 * pc) - 0.625 * K * s2 + 0.5 * K + 2.5 * s2 * s2 + 2.5 * pc - 5 * s2 + 1)
            + s2 ** 3 / 8 + 0.25 * pc * s2 - 0.625 * s2 * s2 + 0.5 * s2)
    for k, (A, C, U) in enumerate(((a, c, u), (c, a, v))):
        E = -T2 + T * (2 / 3 - 1.5 * A - 0.5 * C) + (2 / 3) * A - A * A / 6 - 0.5 * pc
        O = U * (2 / 3 - T - A / 6 - 0.5 * C)
        f[1 + k], f[3 + k] = E + O, E - O
        E = (T3 * (-0.5 * K - 8 / 3) + T2 * (-(0.75 * K + 6.5) * A - (0.25 * K + 2.5) * C + K / 3 + 4 / 3)
             + T * (-(K / 12 + 19 / 12) * A * A - (0.25 * K + 3.5) * A * C + (K / 3 + 7 / 3) * A - 0.25 * C * C + C / 3)
             - A ** 3 / 12 - A * A * C / 3 + A * A / 3 - 0.25 * A * C * C + A * C / 3)
        O = U * (T2 * (-0.5 * K - 3) + T * (-(K / 12 + 7 / 6) * A - (0.25 * K + 2.5) * C + K / 3 + 4 / 3)
                 - A * A / 12 - A * C / 3 + A / 3 - 0.25 * C * C + C / 3)
        h[1 + k], h[3 + k] = E + O, E - O
        E = 0.125 * T2 + T * (0.25 * A - 1 / 24) + (A * A - A) / 24
        O = U * (0.25 * T + (A - 1) / 12)
        f[9 + k], f[11 + k] = E + O, E - O
        E = (T3 * (K / 16 + 1 / 3) + T2 * ((0.125 * K + 17 / 16) * A + C / 16 - K / 48 - 1 / 12)
             + T * ((K / 48 + 1 / 3) * A * A - (K / 48 + 7 / 48) * A + 0.125 * A * C - C / 48)
             + (A ** 3 + A * A * C - A * A - A * C) / 48)
        O = U * (T2 * (0.125 * K + 0.75) + T * ((K / 24 + 11 / 24) * A - K / 24 - 1 / 6 + 0.125 * C)
                 + (A * A + A * C - A - C) / 24)
        h[9 + k], h[11 + k] = E + O, E - O
    for i, (su, sv) in zip((5, 6, 7, 8), ((1, 1), (-1, 1), (-1, -1), (1, -1))):
        f[i] = 0.25 * (T + a + su * u) * (T + c + sv * v)
        h[i] = (T3 * (K / 8 + 2 / 3) + T2 * (K / 8 + 1.125) * s2
                + T * ((K / 8 + 1.5) * pc + 0.125 * (a * a + c * c)) + 0.125 * pc * s2
                + su * u * (T2 * (K / 8 + 0.75) + T * ((K / 8 + 1.125) * c + 0.125 * a) + 0.125 * c * s2)
                + sv * v * (T2 * (K / 8 + 0.75) + T * ((K / 8 + 1.125) * a + 0.125 * c) + 0.125 * a * s2)
                + su * sv * u * v * (T * (K / 8 + 0.75) + 0.125 * s2))
    return [rho * x for x in f], [rho * RTc * x for x in h]


class _Exact:
    """Samples of one flow and size, stacked: fields are [sample, x, y]."""

    def __init__(self, cfgs, fields, dev):
        c0 = cfgs[0]
        one = lambda k: torch.tensor([float(c[k]) for c in cfgs], dtype=torch.float64, device=dev).view(-1, 1, 1)  # noqa: E731
        self.dev, self.fm, self.rk = dev, c0["FMETHOD"], c0["RKMETHOD"]
        self.mu, self.Pr = one("mu"), one("Pr")
        self.per = (bool(c0["periodicX"]), bool(c0["periodicY"]))
        ct = np.asarray(c0["cellType"])[c0["bnd"]]
        self.type = torch.from_numpy(ct).to(dev)
        self.n = tuple(ct.shape)
        self.solid = self.type == 2
        self.edges = tuple(bool((ct != np.roll(ct, 1, k)).any() and (ct == 2).any()) for k in (0, 1))
        self.b = 2 / (c0["gamma"] - 1)
        self.Tc = c0["Tc_Tref"] * c0["T_ref"]
        self.c = math.sqrt(self.Tc)  # R = 1
        dx = c0.get("dx_array") if c0.get("dx_array") is not None else np.full(self.n[0], c0["dx"])
        dy = c0.get("dy_array") if c0.get("dy_array") is not None else np.full(self.n[1], c0["dy"])
        self.dt = c0["CFL"] * min(dx.min(), dy.min()) / (2 * self.c)
        self.d = (torch.from_numpy(dx.copy()).to(dev).view(-1, 1), torch.from_numpy(dy.copy()).to(dev).view(1, -1))
        m = [torch.from_numpy(np.stack([a[k] for a in fields])).to(dev) for k in range(4)]
        self.f, self.h = self.eq(*m)
        self.flu = (self.type == 0).unsqueeze(0)

    def eq(self, rho, ux, uy, T):
        return _equilibrium(rho, ux, uy, T, self.b - 2, self.Tc, self.Tc)

    def macro(self, f, h):
        rho = sum(f)
        ux = self.c * sum(EX[i] * f[i] for i in range(13) if EX[i]) / rho
        uy = self.c * sum(EY[i] * f[i] for i in range(13) if EY[i]) / rho
        T = 2 * (sum(h) / rho - 0.5 * (ux * ux + uy * uy)) / self.b
        return rho, ux, uy, T

    def index(self, axis, shift):
        n = self.n[axis]
        k = torch.arange(n, device=self.dev) + shift
        return k % n if self.per[axis] else k.clamp(0, n - 1)

    def step_index(self, axis, k, shift):
        n = self.n[axis]
        return (k + shift) % n if self.per[axis] else (k + shift).clamp(0, n - 1)

    def face(self, v, e, axis):
        s, ae = (1 if e > 0 else -1), abs(e) * self.c
        L = 5 if self.fm else 3
        idx = [self.index(axis, s * (j - L // 2)) for j in range(L)]
        S = [v.index_select(axis + 1, k) for k in idx]
        if self.edges[axis]:
            sol = [self.solid.index_select(axis, k) for k in idx]
            left = torch.ones_like(sol[0])
            for j in range(L - 1):
                for g, at in ((1, j), (-1, j + 1)):
                    here = left & (sol[j] & ~sol[j + 1] if g > 0 else ~sol[j] & sol[j + 1])
                    k1, k2 = self.step_index(axis, idx[at], s * g), self.step_index(axis, idx[at], 2 * s * g)
                    ext = 2 * v.index_select(axis + 1, k1) - v.index_select(axis + 1, k2)
                    S[at] = torch.where(here, ext, S[at])
                    if 0 <= at - g < L:
                        S[at - g] = torch.where(here, ext, S[at - g])
                left = left & (sol[j] == sol[j + 1])
        q = [ae * x for x in S]
        if not self.fm:
            a, b = q[2] - q[1], q[1] - q[0]
            return q[1] + 0.5 * torch.where(a * b > 0, torch.where(a.abs() < b.abs(), a, b), torch.zeros_like(a))
        q0, q1, q2, q3, q4 = q
        b0 = 13 / 12 * (q0 - 2 * q1 + q2) ** 2 + 0.25 * (q0 - 4 * q1 + 3 * q2) ** 2
        b1 = 13 / 12 * (q1 - 2 * q2 + q3) ** 2 + 0.25 * (q1 - q3) ** 2
        b2 = 13 / 12 * (q2 - 2 * q3 + q4) ** 2 + 0.25 * (3 * q2 - 4 * q3 + q4) ** 2
        w0, w1, w2 = 0.1 / (1e-6 + b0) ** 2, 0.6 / (1e-6 + b1) ** 2, 0.3 / (1e-6 + b2) ** 2
        return (w0 * (2 * q0 - 7 * q1 + 11 * q2) + w1 * (-q1 + 5 * q2 + 2 * q3) + w2 * (2 * q2 + 5 * q3 - q4)) / (
            6 * (w0 + w1 + w2))

    def divergence(self, f, h):
        """dt div F of every direction, f and h."""
        E = (EX, EY)
        FF, HH = ({(i, a): self.face(v[i], E[a][i], a) for i in range(1, 13) for a in (0, 1) if E[a][i]} for v in (f, h))
        if bool(self.solid.any()):
            fin, fout = torch.zeros_like(f[0]), torch.zeros_like(f[0])
            for a, into, out in ((0, (1, 5, 8, 9), (3, 6, 7, 11)), (0, (3, 6, 7, 11), (1, 5, 8, 9)),
                                 (1, (2, 5, 6, 10), (4, 8, 7, 12)), (1, (4, 7, 8, 12), (2, 6, 5, 10))):
                k = self.index(a, -1 if E[a][into[0]] > 0 else 1)
                near = (~self.solid.index_select(a, k)).double()
                for i, o in zip(into, out):
                    fin += near * FF[i, a].index_select(a + 1, k) / self.d[a]
                    fout += near * f[o] * (abs(E[a][o]) * self.c) / self.d[a]
            alpha = torch.where(fout != 0, fin / fout, torch.zeros_like(fin))
            for (i, a), v in list(FF.items()):
                FF[i, a] = torch.where(self.solid, alpha * abs(E[a][i]) * self.c * f[i], v)
                HH[i, a] = torch.where(self.solid, alpha * abs(E[a][i]) * self.c * h[i], HH[i, a])
        zero = torch.zeros_like(f[0])
        out = []
        for G in (FF, HH):
            D = [zero]
            for i in range(1, 13):
                t = zero
                for a in (0, 1):
                    if E[a][i]:
                        up = G[i, a].index_select(a + 1, self.index(a, -1 if E[a][i] > 0 else 1))
                        t = t + self.dt / self.d[a] * (G[i, a] - up)
                D.append(t)
            out.append(D)
        return out

    def rates(self, m):
        q = m[0] * m[3] / self.mu  # 1/tau_f; 1/tau_h = Pr q; 1/tau_hf = (Pr - 1) q
        return q, self.Pr * q, (self.Pr - 1) * q

    def keep(self, new, old):
        return [torch.where(self.flu, a, b) for a, b in zip(new, old)]

    def step(self):
        f, h, dt = self.f, self.h, self.dt
        m = self.macro(f, h)
        q, qh, g = self.rates(m)
        fe, he = self.eq(*m)
        eu = [self.c * (EX[i] * m[1] + EY[i] * m[2]) for i in range(13)]
        w = dt if self.rk == 0 else dt / 2
        f1 = [(f[i] + w * q * fe[i]) / (1 + w * q) for i in range(13)]
        h1 = [(h[i] - w * g * eu[i] * (fe[i] - f1[i]) + w * qh * he[i]) / (1 + w * qh) for i in range(13)]
        if self.rk == 0:
            f1, h1 = self.keep(f1, f), self.keep(h1, h)
            Df, Dh = self.divergence(f1, h1)
            fn = [f[i] - Df[i] + dt * q * (fe[i] - f1[i]) for i in range(13)]
            hn = [h[i] - Dh[i] + dt * qh * (he[i] - h1[i]) - dt * eu[i] * g * (fe[i] - f1[i]) for i in range(13)]
            self.f, self.h = self.keep(fn, f), self.keep(hn, h)
            return
        f2 = [(f[i] - w * q * (fe[i] - f1[i]) + w * q * fe[i]) / (1 + w * q) for i in range(13)]
        h2 = [(h[i] - w * eu[i] * g * (f1[i] - f2[i]) - w * qh * (he[i] - h1[i]) + w * qh * he[i]) / (1 + w * qh)
              for i in range(13)]
        f2, h2 = self.keep(f2, f), self.keep(h2, h)
        Df, Dh = self.divergence(f2, h2)
        m3 = self.macro([a - b for a, b in zip(f, Df)], [a - b for a, b in zip(h, Dh)])
        q3, qh3, g3 = self.rates(m3)
        f3e, h3e = self.eq(*m3)
        eu3 = [self.c * (EX[i] * m3[1] + EY[i] * m3[2]) for i in range(13)]
        f3 = [(f[i] - Df[i] + w * q * (fe[i] - f2[i]) + w * q3 * f3e[i]) / (1 + w * q3) for i in range(13)]
        cpl = [w * (eu[i] * g * (fe[i] - f2[i]) + eu3[i] * g3 * (f3e[i] - f3[i])) for i in range(13)]
        h3 = [(h[i] - Dh[i] - cpl[i] + w * qh * (he[i] - h2[i]) + w * qh3 * h3e[i]) / (1 + w * qh3) for i in range(13)]
        f3, h3 = self.keep(f3, f), self.keep(h3, h)
        D3f, D3h = self.divergence(f3, h3)
        fn = [f[i] - 0.5 * (Df[i] + D3f[i]) + w * (q * (fe[i] - f2[i]) + q3 * (f3e[i] - f3[i])) for i in range(13)]
        hn = [h[i] - 0.5 * (Dh[i] + D3h[i]) + w * (qh * (he[i] - h2[i]) + qh3 * (h3e[i] - h3[i])) - cpl[i]
              for i in range(13)]
        self.f, self.h = self.keep(fn, f), self.keep(hn, h)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    members, samples = _members(case), _samples(case, seed)
    groups = {}
    for k, m in enumerate(members):
        groups.setdefault(m, []).append(k)
    got, residuals = [None] * len(members), []
    for m, ks in groups.items():
        x = _Exact([samples[k][0] for k in ks], [samples[k][1] for k in ks], dev)
        for _ in range(m[5]):
            T0 = x.macro(x.f, x.h)[3] if case["entry"] == "solver" else None
            x.step()
            if T0 is not None:
                d = torch.where(x.flu, x.macro(x.f, x.h)[3] - T0, torch.zeros_like(T0))
                residuals.append(float((d * d).mean().sqrt()))
        rho, ux, uy, T = (v.cpu() for v in x.macro(x.f, x.h))
        for j, k in enumerate(ks):
            got[k] = (rho[j], torch.stack([ux[j], uy[j]]), T[j], rho[j] * T[j])
    if case["entry"] == "server":
        return [dict(status=None, rho=r.numpy(), u=u.numpy(), T=T.numpy()) for r, u, T, _ in got]
    if case["entry"] == "solver":
        r, u, T, p = got[0]
        return dict(status=None, residuals=np.array(residuals), rho=r.numpy(), u=u.numpy(), T=T.numpy(), p=p.numpy())
    flat = lambda v: torch.cat([x.reshape(-1) for x in v])  # noqa: E731
    u = torch.stack([flat([g[1][0] for g in got]), flat([g[1][1] for g in got])])
    return dict(status=None, rho=flat([g[0] for g in got]), u=u, T=flat([g[2] for g in got]), p=flat([g[3] for g in got]))
