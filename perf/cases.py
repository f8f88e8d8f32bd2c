"""Timed workloads of the engine, through the calls a user's program makes.

Each case is one pass of work a seismic inversion program has the engine do: a
shot's forward modeling, a survey's Waveform gradient (device and host
buffers), a line search's misfit, a differentiable forward with a correlation
misfit, the exact discrete adjoint, a large grid, checkpointed recomputation,
velocity receivers, many uneven problems at once.  ``exact`` restates the same
passes in plain torch in 64 bits (masked whole-array updates, no code of the
package).
"""
import math

import numpy as np
import torch

from swit_gb300 import Engine, MultiEngine, misfit
from swit_gb300.autograd import propagate

VMIN, VMAX = 1500.0, 4700.0


def listed():
    return [
        # the smallest call: one shot of forward modeling on a small model (a quick look, a unit
        # test of a user's script); a few hundred short steps, nothing to batch
        dict(name="forward, 1 shot 101x51", kind="forward", nx=101, nz=51, npml=20, ns=1, nt=600),
        # the small survey of the reference's first examples: 5 shots, the whole gradient
        dict(name="gradient, 5 shots 201x101", kind="gradient", nx=201, nz=101, npml=40, ns=5, nt=2000),
        # the headline workload: one inversion iteration of a Marmousi-like survey
        dict(name="gradient, 49 shots 481x141", kind="gradient", nx=481, nz=141, npml=40, ns=49, nt=4000),
        # one trial step of a line search on that survey: forward without strips, misfit only
        dict(name="misfit, 49 shots 481x141", kind="misfit", nx=481, nz=141, npml=40, ns=49, nt=2000),
        # an iteration whose model and data live in host memory (files read by numpy), odd sizes
        dict(name="host gradient, 12 shots 333x117", kind="host", nx=333, nz=117, npml=30, ns=12, nt=1501),
        # the differentiable path with a correlation misfit on the thrust-fold grid; records long
        # enough for the waves to reach every receiver (the misfit divides by the trace's norm)
        dict(name="correlation, 40 shots 501x171", kind="correlation", nx=501, nz=171, npml=40, ns=40, nt=4000),
        # the exact discrete adjoint (model and source gradients)
        dict(name="exact adjoint, 10 shots 241x121", kind="exact", nx=241, nz=121, npml=20, ns=10, nt=1200),
        # a few shots of the large grid, whose fields exceed the caches
        dict(name="gradient, 3 shots 2001x601", kind="gradient", nx=2001, nz=601, npml=60, ns=3, nt=1500),
        # a mid-size grid under a memory budget: checkpoints instead of strips
        dict(name="checkpointed, 10 shots 801x301", kind="checkpoint", nx=801, nz=301, npml=40, ns=10, nt=1600,
             every=160),
        # vertical-velocity receivers, no free surface
        dict(name="vz receivers, 8 shots 401x151", kind="velocity", nx=401, nz=151, npml=35, ns=8, nt=1500),
        # many independent uneven problems stepped together (nx, nz, ns, nt are the largest)
        dict(name="multi, 6 uneven problems", kind="multi", nx=701, nz=251, npml=40, ns=12, nt=1500, count=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed kinds: grids from the smallest to the largest listed ones (aspect
    ratios as there), shots and steps over their range, bounded by the largest listed cost."""
    kind = rng.choice(["forward", "gradient", "gradient", "misfit", "host", "correlation", "exact", "checkpoint",
                       "velocity", "multi"])
    top = {"gradient": 2001, "forward": 2001, "misfit": 1001, "checkpoint": 1001}.get(kind, 701)
    nx = _log(rng, 61, top)
    nz = max(41, int(nx * rng.uniform(0.28, 0.6)))
    npml = rng.randint(12, 60)
    nt = _log(rng, 300, 4000)
    ns = _log(rng, 1, 50)
    if kind == "correlation":  # the waves reach every receiver
        nx = min(nx, 440)
        nz = max(41, min(nz, nx // 2))
        nt = int(nx * rng.uniform(8.0, 9.0))
    points = (nx + 2 * npml) * (nz + 2 * npml)
    count = rng.randint(3, 7) if kind == "multi" else 1
    limit = 4e10 if kind in ("exact", "multi") else 1.0e11  # shots x steps x points; memory and time
    while ns > 1 and float(ns) * nt * points * count > limit:
        ns -= 1
    while nt > 200 and kind != "correlation" and float(ns) * nt * points * count > limit:
        nt = int(0.9 * nt)
    c = dict(kind=kind, nx=nx, nz=nz, npml=npml, ns=ns, nt=nt)
    if kind == "checkpoint":
        c["every"] = max(8, int(nt * rng.uniform(0.04, 0.3)))
    if kind == "multi":
        c["count"] = count
    return c


# ------------------------------------------------------------------ inputs
def _problems(case):
    """The problems of a case: one, or the uneven ones of a multi-problem case."""
    if case["kind"] != "multi":
        return [case]
    out = []
    for i in range(case["count"]):
        f = [((i * k) % 7) / 6.0 for k in (1, 3, 5, 2)]  # spreads of nx, nz, ns, nt
        out.append(dict(case, nx=max(48, int(case["nx"] * (1 - 0.6 * f[0]))), nz=max(32, int(case["nz"] * (1 - 0.5 * f[1]))),
                        ns=max(1, int(case["ns"] * (1 - 0.6 * f[2]))), nt=max(100, int(case["nt"] * (1 - 0.4 * f[3])))))
    return out


def _inputs(c, seed):
    """Model, geometry, source functions and observed traces of one problem.  Models are
    layered with smooth anomalies, sources integrated Ricker wavelets, observed traces a
    direct and two reflected arrivals per receiver, about as strong as the synthetics."""
    rng = np.random.default_rng(seed)
    nx, nz, ns, nt = c["nx"], c["nz"], c["ns"], c["nt"]
    dx = 10.0 if nx > 1000 else 25.0
    dt = float(np.float32(0.45 * dx / VMAX))
    f0 = 0.1 * VMIN / dx  # ten points per shortest dominant wavelength
    x, z = np.arange(nx) * dx, np.arange(nz) * dx
    trend = VMIN + (0.8 * VMAX - VMIN) * z / z[-1]
    steps = np.sort(rng.uniform(0.15, 0.95, 6)) * z[-1]
    trend = trend + sum(rng.uniform(-80.0, 140.0) * (z > s) for s in steps)
    vp = np.repeat(trend[None, :], nx, axis=0)
    for _ in range(6):
        cx, cz, r = rng.uniform(0, x[-1]), rng.uniform(0.2, 0.9) * z[-1], rng.uniform(0.05, 0.2) * x[-1]
        vp += rng.choice([-250.0, 250.0]) * np.exp(-((x[:, None] - cx) ** 2 + (z[None, :] - cz) ** 2) / (r * r))
    vp = np.clip(vp, VMIN, VMAX).astype(np.float32)
    vp[:, : max(2, nz // 12)] = VMIN
    rho = (310.0 * vp.astype(np.float64) ** 0.25).astype(np.float32)
    sx = np.linspace(0.0, x[-1], ns) if ns > 1 else np.array([x[-1] / 2])
    src_xz = np.stack([sx, np.full(ns, 2 * dx)], axis=1).astype(np.float32)
    rec_xz = np.stack([x, np.full(nx, 2 * dx)], axis=1).astype(np.float32)
    t = np.arange(nt) * dt
    a = (np.pi * f0 * (t - 1.2 / f0)) ** 2
    wav = (1 - 2 * a) * np.exp(-a)
    src = np.concatenate([[0.0], np.cumsum(0.5 * (wav[1:] + wav[:-1]))])
    src = (src[None, :] * rng.uniform(0.9, 1.1, (ns, 1))).astype(np.float32)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tt = torch.arange(nt, device=dev, dtype=torch.float32) * dt
    obs = torch.empty((ns, nx, nt), device=dev, dtype=torch.float32)
    depths = [0.0] + [float(d) for d in rng.uniform(0.3, 0.9, 2) * z[-1]]
    amps = [1.0] + [float(d) for d in rng.uniform(-0.4, 0.4, 2)]
    scale = 0.5 * dt * float(np.abs(src).max())
    xr = torch.as_tensor(x, device=dev, dtype=torch.float32)
    for s in range(ns):
        obs[s].zero_()
        for d, am in zip(depths, amps):
            r = torch.sqrt((xr - float(sx[s])) ** 2 + (2 * d) ** 2)
            b = (math.pi * f0 * (tt[None, :] - 1.2 / f0 - (r / (VMIN + 0.25 * d))[:, None])) ** 2
            obs[s] += (scale * am / torch.sqrt(1 + r / (4 * dx)))[:, None] * (1 - 2 * b) * torch.exp(-b)
    return dict(vp=vp, rho=rho, src_xz=src_xz, rec_xz=rec_xz, src=src, obs=obs, dx=dx, dt=dt)


def _options(case):
    if case["kind"] == "exact":
        return dict(adjoint="exact")
    if case["kind"] == "checkpoint":
        return dict(checkpoint_every=case["every"])
    if case["kind"] == "velocity":
        return dict(receiver_component="vz", free_surface=0)
    return {}


def prepare(case, seed):
    probs = _problems(case)
    ins = [_inputs(c, seed * 1000 + i) for i, c in enumerate(probs)]
    args = [dict(nx=c["nx"], nz=c["nz"], npml=c["npml"], nt=c["nt"], dx=d["dx"], dt=d["dt"], src_xz=d["src_xz"],
                 rec_xz=d["rec_xz"]) for c, d in zip(probs, ins)]
    if case["kind"] == "multi":
        m = MultiEngine(args)
        for e, d in zip(m.engines, ins):
            e.set_model(d["vp"], d["rho"])
        return dict(kind="multi", engine=m, srcs=[torch.from_numpy(d["src"]).cuda() for d in ins],
                    obss=[d["obs"] for d in ins])
    d = ins[0]
    e = Engine(**args[0], **_options(case))
    if case["kind"] == "host":
        def pin(a):
            return torch.as_tensor(a).cpu().pin_memory()
        return dict(kind="host", engine=e, vp=pin(d["vp"]), rho=pin(d["rho"]), src=pin(d["src"]), obs=pin(d["obs"]))
    if case["kind"] == "correlation":
        vp = torch.from_numpy(d["vp"]).cuda().requires_grad_(True)
        return dict(kind="correlation", engine=e, vp=vp, rho=torch.from_numpy(d["rho"]).cuda(),
                    src=torch.from_numpy(d["src"]).cuda(), obs=d["obs"], dt=d["dt"])
    e.set_model(torch.from_numpy(d["vp"]).cuda(), torch.from_numpy(d["rho"]).cuda())
    return dict(kind=case["kind"], engine=e, src=torch.from_numpy(d["src"]).cuda(), obs=d["obs"])


def run(state):
    e, kind = state["engine"], state["kind"]
    if kind == "forward":
        return e.forward(state["src"], save_boundary=False)
    if kind == "misfit":
        return e.misfit_l2(state["src"], state["obs"])
    if kind in ("gradient", "checkpoint"):
        return e.gradient_l2(state["src"], state["obs"])
    if kind == "host":
        e.set_model(state["vp"], state["rho"])
        return e.gradient_l2(state["src"], state["obs"], return_seis=True)
    if kind == "correlation":
        seis = propagate(e, state["vp"], state["rho"], state["src"])
        loss = misfit.global_correlation(seis, state["obs"], state["dt"])
        (grad,) = torch.autograd.grad(loss, state["vp"])
        return dict(loss=loss.detach(), seis=seis.detach(), grad=grad)
    if kind == "exact":
        seis = e.forward(state["src"], save_boundary=True)
        grad, src_grad = e.backward_exact(state["obs"])
        return dict(seis=seis, grad=grad, src_grad=src_grad)
    if kind == "velocity":
        seis = e.forward(state["src"], save_boundary=True)
        grad, fw, bk = e.backward(state["obs"])
        return dict(seis=seis, grad=grad, illum_fw=fw, illum_bk=bk)
    return e.gradient_l2(state["srcs"], state["obss"])


def work(case):
    total = dict(bytes=0.0, flops=0.0)
    for c in _problems(case):
        pml = (c["nx"] + 2 * c["npml"]) * (c["nz"] + 2 * c["npml"])
        inner = c["nx"] * c["nz"]
        traces = 4.0 * c["ns"] * c["nx"] * c["nt"]
        per_step = 25.0 * pml  # p: 11, u: 7, w: 7
        move = 4.0 * c["ns"] * c["nt"] + 2 * 4.0 * pml + traces  # source, coefficients, seismograms or observed traces
        kind = c["kind"]
        if kind == "exact":
            per_step += 27.0 * pml  # the transposed updates and the gradient sum
        elif kind not in ("forward", "misfit"):
            per_step += 25.0 * pml + 32.0 * inner  # adjoint; reconstruction and imaging
        if kind not in ("forward", "misfit"):
            move += 3 * 4.0 * inner
        if kind in ("host", "correlation", "exact", "velocity"):
            move += traces
        total["flops"] += per_step * c["ns"] * (c["nt"] - 1)
        total["bytes"] += move
    return total


# ------------------------------------------------------------------ the same in 64 bits
class _Exact:
    """fd2dmpi's scheme on whole (shot, x, z) arrays in float64: every update is masked to
    its index range, neighbours come from torch.roll."""

    def __init__(self, c, d):
        self.c, self.d = c, d
        L, nx, nz = c["npml"], c["nx"], c["nz"]
        self.L, self.NX, self.NZ = L, nx + 2 * L, nz + 2 * L
        self.flag = 0 if c["kind"] == "velocity" else 1
        self.dev = d["obs"].device
        self.dx, self.dt = float(np.float32(d["dx"])), float(np.float32(d["dt"]))
        self.c1, self.c2 = 9.0 / 8.0, -1.0 / 24.0
        col = np.arange(c["ns"])
        self.rows = torch.as_tensor(col, device=self.dev)
        idx = (d["src_xz"] / np.float32(d["dx"])).astype(np.int64)
        self.sx = torch.as_tensor(idx[:, 0] + L, device=self.dev)  # 0-based on the padded grid
        self.sz = torch.as_tensor(np.maximum(idx[:, 1], 1) + L, device=self.dev)
        rec = (d["rec_xz"] / np.float32(d["dx"])).astype(np.int64)
        self.rx = torch.as_tensor(rec[:, 0] + L, device=self.dev)
        self.rz = torch.as_tensor(np.maximum(rec[:, 1], 1) + L, device=self.dev)
        act = (idx[:, 0] + 1 > 2) & (idx[:, 0] + 1 < nx - 1) & (idx[:, 1] + 1 > 3) & (idx[:, 1] + 1 < nz - 1)
        self.subtract = torch.as_tensor(act.astype(np.float64), device=self.dev)
        self.src = torch.as_tensor(d["src"], device=self.dev).double()
        self.model(torch.as_tensor(d["vp"], device=self.dev).double(), torch.as_tensor(d["rho"], device=self.dev).double())

    def pad(self, m):
        L = self.L
        m = torch.cat([m[:1].expand(L, -1), m, m[-1:].expand(L, -1)], dim=0)
        return torch.cat([m[:, :1].expand(-1, L), m, m[:, -1:].expand(-1, L)], dim=1)

    def model(self, vp, rho):
        L, NX, NZ = self.L, self.NX, self.NZ
        v, r = self.pad(vp), self.pad(rho)
        self.vp = vp
        self.A = r * v * v * self.dt / self.dx
        self.B = self.dt / (r * self.dx)
        a = (L - 1) * self.dx
        vmin = float(vp[:, 1:].min())
        k = 3.0 * vmin * math.log(1000.0) / (2.0 * a)
        prof = k * (np.arange(L) * self.dx / a) ** 2  # prof[i]: i cells from the inner edge
        damp = np.zeros((NX, NZ))
        for i in range(L):  # sides, then top and bottom over their trapezoids
            damp[L - 1 - i, :] = prof[i]
            damp[NX - L + i, :] = prof[i]
        for i in range(L):
            damp[L - i: NX - L + i, L - 1 - i] = prof[i]
            damp[L - i: NX - L + i, NZ - L + i] = prof[i]
        damp = torch.as_tensor(damp, device=self.dev)
        self.fp = 1.0 - damp * self.dt
        self.fu = 1.0 - 0.5 * (damp + torch.roll(damp, -1, 0)) * self.dt
        self.fw = 1.0 - 0.5 * (damp + torch.roll(damp, -1, 1)) * self.dt

    def box(self, x0, x1, z0, z1):
        """Mask of 1-based inclusive ranges."""
        m = torch.zeros((self.NX, self.NZ), dtype=torch.bool, device=self.dev)
        m[x0 - 1:x1, z0 - 1:z1] = True
        return m

    def coef(self, a, m):
        return torch.where(m, a, torch.zeros_like(a))

    def factor(self, f, m):
        return torch.where(m, f, torch.ones_like(f))

    def div(self, u, w):
        r = torch.roll
        return self.c1 * (u - r(u, 1, 1) + w - r(w, 1, 2)) + self.c2 * (r(u, -1, 1) - r(u, 2, 1) + r(w, -1, 2) - r(w, 2, 2))

    def grad_x(self, p):
        r = torch.roll
        return self.c1 * (r(p, -1, 1) - p) + self.c2 * (r(p, -2, 1) - r(p, 1, 1))

    def grad_z(self, p):
        r = torch.roll
        return self.c1 * (r(p, -1, 2) - p) + self.c2 * (r(p, -2, 2) - r(p, 1, 2))

    def zeros(self):
        return torch.zeros((self.c["ns"], self.NX, self.NZ), dtype=torch.float64, device=self.dev)

    def setup_forward(self):
        L, NX, NZ = self.L, self.NX, self.NZ
        fs = L + 1
        mp, mu, mw = self.box(3, NX - 2, fs + 1, NZ - 2), self.box(2, NX - 2, fs, NZ - 1), self.box(2, NX - 1, fs, NZ - 2)
        self.fwd = [self.factor(self.fp, mp), self.coef(self.A, mp), self.factor(self.fu, mu), self.coef(self.B, mu),
                    self.factor(self.fw, mw), self.coef(self.B, mw)]

    def forward_step(self, p, u, w, it, src):
        """Out-of-place step `it` (differentiable); it = 2 .. nt."""
        Fp, Ap, Fu, Bu, Fw, Bw = self.fwd
        L = self.L
        p = Fp * p - Ap * self.div(u, w)
        p = p.index_put((self.rows, self.sx, self.sz), self.dt * src[:, it - 1], accumulate=True)
        if self.flag:
            p = torch.cat([p[:, :, : L - 1], -p[:, :, L + 1: L + 2], p[:, :, L:]], dim=2)
        u = Fu * u - Bu * self.grad_x(p)
        w = Fw * w - Bw * self.grad_z(p)
        if self.flag:
            w = torch.cat([w[:, :, : L - 1], w[:, :, L: L + 1], w[:, :, L:]], dim=2)
        return p, u, w

    def record(self, p, w):
        return (w if self.c["kind"] == "velocity" else p)[:, self.rx, self.rz]

    def forward(self, keep):
        c, L = self.c, self.L
        self.setup_forward()
        p, u, w = self.zeros(), self.zeros(), self.zeros()
        seis = torch.zeros((c["ns"], c["nx"], c["nt"]), dtype=torch.float64, device=self.dev)
        strips = [None, [None] * 6]  # of each step: what the reconstruction re-inserts
        i = slice(L, -L)
        zero = None
        for it in range(2, c["nt"] + 1):
            p, u, w = self.forward_step(p, u, w, it, self.src)
            seis[:, :, it - 1] = self.record(p, w)
            if keep:
                pi, ui, wi = p[:, i, i], u[:, i, i], w[:, i, i]
                strips.append([pi[:, :, :3].clone(), pi[:, :, -2:].clone(), pi[:, :2].clone(), pi[:, -2:].clone(),
                               torch.stack([ui[:, 0], ui[:, -2]], 1), wi[:, :, -2].clone()])
        if keep:
            zero = [torch.zeros_like(s) for s in strips[2]] if c["nt"] >= 2 else None
            strips[1] = zero
            self.strips, self.end = strips, (p, u, w)
        return seis

    def backward(self, adj):
        """Reconstruction, adjoint and imaging: (g, illum_fw, illum_bk)."""
        c, L, NX, NZ = self.c, self.L, self.NX, self.NZ
        nx, nz, fs, dt = c["nx"], c["nz"], L + 1, self.dt
        mu, mw, mp = self.box(2, NX - 2, 2, NZ - 1), self.box(2, NX - 1, 2, NZ - 2), self.box(3, NX - 2, 3, NZ - 2)
        Fu, Au, Fw, Aw = self.factor(self.fu, mu), self.coef(self.A, mu), self.factor(self.fw, mw), self.coef(self.A, mw)
        Fp, Bp = self.factor(self.fp, mp), self.coef(self.B, mp)
        i = slice(L, -L)
        A, B = self.A[i, i], self.B[i, i]

        def inner(x0, x1, z0, z1):
            m = torch.zeros((nx, nz), dtype=torch.bool, device=self.dev)
            m[x0 - 1:x1, z0 - 1:z1] = True
            return m
        Bu, Bw = self.coef(B, inner(2, nx - 2, 2, nz - 1)), self.coef(B, inner(2, nx - 1, 2, nz - 2))
        Ap = self.coef(A, inner(3, nx - 2, 3, nz - 2))
        pe, ue, we = (f[:, i, i].clone() for f in self.end)
        pb, ub, wb = self.zeros(), self.zeros(), self.zeros()
        g, fw, bk = (torch.zeros_like(pe) for _ in range(3))
        src = torch.cat([self.src, torch.zeros_like(self.src[:, :1])], dim=1)
        for it in range(c["nt"], 1, -1):
            top, bot, left, right, us, wrow = self.strips[it - 1]
            ub = Fu * ub - Au * self.grad_x(pb)
            wb = Fw * wb - Aw * self.grad_z(pb)
            if self.flag:
                wb[:, 1:NX - 1, fs - 2] = wb[:, 1:NX - 1, fs - 1]
            ue = ue + Bu * self.grad_x(pe)
            we = we + Bw * self.grad_z(pe)
            we[:, :, -2] = wrow
            ue[:, 0], ue[:, -2] = us[:, 0], us[:, 1]
            old = pb
            pb = Fp * pb - Bp * self.div(ub, wb)
            if c["kind"] != "velocity":
                pb.index_put_((self.rows[:, None], self.rx[None], self.rz[None]), dt * adj[:, :, it - 1], accumulate=True)
            pb[:, :, fs - 2] = -pb[:, :, fs]
            pe = pe.index_put((self.rows, self.sx - L, self.sz - L), -dt * src[:, it] * self.subtract, accumulate=True)
            pe = pe + Ap * self.div(ue, we)
            pe[:, :, -2:] = bot
            pe[:, :2], pe[:, -2:] = left, right
            pe[:, :, :3] = top
            new = pb[:, i, i]
            g += pe * (old[:, i, i] - new)
            fw += pe * pe
            bk += new * new
            if c["kind"] == "velocity":
                wb.index_put_((self.rows[:, None], self.rx[None], self.rz[None]), -dt * adj[:, :, it - 1], accumulate=True)
        return -2.0 * g.sum(0) / self.vp, fw.sum(0), bk.sum(0)

    def exact_adjoint(self, adj):
        """Seismograms, dJ/dvp (damping held fixed) and dJ/dsrc for dJ/dseis = adj, by torch's
        autograd over recomputed segments of steps."""
        c = self.c
        vp = self.vp.clone().requires_grad_(True)
        src = self.src.clone().requires_grad_(True)
        rho = torch.as_tensor(self.d["rho"], device=self.dev).double()

        def build():
            v, r = self.pad(vp), self.pad(rho)
            self.A = r * v * v * self.dt / self.dx
            self.setup_forward()

        def segment(p, u, w, lo, hi):
            out = 0.0
            for it in range(lo, hi + 1):
                p, u, w = self.forward_step(p, u, w, it, src)
                seis[:, :, it - 1] = self.record(p, w).detach()
                out = out + (self.record(p, w) * adj[:, :, it - 1]).sum()
            return p, u, w, out
        seis = torch.zeros((c["ns"], c["nx"], c["nt"]), dtype=torch.float64, device=self.dev)
        size = 24
        segs = [(lo, min(lo + size - 1, c["nt"])) for lo in range(2, c["nt"] + 1, size)]
        starts, f = [], (self.zeros(), self.zeros(), self.zeros())
        with torch.no_grad():
            build()
            for lo, hi in segs:
                starts.append(f)
                f = segment(*f, lo, hi)[:3]
        lam = [torch.zeros_like(x) for x in f]
        gv, gs = torch.zeros_like(vp), torch.zeros_like(src)
        for (lo, hi), f in zip(segs[::-1], starts[::-1]):
            build()
            f = [x.detach().requires_grad_(True) for x in f]
            p, u, w, out = segment(*f, lo, hi)
            grads = torch.autograd.grad([p, u, w, out], f + [vp, src], lam + [torch.ones_like(out)])
            lam = list(grads[:3])
            gv += grads[3]
            gs += grads[4]
        return seis, gv, gs


def _live(a, b):
    return ((a * a).sum(-1) > 0) & ((b * b).sum(-1) > 0)


def _correlation(s, o):
    """Global correlation with the reference's adjoint source (which leaves out the mean removal)."""
    live = _live(s, o)
    sn = torch.linalg.vector_norm(s, dim=-1, keepdim=True)
    on = torch.linalg.vector_norm(o, dim=-1, keepdim=True)
    one = torch.ones_like(sn)
    sh, oh = s / torch.where(sn > 0, sn, one), o / torch.where(on > 0, on, one)
    a, b = sh - sh.mean(-1, keepdim=True), oh - oh.mean(-1, keepdim=True)
    corr = (a * b).sum(-1) / torch.sqrt((a * a).sum(-1) * (b * b).sum(-1)).clamp_min(1e-300)
    adj = (sh * corr[..., None] - oh) / torch.where(sn > 0, sn, one)
    zero = torch.zeros_like(corr)
    return torch.where(live, -corr, zero).sum(), torch.where(live[..., None], adj, torch.zeros_like(adj))


def exact(case, seed):
    probs = _problems(case)
    cells = sum(float(c["ns"]) * c["nt"] * (c["nx"] + 2 * c["npml"]) * (c["nz"] + 2 * c["npml"]) for c in probs)
    steps = sum(c["nt"] for c in probs)
    if cells * (3.0 if case["kind"] == "exact" else 1.0) > 2.6e10 or steps > 12000:
        return None  # more than about 20 seconds
    outs = []
    for i, c in enumerate(probs):
        d = _inputs(c, seed * 1000 + i)
        x = _Exact(c, d)
        obs = d["obs"].double()
        kind = c["kind"]
        if kind == "exact":
            s, g, gs = x.exact_adjoint(obs)
            outs.append(dict(seis=s, grad=g, src_grad=gs))
            continue
        with torch.no_grad():
            s = x.forward(keep=kind not in ("forward", "misfit"))
            if kind == "forward":
                outs.append(s)
                continue
            live = _live(s, obs)
            r = (s - obs) * live[..., None]
            value = torch.sqrt((r * r).sum(-1) * x.dt).sum()
            if kind == "misfit":
                outs.append(value)
            elif kind == "correlation":
                loss, adj = _correlation(s, obs)
                outs.append(dict(loss=loss, seis=s, grad=x.backward(adj)[0] / x.dt))
            elif kind == "velocity":
                g, fw, bk = x.backward(obs)
                outs.append(dict(seis=s, grad=g, illum_fw=fw, illum_bk=bk))
            else:
                g, fw, bk = x.backward(r)
                out = dict(grad=g, illum_fw=fw, illum_bk=bk, misfit=value)
                if kind == "host":
                    out["seis"] = s
                outs.append(out)
    return outs if case["kind"] == "multi" else outs[0]
