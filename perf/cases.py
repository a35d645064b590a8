"""The work a user has this package do, as measurable cases.

A pass of most cases is what a run script does between two frames: ``solver.step(k)`` on a
scene in motion (k = the scene files' ``stepsPerRenderUpdate``, 10; 1 for the large plain
FP64 scenes and the smallest one) and a look at the state it leaves.  FP64 runs hand back
the library's own field views in particle order; FP32-mixed runs hand the state back per
particle id in float32, which is how a script that follows particles uses it (the order
changes whenever the lists are rebuilt).  Ensembles are stepped together, and the
differentiable rollout runs forward and backward.

The listed cases, and what each stands for:

* wc2d_tiny_fp64      a test-sized 2D dambreak, one step per call: latency and launches
* wc2d_fp64           the 2D dambreak at its scene-file size, the default (FP64) form
* wc2d_rk4_fp64       a ragged 2D dambreak with RK4, cubic kernel, CSPM and XSPH
* wc3d_fp64           the 3D dambreak at twice the benchmark's spacing, CSPM, leap-frog
* wc3d_full_fp64      the benchmark's 3D dambreak (911,754 fluid + 1,413,114 dummies), FP64
* mui2d_fp64          the mu(I) granular column at its stated size
* dp2d_fp64           the Drucker-Prager column at its stated size (leap-frog, XSPH)
* wc2d_fp32           the 2D dambreak in the FP32-mixed form: launch-bound
* wc3d_full_fp32      the benchmark's 3D dambreak in the FP32-mixed form
* mui2d_large_fp32    a wide mu(I) column (320,000 soil particles, CSPM), FP32-mixed
* ensemble_fp32       64 dambreaks of uneven size stepped as one batch
* rollout_adjoint     a differentiable dambreak: forward, loss and backward

Every scene starts as its block scene with seeded lattice jitter and a seeded smooth
velocity field (a column already in motion), so viscosity, list rebuilds and the return
mapping do what they do in a run.
"""
import math

import numpy as np
import torch

from tisphi_gb300 import scenes
from tisphi_gb300.adjoint import WCRollout
from tisphi_gb300.batch import SceneBatch
from tisphi_gb300.configer_builder import SimConfiger
from tisphi_gb300.params import native_config
from tisphi_gb300.scene import build_scene, scene_geometry
from tisphi_gb300.simulation import Simulation

WC, MUI, DP = 1, 2, 3
SE, LF, RK4 = 1, 2, 4


def _case(kind, precision, method, dim, spacing, size, domain, dt, steps, ti=LF, kernel=1, corr=0, xsph=False,
          boundary=2, name=None):
    c = {"kind": kind, "precision": precision, "method": method, "dim": dim, "spacing": spacing,
         "width": size[0], "height": size[1], "depth": size[2] if dim == 3 else 0.0,
         "domain_x": domain[0], "domain_y": domain[1], "domain_z": domain[2] if dim == 3 else 0.0,
         "dt": dt, "steps": steps, "ti": ti, "kernel": kernel, "corr": corr, "xsph": xsph, "boundary": boundary}
    if name is not None:
        c["name"] = name
    return c


def listed():
    tank2, tank3 = (3.22, 1.6), (3.22, 1.6, 0.5)
    return [
        _case("scene", "fp64", WC, 2, 0.02, (0.6, 0.4), (1.2, 0.8), 1e-4, 1, name="wc2d_tiny_fp64"),
        _case("scene", "fp64", WC, 2, 0.01, (1.2, 0.6), tank2, 1e-4, 10, name="wc2d_fp64"),
        _case("scene", "fp64", WC, 2, 0.0087, (0.93, 0.57), (2.1, 1.1), 5e-5, 2, ti=RK4, kernel=0, corr=1, xsph=True,
              name="wc2d_rk4_fp64"),
        _case("scene", "fp64", WC, 3, 0.0108, (1.2, 0.6, 0.2), tank3, 2e-5, 1, corr=1, name="wc3d_fp64"),
        _case("scene", "fp64", WC, 3, 0.0054, (1.2, 0.6, 0.2), tank3, 2e-5, 1, corr=1, name="wc3d_full_fp64"),
        _case("scene", "fp64", MUI, 2, 0.001, (0.2, 0.1), (0.5, 0.15), 1e-5, 10, ti=SE, name="mui2d_fp64"),
        _case("scene", "fp64", DP, 2, 0.001, (0.2, 0.1), (0.5, 0.15), 1e-6, 10, ti=LF, xsph=True, name="dp2d_fp64"),
        _case("scene", "fp32_mixed", WC, 2, 0.01, (1.2, 0.6), tank2, 1e-4, 10, name="wc2d_fp32"),
        _case("scene", "fp32_mixed", WC, 3, 0.0054, (1.2, 0.6, 0.2), tank3, 2e-5, 10, corr=1, name="wc3d_full_fp32"),
        _case("scene", "fp32_mixed", MUI, 2, 0.00025, (0.2, 0.1), (0.5, 0.15), 2e-6, 10, ti=SE, corr=1,
              name="mui2d_large_fp32"),
        {"name": "ensemble_fp32", "kind": "ensemble", "scenes": 64, "steps": 10},
        _case("rollout", "fp32_mixed", WC, 2, 0.01, (0.6, 0.4), (1.2, 0.8), 1e-4, 40, ti=SE, name="rollout_adjoint"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """A case of the same ranges: every form, solver, integrator, kernel and option, sizes
    spread over their logarithm, block sizes ragged."""
    kind = rng.choice(("wc2d", "wc2d", "wc3d", "wc3d", "soil", "soil", "ensemble", "rollout"))
    if kind == "ensemble":
        return {"kind": "ensemble", "scenes": int(round(_log(rng, 3, 100))), "steps": rng.choice((5, 10, 16))}
    precision = rng.choice(("fp64", "fp32_mixed"))
    aspect = rng.uniform(0.8, 2.5)
    if kind == "rollout":
        n = _log(rng, 300, 4000)
        h = rng.uniform(0.3, 0.5)
        w = h * aspect
        return _case("rollout", "fp32_mixed", WC, 2, round(math.sqrt(w * h / n), 5), (round(w, 4), round(h, 4)),
                     (round(2 * w, 4), round(2 * h, 4)), 5e-5, rng.randint(10, 40), ti=SE)
    ti = rng.choice((SE, LF, LF, LF, RK4))
    kernel = rng.choice((1, 1, 0))
    corr = rng.choice((0, 1))
    xsph = rng.random() < 0.3
    boundary = 2                             # dummy walls: what every scene of the package uses
    if kind == "wc2d":
        n = _log(rng, 300, 50000) if precision == "fp64" else _log(rng, 300, 400000)
        h = rng.uniform(0.4, 0.8)
        w = h * aspect
        sp = round(math.sqrt(w * h / n), 5)
        return _case("scene", precision, WC, 2, sp, (round(w, 4), round(h, 4)), (round(2.2 * w, 4), round(1.9 * h, 4)),
                     round(0.005 * sp, 8), rng.choice((1, 5, 10)), ti, kernel, corr, xsph, boundary)
    if kind == "wc3d":
        n = _log(rng, 2000, 250000) if precision == "fp64" else _log(rng, 2000, 900000)
        h = rng.uniform(0.3, 0.6)
        w = h * aspect
        z = h * rng.uniform(0.3, 1.0)
        sp = round((w * h * z / n) ** (1 / 3), 5)
        return _case("scene", precision, WC, 3, sp, (round(w, 4), round(h, 4), round(z, 4)),
                     (round(1.9 * w, 4), round(1.6 * h, 4), round(1.3 * z, 4)), round(0.0035 * sp, 8),
                     1 if precision == "fp64" else rng.choice((5, 10)), ti, kernel, corr, xsph, boundary)
    n = _log(rng, 500, 60000) if precision == "fp64" else _log(rng, 500, 300000)
    h = rng.uniform(0.08, 0.15)
    w = h * aspect
    method = rng.choice((MUI, DP))
    sp = round(math.sqrt(w * h / n), 7)
    return _case("scene", precision, method, 2, sp, (round(w, 4), round(h, 4)), (round(2.4 * w, 4), round(1.5 * h, 4)),
                 round((0.008 if method == MUI else 0.001) * sp, 9), rng.choice((5, 10)), ti if ti != RK4 else LF, 1,
                 corr, xsph, boundary)


# ---------------------------------------------------------------- preparation

def _scene_dict(c, seed):
    sp, method = c["spacing"], c["method"]
    if method == WC:
        if c["dim"] == 2:
            d = scenes.dambreak_2d(spacing=sp, width=c["width"], height=c["height"], dt=c["dt"], jitter=0.01 * sp,
                                   seed=seed, domain=(c["domain_x"], c["domain_y"]))
        else:
            d = scenes.dambreak_3d(spacing=sp, dt=c["dt"], seed=seed,
                                   domain=(c["domain_x"], c["domain_y"], c["domain_z"]),
                                   size=(c["width"], c["height"], c["depth"]))
    else:
        d = scenes.column_2d(method=method, spacing=sp, dt=c["dt"], seed=seed, width=c["width"], height=c["height"],
                             domain=(c["domain_x"], c["domain_y"]))
    d["Configuration"].update(timeIntegration=c["ti"], kernel=c["kernel"], kernelCorrection=c["corr"],
                              xsph=bool(c["xsph"]), boundary=c["boundary"])
    return d


def _ensemble_dicts(c, seed):
    """The benchmark's ensemble (its block sizes and fluids), jittered by the seed."""
    out = scenes.dambreak_ensemble(c["scenes"])
    for q, d in enumerate(out):
        d["Configuration"]["seed"] = seed * 1009 + q
    return out


def _velocity(c, x, flow, seed):
    """A smooth divergence-free field over the block with a little noise, zero elsewhere."""
    rng = np.random.Generator(np.random.PCG64(seed + 77))
    u = 0.3 if c["method"] == WC else 0.05
    a, b = math.pi / c["width"], math.pi / c["height"]
    amp = u * rng.uniform(0.7, 1.0)
    v = np.zeros_like(x)
    v[flow, 0] = amp * np.sin(a * x[flow, 0]) * np.cos(b * x[flow, 1])
    v[flow, 1] = -amp * (a / b) * np.cos(a * x[flow, 0]) * np.sin(b * x[flow, 1])
    v[flow, :c["dim"]] += 0.01 * u * rng.standard_normal((int(flow.sum()), c["dim"]))
    return v


def prepare(case, seed):
    """The simulation a script has built and set in motion."""
    if case["kind"] == "ensemble":
        return {"case": case, "batch": SceneBatch(_ensemble_dicts(case, seed))}
    d = _scene_dict(case, seed)
    if case["kind"] == "rollout":
        model = WCRollout(d, nsteps=case["steps"], checkpoint_every=20)
        b = torch.tensor([model.stiffness, model.viscosity], dtype=torch.float64)
        return {"case": case, "model": model, "params": b,
                "target": _rollout_target(case)}
    sim = Simulation(SimConfiger(config=d), precision=case["precision"])
    ps = sim.ps
    flow = np.asarray(ps.scene.mat_type) > 0
    ids = ps.field("id0").long().cpu().numpy()
    ps.write_field("v", _velocity(case, np.asarray(ps.scene.x), flow, seed)[ids])
    return {"case": case, "sim": sim}


def _rollout_target(case):
    return 0.9 * case["width"]


def _distance(x, target):
    """Mean squared distance of every particle from a vertical line: the rollout's loss."""
    return ((x[:, 0] - target) ** 2).mean()


# ---------------------------------------------------------------- one pass

def _by_id(ids, f):
    out = torch.empty(f.shape, dtype=torch.float32, device=f.device)
    out[ids] = f.float()
    return out


def _state_names(case):
    """The state a pass leaves.  The plastic strain is left out of the FP32-mixed form's:
    its rate divides by stress rates that pass through zero, so that form's value is noise."""
    if case["method"] == WC:
        return ("x", "v", "density")
    plastic = case["method"] == DP and case["precision"] == "fp64"
    return ("x", "v", "density", "stress", "strain_equ") + (("strain_equ_p",) if plastic else ())


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        b = state["batch"]
        b.step(case["steps"])
        ids = b.field("id0").long()
        return {k: _by_id(ids, b.field(k)) for k in ("x", "v", "density")}
    if case["kind"] == "rollout":
        params = state["params"].clone().requires_grad_(True)
        x = state["model"](params)
        loss = _distance(x, state["target"])
        loss.backward()
        return {"x": x.detach().float(), "loss": loss.detach().float(), "grad": params.grad.float()}
    sim = state["sim"]
    sim.solver.step(case["steps"])
    ps = sim.ps
    if case["precision"] == "fp64":
        names = _state_names(case) + ("pressure", "id0")
        return {k: ps.field(k) for k in names}
    ids = ps.field("id0").long()
    return {k: _by_id(ids, ps.field(k)) for k in _state_names(case)}


# ---------------------------------------------------------------- what a pass cannot do without

def _counts(case):
    """(flow particles, boundary particles) of a case, from its lattice."""
    sp, d = case["spacing"], case["dim"]
    m = lambda e: int(math.floor(e / sp + 0.5 + 1e-5 / sp))
    flow = m(case["width"]) * m(case["height"]) * (m(case["depth"]) if d == 3 else 1)
    x, y, z = case["domain_x"], case["domain_y"], case["domain_z"]
    if d == 2:
        area = 2 * 3 * sp * y + 3 * sp * (x + 6 * sp)
    else:
        area = 3 * sp * ((x + 6 * sp) * (z + 6 * sp) + 2 * x * y + 2 * z * y + 6 * sp * y)
    return flow, int(area / sp ** d)


def work(case):
    if case["kind"] == "ensemble":
        flow, bdy, d, stages, method = 4500 * case["scenes"], 1944 * case["scenes"], 2, 2, WC
        word, corr = 4, 0
    else:
        flow, bdy = _counts(case)
        d, method, corr = case["dim"], case["method"], case["corr"]
        stages = {SE: 1, LF: 2, RK4: 4}[case["ti"]]
        word = 8 if case["precision"] == "fp64" else 4
    pairs = (28 if d == 2 else 113) * flow
    per_pair = 45 if d == 2 else 60          # kernel gradient, continuity, momentum
    if method != WC:
        per_pair += 35                       # velocity gradient, stress divergence
    flops = case["steps"] * pairs * (stages * per_pair + (40 if corr else 12))
    fields = 8 if method == WC else 8 + 11
    moved = 2 * word * fields * flow + word * 4 * bdy
    if case["kind"] == "rollout":
        flops *= 4                           # forward, recomputation and its reverse sweep
    return {"bytes": moved, "flops": flops}


# ---------------------------------------------------------------- 64-bit values

EPS, EPS_F = 1e-8, 1e-4


class _Exact:
    """The step in plain torch float64, in upload order, from the method's formulas."""

    def __init__(self, d, v0=None):
        cfg = SimConfiger(config=d)
        g = scene_geometry(cfg)
        sc = build_scene(cfg, g)
        k = native_config(cfg, g, "fp64")
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.dev)
        self.k, self.g, self.D = k, g, k.dim
        self.method, self.ti = k.solver, k.time_integration
        self.mt = torch.as_tensor(np.asarray(sc.mat_type), device=self.dev)
        self.flow = self.mt > 0
        self.bdy = ~self.flow
        self.mass, self.mV0 = t(sc.mass), t(sc.m_V)
        self.x, self.v, self.rho = t(sc.x), t(sc.v if v0 is None else v0), t(sc.density)
        n = self.n = self.x.shape[0]
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=self.dev)
        self.mV, self.p = self.mV0.clone(), z(n)
        self.vt, self.rt, self.st = z(n, 3), z(n), z(n, 3, 3)
        self.sig, self.eq, self.eqp = z(n, 3, 3), z(n), z(n)
        self.grav = t([k.gravity[q] for q in range(3)])
        self.B, self.visc = k.stiffness, 2 * (k.dim + 2) * k.viscosity
        self.h, self.R = k.smoothing_len, k.support_radius
        self.order = torch.arange(n, device=self.dev)
        if self.method == MUI:
            self.mu = math.tan(k.friction)
        if self.method == DP:
            tf = math.tan(k.friction)
            den = math.sqrt(9 + 12 * tf * tf)
            self.alpha, self.kc = tf / den, 3 * k.cohesion / den
            self.Gm, self.Km = k.E / (2 * (1 + k.poisson)), k.E / (3 * (1 - 2 * k.poisson))
            self.sd = math.sin(k.dilatancy)
            y = self.x[:, 1]
            vs = k.density0 * k.gravity[1] * (y[self.flow].max() - y)
            K0 = 1 - math.sin(k.friction)
            self.sig = torch.diag_embed(torch.stack((K0 * vs, vs, K0 * vs), 1)) * self.flow[:, None, None]
        vsound = {WC: 60.0, MUI: 24.0}.get(self.method) or math.sqrt(k.E / k.density0)
        self.rep_fac = 0.01 * vsound * vsound

    # cells, pairs and the particle order of the plain form
    def _cells(self, x):
        k = self.k
        vs = torch.tensor([k.vdomain_start[q] for q in range(3)], dtype=torch.float64, device=self.dev)
        c = ((x.detach() - vs) / k.grid_size).trunc().long()
        return (c[:, 0] * k.grid_num[1] + c[:, 1]) * k.grid_num[2] + c[:, 2], c

    def pairs(self, x, centres=None, most=40_000_000):
        k, D = self.k, self.D
        xd = x.detach()
        f, c = self._cells(xd)
        G = int(k.grid_num_total)
        srt = torch.argsort(f, stable=True)
        start = torch.zeros(G + 2, dtype=torch.long, device=self.dev)
        start[1:] = torch.cumsum(torch.bincount(f.clamp(0, G), minlength=G + 1), 0)
        xs = xd[srt]
        who = torch.arange(self.n, device=self.dev) if centres is None else torch.nonzero(centres)[:, 0]
        I, J = [], []
        step = max(1, most // (150 if D == 2 else 1200))
        for b in range(0, who.numel(), step):
            w = who[b:b + step]
            for ox in (-1, 0, 1):
                for oy in ((-1, 0, 1) if D == 3 else (0,)):
                    if D == 3:
                        f0 = ((c[w, 0] + ox) * k.grid_num[1] + c[w, 1] + oy) * k.grid_num[2] + c[w, 2]
                    else:
                        f0 = (c[w, 0] + ox) * k.grid_num[1] + c[w, 1]
                    lo, hi = (f0 - 1).clamp(min=0), (f0 + 1).clamp(max=G - 1)
                    ok = lo <= hi
                    jb = start[lo.clamp(max=G)]
                    m = torch.where(ok, start[(hi + 1).clamp(0, G + 1)] - jb, torch.zeros_like(jb))
                    tot = int(m.sum())
                    if not tot:
                        continue
                    q = torch.repeat_interleave(torch.arange(w.numel(), device=self.dev), m, output_size=tot)
                    jj = jb[q] + torch.arange(tot, device=self.dev) - (torch.cumsum(m, 0) - m)[q]
                    r = xd[w][q] - xs[jj]
                    near = ((r * r).sum(1).sqrt() < self.R) & (srt[jj] != w[q])
                    I.append(w[q[near]])
                    J.append(srt[jj[near]])
        return torch.cat(I), torch.cat(J)

    # kernel value and gradient of pairs
    def geometry(self, x, I, J):
        k, h = self.k, self.h
        r = x[I] - x[J]
        rn = (r * r).sum(1).sqrt()
        q = rn / h
        if k.kernel == 1:
            c = (7 / (4 * math.pi) if self.D == 2 else 21 / (2 * math.pi)) / h ** self.D
            a = 1 - 0.5 * q
            W, s = c * a ** 4 * (1 + 2 * q), c * a ** 3 * (-5 * q) / h / rn
        else:
            c = (15 / 7 / math.pi if self.D == 2 else 1.5 / math.pi) / h ** self.D
            W = torch.where(q <= 1, c * (0.5 * q ** 3 - q * q + 2 / 3), c / 6 * (2 - q) ** 3)
            s = torch.where(q <= 1, c * q * (1.5 * q - 2), -0.5 * c * (2 - q) ** 2) / rn / h
        return r, rn, W, s[:, None] * r

    def total(self, I, a):
        return torch.zeros((self.n,) + a.shape[1:], dtype=a.dtype, device=a.device).index_add(0, I, a)

    def corrections(self):
        I, J = self.I, self.J
        fl = self.flow[J]
        S = self.total(I[fl], (self.mV[J] * self.W)[fl])
        self.f = torch.where(S != 0, 1 / torch.where(S != 0, S, torch.ones_like(S)), torch.ones_like(S))
        self.L = None
        if self.k.kernel_corr:
            D = self.D
            e = fl & self.flow[I]
            A = self.total(I[e], (self.mV[J][:, None, None] * -self.r[:, :D, None] * self.dW[:, None, :D])[e])
            ok = self.flow & (torch.linalg.det(A).abs() > EPS)
            eye = torch.eye(D, dtype=A.dtype, device=A.device)
            self.L = torch.linalg.inv(torch.where(ok[:, None, None], A, eye))

    def corrected(self, e):
        if self.L is None:
            return self.dW[e]
        out = torch.zeros_like(self.dW[e])
        out[:, :self.D] = (self.L[self.I[e]] @ self.dW[e][:, :self.D, None])[:, :, 0]
        return out

    def boundary_values(self):
        k = self.k
        e = self.bdy[self.I] & self.flow[self.J]
        I, J = self.I[e], self.J[e]
        w = self.mV[J] * self.W[e]
        f, b = self.f, self.bdy
        vt = 2 * self.v - self.total(I, w[:, None] * self.vt[J]) * f[:, None]
        self.vt = torch.where(b[:, None], vt, self.vt)
        rj = self.rt[J]
        if self.method == WC:
            p = (self.total(I, w * (self.p[J] + rj * self.grav[1] * self.r[e, 1])) * f).clamp(min=0)
            self.p = torch.where(b, p, self.p)
            rt = torch.full_like(self.rt, k.density0)
        else:
            m = self.st[J] + torch.diag_embed(rj[:, None] * self.grav * self.r[e])
            self.st = torch.where(b[:, None, None], self.total(I, w[:, None, None] * m) * f[:, None, None], self.st)
            rt = (self.total(I, w * rj) * f).clamp(min=k.density0) if self.method == MUI else \
                torch.full_like(self.rt, k.density0)
        self.rt = torch.where(b, rt, self.rt)

    def repulsion(self, e):
        k = self.k
        rep = e & (self.mt[self.J] == -2)
        if k.boundary not in (3, 4) or not bool(rep.any()):
            return 0.0
        rn = self.rn[rep]
        chi = torch.where(rn < k.particle_diameter, 1 - rn / k.particle_diameter, torch.zeros_like(rn))
        gm = rn / (0.75 * self.h)
        f = torch.where(gm <= 2 / 3, torch.full_like(gm, 2 / 3), torch.where(gm <= 1, 2 * gm - 1.5 * gm * gm,
                        torch.where(gm < 2, 0.5 * (2 - gm) ** 2, torch.zeros_like(gm))))
        return self.total(self.I[rep], (self.rep_fac * chi * f / rn ** 2)[:, None] * self.r[rep])

    def gradient(self):
        """Velocity gradient and continuity of the flow particles (granular solvers)."""
        e = self.flow[self.I]
        I, J = self.I[e], self.J[e]
        kc, mV = self.corrected(e), self.mV[J]
        u = self.vt[J] - self.vt[I]
        vg = self.total(I, mV[:, None, None] * u[:, :, None] * kc[:, None, :])
        return e, kc, vg, -self.total(I, mV * (u * kc).sum(1)) * self.rt

    def stress_divergence(self, e, kc):
        I, J = self.I[e], self.J[e]
        m = self.st[J] / self.rt[J][:, None, None] ** 2 + self.st[I] / self.rt[I][:, None, None] ** 2
        dv = self.total(I, (self.mV[J] * self.rt[J])[:, None] * (m @ kc[:, :, None])[:, :, 0])
        dv[:, self.D:] = 0
        damp = -self.k.damping_eps * torch.sqrt(self.k.E / (self.rt * self.h ** 2))
        return dv, damp[:, None] * self.vt

    def one_step(self):
        k = self.k
        I3 = torch.eye(3, dtype=torch.float64, device=self.dev)
        if self.method == WC:
            ratio = torch.where(self.flow, self.rt / k.density0, torch.ones_like(self.rt))
            self.p = torch.where(self.flow, (self.B * (ratio ** k.exponent - 1)).clamp(min=0), self.p)
            self.boundary_values()
            e = self.flow[self.I]
            I, J = self.I[e], self.J[e]
            u, r, kd, mV = self.vt[I] - self.vt[J], self.r[e], self.dW[e], self.mV[J]
            self.dd = self.total(I, mV * (u * self.corrected(e)).sum(1)) * self.rt
            rho0 = k.density0
            mn = (u * r).sum(1).clamp(max=0)
            cv = self.visc * mV * mn / (self.rn[e] ** 2 + 0.01 * self.h ** 2)
            cv = torch.where(self.flow[J], cv, cv * rho0 / self.rt[I])
            cp = -rho0 * mV * (self.p[I] / self.rt[I] ** 2 + self.p[J] / self.rt[J] ** 2)
            self.dv = self.total(I, (cv + cp)[:, None] * kd) + self.repulsion(e) + self.grav
            return
        if self.method == MUI:
            e, kc, vg, self.dd = self.gradient()
            p = (24.0 ** 2 * (self.rho - k.density0)).clamp(min=0)
            self.p = torch.where(self.flow, p, self.p)
            er = 0.5 * (vg + vg.transpose(1, 2))
            sc = (k.cohesion + p * self.mu) / ((0.5 * (er * er).sum((1, 2))).sqrt() + EPS)
            st = sc[:, None, None] * er - p[:, None, None] * I3
            self.st = torch.where(self.flow[:, None, None], st, self.st)
            ed = er - er.diagonal(dim1=1, dim2=2).sum(1)[:, None, None] / 3 * I3
            self.deq = ((ed * ed).sum((1, 2)) * 2 / 3).sqrt()
            self.boundary_values()
            dv, fd = self.stress_divergence(e, kc)
            self.dv = dv + self.repulsion(e) + self.grav + fd
            return
        self.st = torch.where(self.flow[:, None, None], self.adapted(self.st)[0], self.st)
        self.boundary_values()
        e, kc, vg, self.dd = self.gradient()
        dv, fd = self.stress_divergence(e, kc)
        self.dv = dv + self.grav + fd
        s, I1, sJ2, f = self.invariants(self.st)
        er, wr = 0.5 * (vg + vg.transpose(1, 2)), 0.5 * (vg - vg.transpose(1, 2))
        J = self.st @ wr.transpose(1, 2) + (wr @ self.st)
        tr = er.diagonal(dim1=1, dim2=2).sum(1)
        ed = er - tr[:, None, None] / 3 * I3
        pl = (f >= -EPS_F) & (sJ2 > EPS)
        safe = torch.where(pl, sJ2, torch.ones_like(sJ2))
        lam = (3 * self.alpha * self.Km * tr + self.Gm / safe * (s * er).sum((1, 2))) / \
            (27 * self.alpha * self.Km * self.sd + self.Gm)
        tg = lam[:, None, None] * (9 * self.Km * self.sd * I3 + (self.Gm / safe)[:, None, None] * s)
        self.ds = J + 2 * self.Gm * ed + (self.Km * tr)[:, None, None] * I3 - \
            torch.where(pl[:, None, None], tg, torch.zeros_like(tg))
        self.deq = ((ed * ed).sum((1, 2)) * 2 / 3).sqrt()
        gd = sJ2 + 3 * I1 * self.sd
        big = self.ds.abs() > EPS
        ep = lam[:, None, None] * torch.where(big, gd[:, None, None] / torch.where(big, self.ds,
                                              torch.ones_like(self.ds)), torch.zeros_like(self.ds))
        epd = ep - ep.diagonal(dim1=1, dim2=2).sum(1)[:, None, None] / 3 * I3
        self.deqp = torch.where(pl, ((epd * epd).sum((1, 2)) * 2 / 3).sqrt(), torch.zeros_like(sJ2))

    def invariants(self, st):
        I3 = torch.eye(3, dtype=torch.float64, device=self.dev)
        I1 = st.diagonal(dim1=1, dim2=2).sum(1)
        s = st - I1[:, None, None] / 3 * I3
        sJ2 = (0.5 * (s * s).sum((1, 2))).sqrt()
        return s, I1, sJ2, sJ2 + self.alpha * I1 - self.kc

    def adapted(self, st):
        I3 = torch.eye(3, dtype=torch.float64, device=self.dev)
        s, I1, sJ2, f = self.invariants(st)
        out = f > EPS_F
        cut = out & (f > sJ2)
        st = torch.where(cut[:, None, None], st - ((I1 - self.kc / self.alpha) / 3)[:, None, None] * I3, st)
        s, I1, sJ2, _ = self.invariants(st)
        r = (-I1 * self.alpha + self.kc) / torch.where(sJ2 > 0, sJ2, torch.ones_like(sJ2))
        new = r[:, None, None] * s + I1[:, None, None] / 3 * I3
        return torch.where(out[:, None, None], new, st), f

    def full(self, a, b):
        """Flow particles take a, the others keep b."""
        return torch.where(self.flow.reshape((-1,) + (1,) * (a.dim() - 1)), a, b)

    def volume(self, rho):
        self.mV = self.full(self.mass / torch.where(self.flow, rho, torch.ones_like(rho)), self.mV)

    def step(self):
        k, dt = self.k, self.k.dt
        f, _ = self._cells(self.x)
        self.order = self.order[torch.argsort(f[self.order], stable=True)]
        self.I, self.J = self.pairs(self.x)
        self.r, self.rn, self.W, self.dW = self.geometry(self.x, self.I, self.J)
        self.corrections()
        self.rt, self.vt = self.full(self.rho, self.rt), self.full(self.v, self.vt)
        if self.method != WC:
            self.st = self.full(self.sig, self.st)
        dp = self.method == DP
        if self.ti == RK4:
            acc = [0.0, 0.0, 0.0]
            for q, m in enumerate((1, 2, 2, 1)):
                self.one_step()
                acc = [acc[0] + m * self.dd, acc[1] + m * self.dv, acc[2] + (m * self.ds if dp else 0.0)]
                if q < 3:
                    self.rt = self.full(self.rho + 0.5 * dt * self.dd, self.rt)
                    self.volume(self.rt)
                    self.vt = self.full(self.v + 0.5 * dt * self.dv, self.vt)
                    if dp:
                        self.st = self.full(self.sig + 0.5 * dt * self.ds, self.st)
            dd, dv, ds, w = acc[0], acc[1], acc[2], dt / 6
        else:
            self.one_step()
            if self.ti == LF:
                self.rt = self.full(self.rt + 0.5 * dt * self.dd, self.rt)
                self.volume(self.rt)
                self.vt = self.full(self.vt + 0.5 * dt * self.dv, self.vt)
                if dp:
                    self.st = self.full(self.st + 0.5 * dt * self.ds, self.st)
                self.one_step()
            dd, dv, ds, w = self.dd, self.dv, self.ds if dp else 0.0, dt
        self.rho = self.full(self.rho + w * dd, self.rho)
        self.volume(self.rho)
        self.v = self.full(self.v + w * dv, self.v)
        if dp:
            self.sig = self.full(self.sig + w * ds, self.sig)
        move = self.v
        if k.xsph:
            e = self.mt[self.I] == self.mt[self.J]
            I, J = self.I[e], self.J[e]
            move = self.v + 0.5 * self.total(I, (self.mV[J] * self.W[e])[:, None] * (self.v[J] - self.v[I]))
        self.x = self.full(self.x + dt * move, self.x)
        self.rho = self.full(self.rho.clamp(min=k.density0), self.rho)
        self.volume(self.rho)
        if self.method == MUI:
            self.eq = self.full(self.eq + dt * self.deq, self.eq)
            I, J = self.pairs(self.x, self.flow)
            e = self.flow[J]
            I, J = I[e], J[e]
            W = self.geometry(self.x, I, J)[2]
            sm = self.total(I, (self.mV[J] * W)[:, None, None] * self.st[J]) * self.f[:, None, None]
            self.sig = self.full(sm, self.sig)
        elif dp:
            self.sig = self.full(self.adapted(self.sig)[0], self.sig)
            self.eq = self.full(self.eq + dt * self.deq, self.eq)
            self.eqp = self.full(self.eqp + dt * self.deqp, self.eqp)


def exact(case, seed):
    """The pass in 64 bits, by plain torch; None where that takes too long (the full-size 3D
    scenes and large ensembles)."""
    if case["kind"] == "ensemble":
        if case["scenes"] > 16:
            return None
        parts = []
        for d in _ensemble_dicts(case, seed):
            e = _Exact(d)
            for _ in range(case["steps"]):
                e.step()
            parts.append((e.v, e.rho))
        return {"x": None, "v": torch.cat([a for a, _ in parts]), "density": torch.cat([b for _, b in parts])}
    flow, bdy = _counts(case)
    per = (1 if case["dim"] == 2 else 5) * case["steps"] * {SE: 1, LF: 2, RK4: 4}[case["ti"]]
    if (flow + bdy) * per > 6_000_000:
        return None
    d = _scene_dict(case, seed)
    if case["kind"] == "rollout":
        d["Configuration"]["neighbourSkin"] = 0.0
        e = _Exact(d)
        par = torch.tensor([e.k.stiffness, e.k.viscosity], dtype=torch.float64, device=e.dev, requires_grad=True)
        e.B, e.visc = par[0], 2 * (e.D + 2) * par[1]
        for _ in range(case["steps"]):
            e.step()
        x = e.x[e.flow][:, :2]
        loss = _distance(x, _rollout_target(case))
        loss.backward()
        return {"x": x.detach(), "loss": loss.detach(), "grad": par.grad}
    cfg = SimConfiger(config=d)
    sc = build_scene(cfg, scene_geometry(cfg))
    e = _Exact(d, _velocity(case, np.asarray(sc.x), np.asarray(sc.mat_type) > 0, seed))
    for _ in range(case["steps"]):
        e.step()
    out = {"x": e.x, "v": e.v, "density": e.rho, "stress": e.sig, "strain_equ": e.eq, "strain_equ_p": e.eqp}
    out = {k: out[k] for k in _state_names(case)}
    if case["precision"] == "fp64":
        out = {k: a[e.order] for k, a in out.items()}
        out["pressure"] = e.p[e.order]
        out["id0"] = None
    return out
