"""Performance cases of the ocean step and of what runs around it.

Every case goes through the package's public entry points, with the states,
forcing and handles a model run holds: the step in its forms (the drop-in call
``step(state)``, several steps per call, host arrays), an ensemble, the
learned closure's inference and training, and the history output of a state.
``exact`` gives the same results in float64 torch arithmetic of its own.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

import zhenmode_b200
from zhenmode_b200 import workloads
from zhenmode_b200.closure import ClosureMLP, init_params
from zhenmode_b200.ensemble import Ensemble

G, RHO0, ALPHA, BETA, CP = 9.81, 1025.0, 2.0e-4, 7.6e-4, 3992.0
R_EARTH, OMEGA = 6371.0e3, 7.2921e-5
DEV = "cuda"


# --------------------------------------------------------------- the cases
def listed():
    """The cases with names; each comment says what they stand for."""
    return [
        # the synthetic smoke preset, one call per step as the run loop makes it: the smallest grid, all latency
        dict(name="smoke_step_90x45x15", kind="step", form="smoke", nx=90, ny=45, nz=15, steps=1),
        # a 2 degree spin-up on device states, several steps per call
        dict(name="plain_advance8_180x90x50", kind="step", form="plain", nx=180, ny=90, nz=50, steps=8),
        # the 0.5 degree production grid, the run loop's own call
        dict(name="plain_step_720x360x50", kind="step", form="plain", nx=720, ny=360, nz=50, steps=1),
        # sponge, bulk and SSS restoring, coastal coefficients, donor-cell faces, conservative vertical
        # diffusion, on a grid that divides by no tile
        dict(name="options_step_450x219x37", kind="step", form="options", nx=450, ny=219, nz=37, steps=1),
        # the 0.45 degree precision form: implicit vertical solve, seasonal forcing blended before the step
        dict(name="precision_step_800x400x50", kind="step", form="precision", nx=800, ny=400, nz=50, steps=1),
        # the 0.5 degree preset's column projection, on a 1 degree grid
        dict(name="projected_step_360x180x50", kind="step", form="projected", nx=360, ny=180, nz=50, steps=1),
        # the step with the learned vertical-mixing closure on
        dict(name="learned_step_360x180x50", kind="step", form="learned", nx=360, ny=180, nz=50, steps=1),
        # a caller whose states live in NumPy arrays: the whole call with its transfers
        dict(name="host_step_360x180x30", kind="host", form="plain", nx=360, ny=180, nz=30, steps=1),
        # perturbed members on two grid sizes, one ensemble step with the states loaded and read
        dict(name="ensemble_6x180x90x20_2x360x180x30", kind="ensemble", nx=180, ny=90, nz=20, small=6, large=2),
        # history output of a 0.5 degree state: density, pressure, w, the tracer terms and the budget
        dict(name="history_720x360x50", kind="history", form="plain", nx=720, ny=360, nz=50),
        # the closure network on every column of the 0.5 degree grid
        dict(name="closure_infer_259200", kind="infer", rows=259200),
        # one Adam step of the closure's training at its default batch
        dict(name="closure_train_8192", kind="train", rows=8192),
    ]


def _five_smooth(n):
    for f in (2, 3, 5):
        while n % f == 0:
            n //= f
    return n == 1


# widths the longitude filter accepts, between the smoke and the 0.45 degree grid
_WIDTHS = [n for n in range(90, 801) if _five_smooth(n)]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: kinds as often as they are listed, sizes over the whole range."""
    kind = rng.choice(["smoke", "plain", "plain", "options", "precision", "projected", "learned", "host", "ensemble",
                       "history", "infer", "train"])
    if kind == "infer":
        return dict(kind="infer", rows=_log_int(rng, 4000, 300000))
    if kind == "train":
        return dict(kind="train", rows=_log_int(rng, 500, 12000))
    widest = dict(smoke=400, projected=360, learned=640, host=360, ensemble=180).get(kind, 800)
    target = math.exp(rng.uniform(math.log(90), math.log(widest)))
    nx = min(_WIDTHS, key=lambda n: abs(n - target))
    ny = max(45, int(nx * rng.uniform(0.46, 0.5)))
    nz = rng.randint(15, 30 if kind in ("host", "ensemble") else 50)
    if kind == "ensemble":
        return dict(kind="ensemble", nx=nx, ny=ny, nz=nz, small=rng.randint(2, 6), large=rng.randint(0, 2))
    if kind in ("history", "host"):
        return dict(kind=kind, form="plain", nx=nx, ny=ny, nz=nz, **({"steps": 1} if kind == "host" else {}))
    # several steps per call where they stay below the cost of one step of the largest grid
    most = 1 if kind in ("projected", "precision") else max(1, int(5.0 / (0.5 + nx * ny * nz / 3.0e6)))
    return dict(kind="step", form=kind, nx=nx, ny=ny, nz=nz, steps=min(most, rng.choice([1, 1, 2, 4, 8])))


# ------------------------------------------------------- grids, options, states
def _config(form, nx, ny, nz, gen):
    """(grid, physics, dt, options, initial T and S) of a step form."""
    grid = workloads.build_grid(nx, ny, nz)
    wl = workloads.WORKLOADS["smoke" if form == "smoke" else "precision" if form == "precision" else "plain"]
    dev = gen.device
    T0, S0 = _thermocline(grid, gen)
    kw = dict(wl.options, forcing=workloads.wind_forcing(grid), dt_bt=wl.dt_bt, dtype="float32")
    physics = wl.physics
    sst = T0[:, :, 0].double().cpu().numpy()
    wet = np.asarray(grid.wet_mask)
    if form != "smoke":
        kw.update(coastal_restore_mask=wet, coastal_restore_days=wl.restore_days, coastal_restore_T=sst)
    if form == "precision":
        kw.update(vertical_diffusion="implicit")
    if form == "projected":
        kw.update(project_adv_vel=True)
    if form == "options":
        coast = wet * np.clip(np.abs(_smooth2(nx, ny, gen, dev).double().cpu().numpy()), 0.0, 1.0)
        kw.update(fct_adv=False, monotone_adv=True, conservative_kv=True, T_atm=sst - 1.0, lambda_bulk=30.0,
                  S_ref_surf=np.full((nx, ny), 35.0), sss_restore_days=60.0, coastal_kappa_h_mask=coast,
                  coastal_kappa_h=200.0, coastal_kappa_v_mask=coast, coastal_kappa_v=1.0e-4, sponge_days=5.0,
                  sponge_cells=max(4, ny // 5), T_init=T0.cpu().numpy(), S_init=S0.cpu().numpy())
    return grid, physics, wl.dt, kw, T0, S0


def _smooth2(nx, ny, gen, dev, modes=12):
    """A smooth periodic-in-longitude random field (nx, ny) of unit variance."""
    lon = torch.arange(nx, device=dev, dtype=torch.float32) * (2 * math.pi / nx)
    lat = torch.linspace(0, math.pi, ny, device=dev)
    out = torch.zeros((nx, ny), device=dev)
    for _ in range(modes):
        r = torch.rand(4, generator=gen, device=dev)
        kx = torch.floor(r[0] * 9)
        out += torch.cos(kx * lon + 6.2832 * r[1])[:, None] * torch.cos(r[2] * 9 * lat + 6.2832 * r[3])[None, :]
    return out / math.sqrt(modes / 4)


def _thermocline(grid, gen):
    """Initial T and S: the workloads' thermocline and noise, from this generator."""
    nx, ny, nz, dev = grid.nx, grid.ny, grid.nz, gen.device
    prof = torch.exp(torch.as_tensor(grid.z, dtype=torch.float32, device=dev) / 500.0)
    cosl = torch.as_tensor(grid.cos_lat, dtype=torch.float32, device=dev)
    T = 2.0 + (26.0 * cosl[None, :] + 0.2 * _smooth2(nx, ny, gen, dev))[:, :, None] * prof
    S = 35.0 + (0.1 * torch.randn((nx, ny, nz), generator=gen, device=dev)).clamp_(-0.5, 0.5)
    return T, S


def _state(grid, physics, T, S, gen, moving=True):
    """A state in motion on the wet points; land and ghost points as init_state leaves them."""
    nx, ny, nz, dev = grid.nx, grid.ny, grid.nz, gen.device
    wet = torch.as_tensor(grid.wet_mask_3d, dtype=torch.float32, device=dev)
    prof = torch.exp(torch.as_tensor(grid.z, dtype=torch.float32, device=dev) / 1000.0)
    amp = 0.1 if moving else 0.0
    u = (amp * _smooth2(nx, ny, gen, dev))[:, :, None] * prof * wet
    v = (0.5 * amp * _smooth2(nx, ny, gen, dev))[:, :, None] * prof * wet
    v[:, 0] = 0.0
    v[:, -1] = 0.0
    T = T * wet + (1.0 - wet) * physics.T_ref
    S = S * wet + (1.0 - wet) * physics.S_ref
    eta = 0.1 * _smooth2(nx, ny, gen, dev) * torch.as_tensor(grid.wet_mask, dtype=torch.float32, device=dev)
    return [t.contiguous() for t in (u, v, T, S, eta)]


def _months(grid, gen):
    """(12, nx, ny) monthly wind stress and heat flux."""
    lat = torch.as_tensor(np.radians(grid.lat), dtype=torch.float32, device=gen.device)
    base = (0.1 * torch.sin(2 * lat) * torch.cos(lat))[None, :] * torch.ones((grid.nx, 1), device=gen.device)
    s = torch.cos(torch.arange(12, device=gen.device) * (2 * math.pi / 12))
    noise = torch.stack([_smooth2(grid.nx, grid.ny, gen, gen.device, 4) for _ in range(2)])
    tx = base[None] * (1 + 0.3 * s)[:, None, None]
    ty = 0.02 * noise[0][None] * (1 + s)[:, None, None]
    q = 100.0 * s[:, None, None] * torch.sign(lat)[None, None, :] + 10.0 * noise[1][None]
    return [t.contiguous() for t in (tx, ty, q)]


def _closure_rows(n, gen):
    """Closure feature rows (T, S, u, v, N^2, forcing), targets and mask of a snapshot's wet columns."""
    dev = gen.device
    rn = lambda *s: torch.randn(s, generator=gen, device=dev)  # noqa: E731
    lev = torch.arange(50, device=dev, dtype=torch.float32)
    depth = (torch.rand((n, 1), generator=gen, device=dev) * 45 + 5).floor()
    wet = (lev[None, :] < depth).float()
    X = torch.zeros((n, 256), device=dev)
    X[:, 0:50] = (torch.exp(-lev / 12)[None, :] * (1 + 0.4 * rn(n, 1)) - 0.8 + 0.01 * rn(n, 50)) * wet
    X[:, 50:100] = 0.1 * rn(n, 50) * wet
    X[:, 100:150] = 0.2 * rn(n, 1) * torch.exp(-lev / 20) * wet
    X[:, 150:200] = 0.1 * rn(n, 1) * torch.exp(-lev / 20) * wet
    M = torch.zeros((n, 64), device=dev)
    M[:, :49] = wet[:, 1:]
    n2 = 2.0 + 0.7 * rn(n, 49)
    X[:, 200:249] = n2 * M[:, :49]
    X[:, 250] = rn(n).abs()
    X[:, 251] = rn(n)
    T = torch.zeros((n, 64), device=dev)
    T[:, :49] = torch.where(n2 > 0.5, -6.0, -2.0) * M[:, :49]
    return X, T, M


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000003 * seed + 17)


def _members(case):
    sizes = [(case["nx"], case["ny"], case["nz"])] * case["small"] + [(360, 180, 30)] * case["large"]
    return list(enumerate(sizes))


# ------------------------------------------------------------------ prepare, run
def prepare(case, seed):
    """What a user's program holds before the call."""
    kind, gen = case["kind"], _gen(seed)
    if kind == "infer":
        return dict(kind=kind, net=ClosureMLP(seed=seed), X=_closure_rows(case["rows"], gen)[0])
    if kind == "train":
        X, T, M = _closure_rows(case["rows"], gen)
        net = ClosureMLP(seed=seed)
        # Adam's moments as they are some steps into the training
        net.m.copy_(1e-3 * torch.randn(net.m.shape, generator=gen, device=DEV))
        net.v.copy_(1e-5 * (0.1 + torch.rand(net.v.shape, generator=gen, device=DEV)))
        net.step_count = 100
        return dict(kind=kind, net=net, rows=(X, T, M))
    if kind == "ensemble":
        steps, states = [], []
        for q, (nx, ny, nz) in _members(case):
            mgen = _gen(seed + 101 * q)
            grid, physics, dt, kw, T, S = _config("plain", nx, ny, nz, mgen)
            steps.append(zhenmode_b200.make_solver_global(grid, physics, dt, **kw)[0])
            states.append(zhenmode_b200.JaxStateG(*_state(grid, physics, T, S, mgen), 0.0))
        return dict(kind=kind, ens=Ensemble(steps), states=states)
    form = case["form"]
    grid, physics, dt, kw, T, S = _config(form, case["nx"], case["ny"], case["nz"], gen)
    made = zhenmode_b200.make_solver_global(grid, physics, dt, return_params=kind == "history", **kw)
    fields = _state(grid, physics, T, S, gen, moving=form != "smoke")
    if kind == "host":
        fields = [t.cpu().numpy() for t in fields]
    s = dict(kind=kind, form=form, step=made[0], state=zhenmode_b200.JaxStateG(*fields, 0.0), steps=case.get("steps", 1))
    if kind == "history":
        s.update(diagnostics=made[2], terms=made[4])
    if form == "learned":
        made[0].set_closure(ClosureMLP(seed=seed))
    if form == "precision":
        s.update(months=_months(grid, gen), day=28.0 + (seed % 5))
    return s


def _named(state):
    return {k: getattr(state, k) for k in ("u", "v", "T", "S", "eta")}


def run(s):
    """One pass through the public entry points."""
    kind = s["kind"]
    if kind == "infer":
        return s["net"].forward_bf16(s["X"])
    if kind == "train":
        net = s["net"]
        net.train_step(*s["rows"])
        return dict(params=net.params, m=net.m, v=net.v)
    if kind == "ensemble":
        s["ens"].load(s["states"])
        s["ens"].advance(1)
        return [_named(st) for st in s["ens"].store()]
    step, state = s["step"], s["state"]
    if kind == "history":
        rho, pressure, w = s["diagnostics"](state)
        budget = step.budget_diagnostics(state).as_dict()
        return dict(rho=rho, pressure=pressure, w=w, terms=s["terms"](state), budget=budget)
    if s["form"] == "precision":
        step.set_forcing_seasonal(*s["months"], day=s["day"])
    return _named(step(state) if s["steps"] == 1 else step.advance(state, s["steps"]))


# ------------------------------------------------------------------------- work
def _step_work(nx, ny, nz, form, steps):
    n3, n2 = nx * ny * nz, nx * ny
    n_bt, n_nu, na = (2, 0, 1) if form == "smoke" else (27, 27, 2) if form == "precision" else (24, 24, 2)
    # flops a point: the nu_h subcycles of u and v, diffusion, advection, pressure; two FFTs of a complex line
    per = 2 * n_nu * 2 * 13 + 2 * 2 * 2 * 2 * 15 + 2 * na * 2 * 60 + 3 * 40 + 60 + 10 * math.log2(nx)
    if form == "learned":
        per += 2 * 148032 / nz
    flops = steps * (n3 * per + n2 * n_bt * 80)
    if form == "projected":
        flops += steps * n2 * 450 * 45
    months = 3 * n2 if form == "precision" else 0
    return 4.0 * (2 * (4 * n3 + n2) + months), float(flops)


def work(case):
    """Inputs read once, outputs written once; the arithmetic of one pass."""
    kind = case["kind"]
    if kind == "infer":
        n = case["rows"]
        return dict(bytes=4.0 * n * (256 + 64) + 2 * 148032, flops=2.0 * 147456 * n)
    if kind == "train":
        n = case["rows"]
        return dict(bytes=4.0 * (n * (256 + 2 * 64) + 6 * 148032), flops=2.0 * (3 * 147456 - 65536) * n)
    if kind == "ensemble":
        w = [_step_work(*size, "plain", 1) for _, size in _members(case)]
        return dict(bytes=sum(x[0] for x in w), flops=sum(x[1] for x in w))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind == "history":
        return dict(bytes=4.0 * nx * ny * (13 * nz + 1), flops=150.0 * nx * ny * nz)
    b, f = _step_work(nx, ny, nz, case["form"], case["steps"])
    return dict(bytes=b, flops=f)


# ------------------------------------------------ float64 restatement of the results
# Layout (nx, ny, nz), longitude periodic on the first axis, closed latitude walls.
def _e(a):
    return torch.roll(a, -1, 0)


def _w(a):
    return torch.roll(a, 1, 0)


def _n(a):
    return torch.cat((a[:, 1:], a[:, -1:]), 1)


def _s(a):
    return torch.cat((a[:, :1], a[:, :-1]), 1)


def _zero_row(a, j):
    a = a.clone()
    a[:, j] = 0.0
    return a


class _Exact:
    """The step's operators for one configuration, in float64."""

    def __init__(self, grid, physics, dt, kw, form):
        t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEV)  # noqa: E731
        self.nx, self.ny, self.nz, self.dt, self.form, self.ph = grid.nx, grid.ny, grid.nz, float(dt), form, physics
        self.wm, self.w2 = t(grid.wet_mask_3d), t(grid.wet_mask)
        self.dx = t(grid.dx_2d)
        self.rdx, self.dy, self.rdy = (1.0 / self.dx)[:, :, None], float(grid.dy), 1.0 / float(grid.dy)
        c = t(grid.cos_lat)
        self.c = c[None, :, None]
        self.cf = 0.5 * (c + torch.roll(c, -1))[None, :, None]
        self.cb = 0.5 * (c + torch.roll(c, 1))[None, :, None]
        self.f = t(grid.f)[:, :, None]
        self.tanr = ((self.f[0, :, 0] / (2 * OMEGA)) / c / R_EARTH)[None, :, None]
        z = t(grid.z)
        self.z, self.gap = z, (z[1:] - z[:-1]).abs()
        g = self.gap
        self.dzn = torch.cat((g[:1], 0.5 * (g[:-1] + g[1:]), g[-1:]))
        self.H = float(g.sum())
        lev = torch.arange(self.nz, device=DEV)
        self.kb = ((self.wm > 0.5) * lev).amax(-1)
        self.fill = torch.minimum(lev[None, None, :].expand(self.wm.shape), self.kb[:, :, None])
        self.wif = self.wm[..., :-1] * self.wm[..., 1:]
        opt = kw.get
        zero2 = torch.zeros((self.nx, self.ny), dtype=torch.float64, device=DEV)
        self.tau_x, self.tau_y, self.q = (t(a) for a in kw["forcing"])
        self.lim = 2 if opt("fct_adv") else 1 if opt("monotone_adv") else 0
        self.local, self.cons = bool(opt("localize_conv")), bool(opt("conservative_kv"))
        self.implicit, self.project = opt("vertical_diffusion") == "implicit", bool(opt("project_adv_vel"))
        field = lambda m, k: t(kw[m]) * kw[k] if opt(m) is not None else zero2  # noqa: E731
        self.kh = physics.kappa_h + field("coastal_kappa_h_mask", "coastal_kappa_h")[:, :, None]
        self.kv = physics.kappa_v + field("coastal_kappa_v_mask", "coastal_kappa_v")[:, :, None]
        self.lam, self.t_atm = opt("lambda_bulk", 0.0), t(kw["T_atm"]) if opt("T_atm") is not None else zero2
        self.rs = 1.0 / (kw["sss_restore_days"] * 86400.0) if opt("sss_restore_days") else 0.0
        self.s_ref = t(kw["S_ref_surf"]) if opt("S_ref_surf") is not None else zero2
        days = opt("coastal_restore_days", 0.0)
        self.rc = t(kw["coastal_restore_mask"]) / (days * 86400.0) if days else zero2
        self.rt = t(kw["coastal_restore_T"]) if days else zero2
        self.rate = None
        if opt("sponge_days"):
            edge = np.minimum(np.arange(self.ny), self.ny - 1 - np.arange(self.ny))
            n = kw["sponge_cells"]
            tap = np.where(edge < n, 0.5 * (1 + np.cos(np.pi * edge / n)), 0.0) / (kw["sponge_days"] * 86400.0)
            self.rate = t(tap)[None, :].expand(self.nx, self.ny)
            self.Tc = t(kw["T_init"]) * self.wm + (1 - self.wm) * physics.T_ref
            self.Sc = t(kw["S_init"]) * self.wm + (1 - self.wm) * physics.S_ref
        rows, tap = opt("polar_cap_rows", 2), opt("polar_cap_taper", 3)
        self.nb = rows + tap if rows > 0 else 0
        ramp = np.cos(np.linspace(0, np.pi / 2, tap + 2)[1:-1]) ** 2
        self.wts = t(np.concatenate((np.ones(rows), ramp)))
        k = np.abs(np.fft.fftfreq(self.nx) * self.nx)
        self.keep = t(k <= max(1, int((self.nx // 2) * 2 / 3)))[:, None, None]
        self.nsub = max(1, int(round(dt / kw["dt_bt"])))
        dzmin = float(g.min())
        self.nconv = max(1, math.ceil(physics.kappa_conv * dt / (0.4 * dzmin ** 2)))
        self.nadv = max(1, math.ceil(dt * 4.0e-3 / (0.5 * dzmin)))
        self.bot = torch.zeros(self.nz, dtype=torch.float64, device=DEV)
        self.bot[-1] = 1.0
        self.kappa = None  # the learned closure's diffusivity per interface

    # ---- column operators
    def ghost(self, a):
        return torch.gather(a, -1, self.fill)

    def d2z(self, a):
        a, g = self.ghost(a), self.gap
        hm, hp = g[:-1], g[1:]
        out = torch.empty_like(a)
        out[..., 1:-1] = (a[..., 2:] * hm + a[..., :-2] * hp - a[..., 1:-1] * (hm + hp)) / (hm * hp * (hm + hp) / 2)
        out[..., 0] = 2 * (a[..., 1] - a[..., 0]) / g[0] ** 2
        out[..., -1] = 2 * (a[..., -2] - a[..., -1]) / g[-1] ** 2
        return out

    def iface_div(self, F):
        F = torch.nn.functional.pad(F, (1, 1))
        return (F[..., :-1] - F[..., 1:]) / self.dzn

    def vdiff(self, a):
        if not self.cons:
            return self.kv * self.d2z(a)
        cf = self.ghost(a)
        return self.iface_div(-self.kv * (cf[..., 1:] - cf[..., :-1]) / self.gap * self.wif) * self.wm

    def solve(self, rhs, lo, up, n):
        """Tridiagonal (I + ...) solve of the levels below n per column: unit row sums, off-diagonals lo and up."""
        live = torch.arange(self.nz, device=DEV)[None, None, :] < n[:, :, None]
        lo, up = torch.where(live, lo, 0.0), torch.where(live, up, 0.0)
        dg = 1.0 - lo - up
        cp, y = torch.zeros_like(rhs), rhs.clone()
        cp[..., 0], y[..., 0] = up[..., 0] / dg[..., 0], rhs[..., 0] / dg[..., 0]
        for k in range(1, self.nz):
            den = dg[..., k] - lo[..., k] * cp[..., k - 1]
            cp[..., k] = up[..., k] / den
            y[..., k] = (rhs[..., k] - lo[..., k] * y[..., k - 1]) / den
        for k in range(self.nz - 2, -1, -1):
            y[..., k] -= cp[..., k] * y[..., k + 1]
        return torch.where(live, y, rhs)

    def implicit_solve(self, a, kappa, h):
        n = torch.where((self.kb > 0) & (self.wm[..., 0] > 0.5), self.kb + 1, 0)
        lo, up = torch.zeros_like(a), torch.zeros_like(a)
        below = torch.arange(self.nz, device=DEV)[None, None, :] < (n - 1)[:, :, None]
        if torch.is_tensor(kappa) and kappa.shape[-1] == self.nz - 1:  # flux form, a diffusivity per interface
            q = h * kappa / self.gap
            up[..., :-1] = -q / self.dzn[:-1]
            lo[..., 1:] = -q / self.dzn[1:]
        else:
            g = self.gap
            hm, hp = g[:-1], g[1:]
            den = hm * hp * (hm + hp) / 2
            lo[..., 1:-1] = -h * kappa * (hp / den)
            up[..., 1:-1] = -h * kappa * (hm / den)
            up[..., 0:1] = -h * kappa * 2 / g[0] ** 2
            lo[..., -1:] = -h * kappa * 2 / g[-1] ** 2
        return self.solve(a, lo, torch.where(below, up, 0.0), n)

    # ---- horizontal operators
    def lap(self, a):
        w, we, ww, wn, ws = self.wm, _e(self.wm), _w(self.wm), _n(self.wm), _s(self.wm)
        x = ((_e(a) - a) * w * we - (a - _w(a)) * w * ww) * self.rdx ** 2
        y = ((_n(a) - a) * w * wn - (a - _s(a)) * w * ws) * self.rdy ** 2
        return x + y - (_n(a) - _s(a)) * (0.5 * self.rdy) * self.tanr

    def hdiff(self, a, kap):
        w = self.wm
        fx = 0.5 * (kap + _e(kap)) * (_e(a) - a) * self.rdx * w * _e(w)
        fy = _zero_row(0.5 * (kap + _n(kap)) * (_n(a) - a) * self.rdy * w * _n(w) * self.cf, -1)
        return (fx - _w(fx)) * self.rdx + (fy - torch.roll(fy, 1, 1)) * self.rdy / self.c

    def grad(self, a, w):
        gx = 0.5 * self.rdx * ((_e(a) - a) * w * _e(w) + (a - _w(a)) * w * _w(w))
        up, dn = _zero_row(w * torch.roll(w, -1, 1), -1), _zero_row(w * torch.roll(w, 1, 1), 0)
        gy = 0.5 * self.rdy / self.c * ((torch.roll(a, -1, 1) - a) * up * self.cf
                                        + (a - torch.roll(a, 1, 1)) * dn * self.cb)
        return gx, gy

    def div(self, u, v, w):
        fx = 0.5 * (u + _e(u)) * w * _e(w)
        fy = _zero_row(0.5 * (v + _n(v)) * w * _n(w) * self.cf, -1)
        return (fx - _w(fx)) * self.rdx + (fy - torch.roll(fy, 1, 1)) * self.rdy / self.c

    def transport(self, u, v):
        d = self.div(u, v, self.wm) * self.dzn
        return torch.flip(torch.cumsum(torch.flip(d, (-1,)), -1), (-1,))

    def cap(self, a, w):
        if not self.nb:
            return a
        nb, out = self.nb, a.clone()
        wt = self.wts.reshape((1, nb) + (1,) * (a.dim() - 2))
        for sl, q in ((slice(0, nb), wt), (slice(self.ny - nb, self.ny), torch.flip(wt, (1,)))):
            m, s = w[:, sl], a[:, sl] * w[:, sl]
            mean = s.sum(0, keepdim=True) / m.sum(0, keepdim=True).clamp_min(1.0)
            out[:, sl] = q * (mean * m) + (1 - q) * s
        return out

    # ---- the parts of the step
    def linear(self, u0, v0, T0, S0):
        h, ph, wm = self.dt / 2, self.ph, self.wm
        u, v = u0, v0
        for _ in range(self.nsub):
            u, v = (a + ph.nu_h * self.lap(a) * (h / self.nsub) for a in (u, v))
        one = torch.ones((self.nx, self.ny, 1), dtype=torch.float64, device=DEV)
        out = []
        for a, a0, vel in ((u, u0, 1), (v, v0, 1), (T0, T0, 0), (S0, S0, 0)):
            if vel:
                a = a - ph.nu_bi * self.lap(self.lap(a0)) * h
            else:
                a = a + self.hdiff(a0, self.kh) * h - ph.kappa_bi * self.hdiff(self.hdiff(a0, one), one) * h
            if self.implicit or self.kappa is not None:
                k = ph.nu_v if vel else self.kappa if self.kappa is not None else self.kv
                a = self.implicit_solve(a, k, h)
            else:
                a = a + (ph.nu_v * self.d2z(a0) if vel else self.vdiff(a0)) * h
            out.append(a * wm + a0 * (1 - wm))
        u, v, T, S = out
        if self.rate is not None:
            d = torch.exp(-self.rate * h)[:, :, None]
            u, v, T, S = u * d, v * d, self.Tc + (T - self.Tc) * d, self.Sc + (S - self.Sc) * d
        ca, sa = torch.cos(self.f * h), torch.sin(self.f * h)
        return ca * u + sa * v, -sa * u + ca * v, T, S

    def face(self, a, vel, axis):
        nxt, prv = (_e, _w) if axis == 0 else (_n, _s)
        if self.lim == 0:
            return 0.5 * (a + nxt(a))
        if self.lim == 1:
            return torch.where(vel >= 0, a, nxt(a))
        lft, rgt = a - prv(a), nxt(a) - a
        s = 0.5 * (torch.sign(lft) + torch.sign(rgt)) * torch.minimum(lft.abs(), rgt.abs())
        s = s * self.wm * prv(self.wm) * nxt(self.wm)
        return torch.where(vel >= 0, a + 0.5 * s, nxt(a) - 0.5 * nxt(s))

    def advect(self, a, u, v, Fz):
        w = self.wm
        ux, vy = 0.5 * (u + _e(u)), 0.5 * (v + _n(v))
        fx = ux * self.face(a, ux, 0) * w * _e(w)
        fy = _zero_row(vy * self.face(a, vy, 1) * w * _n(w) * self.cf, -1)
        h = (fx - _w(fx)) * self.rdx + (fy - torch.roll(fy, 1, 1)) * self.rdy / self.c
        mid = Fz[..., 1:] * torch.where(Fz[..., 1:] > 0, a[..., :-1], self.ghost(a)[..., 1:]) * self.wif
        up = torch.cat((Fz[..., :1] * a[..., :1], mid), -1)
        dn = torch.nn.functional.pad(mid, (0, 1))
        return -(h + (dn - up) / self.dzn) * w

    def gates(self, T, S):
        rho = (-ALPHA * (T - self.ph.T_ref) + BETA * (S - self.ph.S_ref)) * self.wm
        u = (rho[..., :-1] > rho[..., 1:]) & (self.wif > 0.5)
        return u.double() if self.local else u.any(-1, keepdim=True) * self.wif

    def convect(self, a, gate, kappa):
        cf = self.ghost(a)
        return self.iface_div(-kappa * (cf[..., 1:] - cf[..., :-1]) / self.gap * gate) * self.wm

    def tracer_rate(self, u, v, T, S):
        """Residual rates of T and S: advection, convection and surface sources."""
        Fz = self.transport(u, v)
        gate = self.gates(T, S)
        out = []
        for a in (T, S):
            adv, b = 0.0, a
            for _ in range(self.nadv):
                r = self.advect(b, u, v, Fz)
                adv, b = adv + r / self.nadv, b + r * (self.dt / self.nadv)
            if self.ph.kappa_conv > 0 and self.kappa is None:
                b = a
                for _ in range(self.nconv):
                    r = self.convect(b, gate, self.ph.kappa_conv / self.nconv)
                    adv, b = adv + r / self.nconv, b + r * (self.dt / self.nconv)
            out.append(adv)
        rT, rS = out
        hf = self.wm[..., 0] / float(self.gap[0]) / (RHO0 * CP)
        sst = T[..., 0]
        rT[..., 0] += (self.q + self.lam * (self.t_atm - sst)) * hf + self.rc * (self.rt - sst)
        rS[..., 0] += self.rs * (self.s_ref - S[..., 0])
        return rT * self.wm, rS * self.wm

    def pressure_grad(self, T, S):
        """-grad(p)/rho0 of the baroclinic pressure and its wet-interface depth mean."""
        rho = RHO0 * (-ALPHA * (T - self.ph.T_ref) + BETA * (S - self.ph.S_ref)) * self.wm
        p = torch.nn.functional.pad(torch.cumsum(G * 0.5 * (rho[..., :-1] + rho[..., 1:]) * self.gap, -1), (1, 0))
        out = []
        for g in self.grad(p, self.wm):
            F = -(0.5 * (g[..., :-1] + g[..., 1:]) * self.wif * self.gap).sum(-1) / (RHO0 * self.H)
            out.append((-g / RHO0, F))
        return out

    def momentum_adv(self, u, v):
        wm = self.wm
        w = -self.transport(u, v) * wm
        out = []
        for a, tau in ((u, self.tau_x), (v, self.tau_y)):
            b, z = self.ghost(a), self.z
            dz = torch.empty_like(a)
            dz[..., 0] = (b[..., 1] - b[..., 0]) / (z[1] - z[0])
            dz[..., 1:-1] = (b[..., 2:] - b[..., :-2]) / (z[2:] - z[:-2])
            dz[..., -1] = (b[..., -1] - b[..., -2]) / (z[-1] - z[-2])
            gx = 0.5 * self.rdx * ((_e(a) - a) * wm * _e(wm) + (a - _w(a)) * wm * _w(wm))
            gy = 0.5 * self.rdy * ((_n(a) - a) * wm * _n(wm) + (a - _s(a)) * wm * _s(wm))
            r = -(u * gx + v * gy + w * dz)
            r = torch.fft.ifft(torch.fft.fft(r, dim=0) * self.keep, dim=0).real
            n1, s1 = _n(r), _s(r)
            r = (_s(s1) + 4 * s1 + 6 * r + 4 * n1 + _n(n1)) / 16
            r[..., 0] += tau / (RHO0 * float(self.gap[0]))
            out.append((r - (tau / (RHO0 * self.H))[:, :, None]) * wm)
        return out

    def column_project(self, u, v):
        dtg, area = self.dt * G, self.dx * self.dy * self.w2
        cdiv = lambda a, b: (self.div(a, b, self.wm) * self.dzn).sum(-1) * self.w2  # noqa: E731
        A = lambda psi: -cdiv(*self.grad(psi[:, :, None], self.wm)) * area  # noqa: E731
        eps = 32 * float(np.finfo(np.float32).eps)
        norm2 = lambda d: float((d ** 2 * self.dx * self.dy).sum())  # noqa: E731
        rhs = -(cdiv(u, v) / dtg) * area
        floor, first = eps * float(rhs.norm()), norm2(cdiv(u, v))
        for n in range(3):
            if n and not norm2(cdiv(u, v)) > eps ** 2 * first:
                break
            b = rhs if n == 0 else -(cdiv(u, v) / dtg) * area
            x, r = torch.zeros_like(b), b
            p, gam = r, float((r * r).sum())
            stop = max((eps * float(b.norm())) ** 2, floor ** 2 if n else 0.0)
            k = 0
            while gam > stop and k < 150:
                q = A(p)
                al = gam / float((p * q).sum())
                x, r = x + al * p, r - al * q
                new = float((r * r).sum())
                p, gam, k = r + (new / gam) * p, new, k + 1
            gx, gy = self.grad(x[:, :, None], self.wm)
            u, v = u - dtg * gx, v - dtg * gy
        return u, v

    def nonlinear(self, u, v, T, S):
        dt, wm = self.dt, self.wm
        Au, Av = self.momentum_adv(u, v)
        rT, rS = self.tracer_rate(u, v, T, S)
        Tp, Sp = T + rT * dt, S + rS * dt
        (gx, fx), (gy, fy) = self.pressure_grad(Tp, Sp)
        P1, Q1 = (gx - fx[:, :, None]) * wm, (gy - fy[:, :, None]) * wm
        up, vp = u + (Au + P1) * dt, v + (Av + Q1) * dt
        if self.project:
            up, vp = self.column_project(up, vp)
        rT2, rS2 = self.tracer_rate(up, vp, Tp, Sp)
        T, S = T + 0.5 * (rT + rT2) * dt, S + 0.5 * (rS + rS2) * dt
        (gx, fx), (gy, fy) = self.pressure_grad(T, S)
        P2, Q2 = (gx - fx[:, :, None]) * wm, (gy - fy[:, :, None]) * wm
        dec = torch.exp(-self.ph.r_bot * dt * self.bot * wm)
        return (u + (Au + 0.5 * (P1 + P2)) * dt) * dec, (v + (Av + 0.5 * (Q1 + Q2)) * dt) * dec, T, S

    def barotropic(self, eta, ub, vb, fx, fy):
        w, dtb = self.w2[:, :, None], self.dt / self.nsub
        fx, fy = fx + self.tau_x / (RHO0 * self.H), fy + self.tau_y / (RHO0 * self.H)
        fd, drag = self.f[..., 0] * dtb, 1.0 / (1.0 + self.ph.r_bot * dtb)
        area, w2 = self.dx * self.dy, self.w2
        for _ in range(self.nsub):
            d = self.div((ub * w2)[:, :, None], (vb * w2)[:, :, None], w)[..., 0]
            eta = (eta - dtb * self.H * d) * w2
            sp = 1.0
            if self.rate is not None:
                sp = torch.exp(-self.rate * dtb)
                new = eta * sp
                eta = new - (area * (new - eta)).sum() / (area * w2).sum() * w2
            eta = self.cap(eta, w2)
            gx, gy = self.grad(eta[:, :, None], w)
            us, vs = ub + dtb * (fx - G * gx[..., 0]), vb + dtb * (fy - G * gy[..., 0])
            q = drag / (1 + fd * fd) * w2 * sp
            ub, vb = self.cap((us + fd * vs) * q, w2), self.cap((vs - fd * us) * q, w2)
        return eta, ub, vb

    def step(self, u0, v0, T0, S0, eta):
        if self.form == "learned":
            self.kappa = self.closure(u0, v0, T0, S0)
        u, v, T, S = self.linear(*self.nonlinear(*self.linear(u0, v0, T0, S0)))
        fx, fy = (F for _, F in self.pressure_grad(T, S))
        mean = lambda a: (0.5 * (a[..., :-1] + a[..., 1:]) * (self.gap / self.H)).sum(-1)  # noqa: E731
        ub0, vb0 = mean(u), mean(v)
        eta, ub, vb = self.barotropic(eta, ub0, vb0, fx, fy)
        new = (u + (ub - ub0)[:, :, None], v + (vb - vb0)[:, :, None], T, S)
        out = [self.cap(a, self.wm) * self.wm + h * (1 - self.wm) for a, h in zip(new, (u0, v0, T0, S0))]
        out[1] = _zero_row(_zero_row(out[1], 0), -1)
        return (*out, eta)

    def closure(self, u, v, T, S):
        """Diffusivity per interface from the network on the state's columns."""
        wm, nz, dev = self.wm, self.nz, T.device
        X = torch.zeros((self.nx, self.ny, 256), dtype=torch.float64, device=dev)
        Ta, Sa = T - self.ph.T_ref, S - self.ph.S_ref
        for q, a in enumerate((Ta * 0.1, Sa, u * 2, v * 2)):
            X[..., 50 * q:50 * q + nz] = a * wm
        n2 = G * (-ALPHA * (Ta[..., 1:] - Ta[..., :-1]) + BETA * (Sa[..., 1:] - Sa[..., :-1])) / self.gap
        X[..., 200:199 + nz] = torch.asinh(n2 * 1e8) * 0.25 * self.wif
        X[..., 250] = torch.hypot(self.tau_x, self.tau_y) * 10
        X[..., 251] = self.q * 0.01
        k = (10.0 ** _mlp(self.net, X.reshape(-1, 256))[0]).clamp(1e-7, 1.0).reshape(self.nx, self.ny, 64)[..., :nz - 1]
        plain = self.kv + self.ph.kappa_conv * self.gates(T, S)
        trusted = X.abs().amax(-1, keepdim=True) <= 8.0
        return torch.where(trusted, k, plain) * self.wif


def _blocks(p):
    W1, b1, W2, b2, W3, b3 = torch.split(p, [65536, 256, 65536, 256, 16384, 64])
    return W1.view(256, 256), b1, W2.view(256, 256), b2, W3.view(64, 256), b3


def _mlp(params, X):
    W1, b1, W2, b2, W3, b3 = _blocks(params)
    gelu = lambda x: 0.5 * x * (1 + torch.erf(x / math.sqrt(2)))  # noqa: E731
    Z1 = X @ W1.T + b1
    H1 = gelu(Z1)
    Z2 = H1 @ W2.T + b2
    H2 = gelu(Z2)
    return H2 @ W3.T + b3, Z1, H1, Z2, H2


def _exact_train(case, seed, gen):
    X, T, M = (a.double() for a in _closure_rows(case["rows"], gen))
    p = torch.as_tensor(init_params(seed), device=DEV).double()
    m = (1e-3 * torch.randn(p.shape, generator=gen, device=DEV)).double()
    v = (1e-5 * (0.1 + torch.rand(p.shape, generator=gen, device=DEV))).double()
    W1, _, W2, _, W3, _ = _blocks(p)
    Y, Z1, H1, Z2, H2 = _mlp(p, X)
    slope = lambda x: 0.5 * (1 + torch.erf(x / math.sqrt(2))) + x * torch.exp(-0.5 * x * x) / math.sqrt(2 * math.pi)  # noqa: E731
    dY = 2 * (Y - T) * M / M.sum()
    d2 = (dY @ W3) * slope(Z2)
    d1 = (d2 @ W2) * slope(Z1)
    g = torch.cat([a.reshape(-1) for a in (d1.T @ X, d1.sum(0), d2.T @ H1, d2.sum(0), dY.T @ H2, dY.sum(0))])
    m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
    p = p - 1e-3 * (m / (1 - 0.9 ** 101)) / (torch.sqrt(v / (1 - 0.999 ** 101)) + 1e-8)
    return dict(params=p, m=m, v=v)


def _exact_history(x, u, v, T, S, eta):
    rho = RHO0 * (-ALPHA * (T - x.ph.T_ref) + BETA * (S - x.ph.S_ref))
    r = rho * x.wm
    p = torch.nn.functional.pad(torch.cumsum(G * 0.5 * (r[..., :-1] + r[..., 1:]) * x.gap, -1), (1, 0))
    Fz = x.transport(u, v)
    zero = torch.zeros_like(T)
    terms = [x.advect(T, u, v, Fz), x.hdiff(T, x.kh), x.vdiff(T), x.convect(T, x.gates(T, S), x.ph.kappa_conv)]
    area = x.dx * x.dy
    vol = area[:, :, None] * x.dzn * x.wm
    top = area * x.wm[..., 0]
    V, VT, VS, A = vol.sum(), (vol * T).sum(), (vol * S).sum(), top.sum()
    budget = dict(mean_T=VT / V, mean_S=VS / V, mean_T_top=(top * T[..., 0]).sum() / A,
                  mean_S_top=(top * S[..., 0]).sum() / A, heat_content_J=RHO0 * CP * VT,
                  salt_content_kg=RHO0 / 1000 * VS, total_volume_m3=V, mean_depth_m=V / area.sum())
    return dict(rho=RHO0 + rho, pressure=RHO0 * G * eta[:, :, None] + p, w=-Fz * x.wm,
                terms=torch.stack([a * x.wm for a in terms] + [zero, zero]),
                budget={k: float(a) for k, a in budget.items()})


def _exact_step(form, nx, ny, nz, steps, gen, seed):
    grid, physics, dt, kw, T, S = _config(form, nx, ny, nz, gen)
    fields = [a.double() for a in _state(grid, physics, T, S, gen, moving=form != "smoke")]
    x = _Exact(grid, physics, dt, kw, form)
    if form == "learned":
        x.net = torch.as_tensor(init_params(seed), device=DEV).double()
    if form == "precision":
        day, pos = 28.0 + (seed % 5), (28.0 + (seed % 5)) % 30.0
        mi = int(day // 30) % 12
        after, before = min(1.0, max(0.0, (pos - 27.5) / 5)), min(1.0, max(0.0, (2.5 - pos) / 5))
        x.tau_x, x.tau_y, x.q = ((1 - after - before) * m[mi].double() + after * m[(mi + 1) % 12].double()
                                 + before * m[(mi - 1) % 12].double() for m in _months(grid, gen))
    return x, fields, steps


def exact(case, seed):
    """The outputs of ``run`` for these inputs in float64."""
    kind, gen = case["kind"], _gen(seed)
    if kind == "infer":
        X = _closure_rows(case["rows"], gen)[0].double()
        p = torch.as_tensor(init_params(seed), device=DEV).double()
        return torch.cat([_mlp(p, a)[0] for a in X.split(32768)])
    if kind == "train":
        return _exact_train(case, seed, gen)
    if kind == "ensemble":
        out = []
        for q, size in _members(case):
            x, f, _ = _exact_step("plain", *size, 1, _gen(seed + 101 * q), seed)
            out.append(dict(zip(("u", "v", "T", "S", "eta"), x.step(*f))))
        return out
    size = case["nx"], case["ny"], case["nz"]
    x, f, steps = _exact_step(case["form"], *size, case.get("steps", 1), gen, seed)
    if kind == "history":
        return _exact_history(x, *f)
    for _ in range(steps):
        f = x.step(*f)
    out = dict(zip(("u", "v", "T", "S", "eta"), f))
    return {k: a.cpu().numpy() for k, a in out.items()} if kind == "host" else out
