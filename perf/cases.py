"""Timed workloads of the modeling / RTM library, through its public entry points.

A case is one call that a program makes: model a shot, migrate a shot or a
batch, model with the first-order scheme, or train the learned corrector.
Kinds:

  forward   Context.forward: one shot, gathers (and fields) to the host
  rtm       Context.rtm_batch of n shots on given records, then Context.stack
  survey    Context.survey_rtm of n shots on sub-grids of uneven width
  gradient  rtm with the FWI gradient, then Context.gradient
  fo_fwd    Context.forward_first_order with the final fields
  fo_bwd    Context.backward_first_order of given records
  train     Net.forward_dev + zero_grad + backward_dev + grads

All arrays of a wave-equation call are host arrays: that is what these entry
points take and return.  ``exact`` is the same mathematics in 64-bit torch.
"""
import math

import numpy as np
import torch

import ouc_b200 as o
from ouc_b200.corrector import N_IN, N_OUT, WIDTH, Net
from ouc_b200.learned import LAYERS, TAPS, init_params

# 64-bit staggered weights by half-order; the first-order scheme has its own
# five-digit ones at half-order 6
WEIGHTS = {
    2: (1.125, -1.0 / 24.0),
    5: (19845.0 / 16384.0, -735.0 / 8192.0, 567.0 / 40960.0, -405.0 / 229376.0, 35.0 / 294912.0),
    6: (1.2213364, -9.6931458e-2, 1.7447662e-2, -2.9672895e-3, 3.5900540e-4, -2.1847812e-5),
}
FO_WEIGHTS6 = (1.2213, -9.6931e-2, 1.7448e-2, -2.9673e-3, 3.5901e-4, -2.1848e-5)

BASE = dict(kind="forward", nx=256, nz=256, npml=20, N=5, dx=10.0, nt=1000, n=1, density=0, force=0, tx=0, fields=0,
            snap=0, prec="fp32", comp=0, exact_align=0, mute=1)


def _case(name=None, **kw):
    c = dict(BASE)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a quick look at a small model, one shot, with the reference's own stencil order
        _case("forward_tiny", nx=120, nz=80, npml=20, N=6, dx=10.0, nt=400, fields=1),
        # plain single-shot modeling on the 256 x 256 two-layer sized grid
        _case("forward_256", nx=256, nz=256, npml=20, N=5, dx=10.0, nt=1000),
        # the cheap fourth-order run on a coarse grid, time-major gathers, vertical-force source
        _case("forward_coarse_n2", nx=501, nz=250, npml=15, N=2, dx=10.0, nt=1000, tx=1, force=1),
        # one shot on a large model with a density model
        _case("forward_large_density", nx=4000, nz=1500, npml=30, N=5, dx=4.0, nt=80, density=1, fields=1),
        # one RTM shot of field records on an odd-sized mid-size model, sixth-order stencil
        _case("rtm_shot_odd", kind="rtm", nx=347, nz=251, npml=25, N=6, dx=8.0, nt=2100),
        # the flagship: a batch of 16 RTM shots on the 1000 x 500 grid
        _case("rtm_batch_1000x500", kind="rtm", nx=1000, nz=500, npml=30, N=5, dx=5.0, nt=300, n=16),
        # the precision form: scaled-FP16 snapshots every 4 levels and compensated sums
        _case("rtm_snap_fp16", kind="rtm", nx=301, nz=200, npml=30, N=5, dx=8.0, nt=1750, n=6, snap=4, prec="fp16", comp=1,
              exact_align=1),
        # a survey batch: uneven apertures of a 2000 x 800 model, time-major records
        _case("survey_2000x800", kind="survey", nx=2000, nz=800, npml=30, N=5, dx=5.0, nt=160, n=6, tx=1),
        # FWI: gradient of a small batch
        _case("gradient_batch", kind="gradient", nx=240, nz=150, npml=20, N=5, dx=10.0, nt=1350, n=6, mute=0),
        # the first-order scheme, forward on the 1000 x 500 grid
        _case("first_order_forward", kind="fo_fwd", nx=1000, nz=500, npml=30, N=5, dx=5.0, nt=400),
        # the first-order scheme, back-propagation of records on a small odd grid
        _case("first_order_backward", kind="fo_bwd", nx=301, nz=203, npml=20, N=6, dx=10.0, nt=600),
        # one training step of the corrector on a minibatch of coarse states (n images of nx x nz cells)
        _case("corrector_step", kind="train", nx=290, nz=158, n=4, npml=0, nt=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "rtm", "rtm", "survey", "gradient", "fo_fwd", "fo_bwd", "train"])
    N = rng.choice([2, 5, 5, 6])
    npml = rng.randint(max(N, 10), 34)
    dx = rng.choice([5.0, 8.0, 10.0])
    if kind == "train":
        return _case(kind=kind, nx=_log(rng, 60, 400), nz=_log(rng, 60, 300), n=rng.randint(1, 6), npml=0, nt=1)
    tx = rng.randint(0, 1)
    if kind == "forward":
        nx, nz = _log(rng, 60, 2500), _log(rng, 50, 900)
        density, force, fields = rng.randint(0, 1), rng.randint(0, 1), rng.randint(0, 1)
        nt = max(60, min(1000, int(6e7 / (nx * nz))))
        return _case(kind=kind, nx=nx, nz=nz, npml=npml, N=N, dx=dx, nt=nt, tx=tx, density=density, force=force,
                     fields=fields)
    if kind in ("fo_fwd", "fo_bwd"):
        nx, nz = _log(rng, 60, 1200), _log(rng, 50, 600)
        return _case(kind=kind, nx=nx, nz=nz, npml=npml, N=N, dx=dx, nt=max(60, min(800, int(6e7 / (nx * nz)))), tx=tx)
    n = 1 if rng.random() < 0.4 else rng.randint(2, 12)
    nx, nz = _log(rng, 90, 1100), _log(rng, 70, 500)
    nt = max(60, min(1200, int(1.2e8 / (nx * nz * n))))
    if kind == "survey":
        return _case(kind=kind, nx=nx + 200, nz=nz, npml=npml, N=N, dx=dx, nt=max(60, nt // 2), n=n, tx=tx)
    if kind == "gradient":
        return _case(kind=kind, nx=nx, nz=nz, npml=npml, N=N, dx=dx, nt=max(60, nt // 2), n=min(n, 6), mute=0, tx=tx)
    snap = rng.choice([0, 0, 2, 4])
    return _case(kind=kind, nx=nx, nz=nz, npml=npml, N=N, dx=dx, nt=nt, n=n, tx=tx, snap=snap,
                 prec=rng.choice(["fp16", "bf16", "fp32"]) if snap else "fp32", comp=rng.randint(0, 1),
                 exact_align=rng.randint(0, 1), mute=rng.randint(0, 1))


# ---- inputs -------------------------------------------------------------------

def _dt(c):
    return c["dx"] * 1e-4          # Courant number 0.84 at 4500 m/s for half-order 5


def _fm(c):
    return 125.0 / c["dx"]


def _inputs(c, seed):
    """Model, wavelet, shots and records of a case, from the seed alone."""
    rng = np.random.default_rng(seed)
    nx, nz, nt, dx, dt, n = c["nx"], c["nz"], c["nt"], c["dx"], _dt(c), c["n"]
    # flat layers with a gentle lateral trend, smoothed along depth for migration
    z = np.arange(nz)
    cuts = np.sort(rng.choice(np.arange(1, nz), size=7, replace=False))
    v1 = rng.uniform(1800.0, 4400.0, 8)[np.searchsorted(cuts, z, side="right")]
    if c["kind"] in ("rtm", "survey", "gradient"):
        k = np.exp(-0.5 * (np.arange(-30, 31) / 10.0) ** 2)
        v1 = np.convolve(np.pad(v1, 30, mode="edge"), k / k.sum(), mode="valid")
    trend = 1.0 + 0.015 * np.sin(2 * np.pi * (np.arange(nx) / nx + rng.uniform()))
    vp = (trend[:, None] * v1[None, :]).astype(np.float32)
    vs = (vp / np.float32(rng.uniform(1.6, 2.0))).astype(np.float32)
    rho = (310.0 * vp.astype(np.float64) ** 0.25).astype(np.float32)
    w, t0 = o.ricker(_fm(c), dt, nt)
    w = (w * np.float32(rng.uniform(0.5, 2.0))).astype(np.float32)
    d = dict(vp=vp, vs=vs, rho=rho, w=w)
    src_type = o.SRC_FORCE_Z if c["force"] else o.SRC_THETA
    sx = np.linspace(nx * 0.25, nx * 0.75, n) + rng.uniform(-0.1, 0.1, n) * nx / max(n, 2)
    row = int(rng.integers(2, 6))
    d["shots"] = [o.Shot(int(x), row, row, src_type, t0, c["mute"]) for x in sx]
    if c["kind"] == "survey":
        d["ap"] = []
        for k, s in enumerate(d["shots"]):
            wd = int((0.3 + 0.45 * ((k + 1) * 0.618034 % 1.0)) * nx)     # uneven widths, the same for every seed
            x0 = int(max(0, min(s.sx - wd // 2, nx - wd)))
            d["ap"].append((x0, x0 + wd))
    if c["kind"] in ("rtm", "survey", "gradient", "fo_bwd"):
        d["recs"] = []
        for k, s in enumerate(d["shots"]):
            x0, x1 = d["ap"][k] if "ap" in d else (0, nx)
            d["recs"].append(_records(c, rng, s, x0, x1 - x0 + 2 * c["npml"]))
    return d


def _records(c, rng, shot, x0, X):
    """Field-like records of a shot: a direct arrival and hyperbolic reflections
    (Ricker wavelets), both components, in the case's gather layout."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nt, dt, fm = c["nt"], _dt(c), _fm(c)
    off = (torch.arange(X, device=dev) - c["npml"] + x0 - shot.sx) * c["dx"]
    t = torch.arange(nt, device=dev) * dt
    out = [torch.zeros(X, nt, device=dev) for _ in range(2)]
    for _ in range(6):
        ta, v, amp = rng.uniform(0.02, 0.9) * nt * dt, rng.uniform(1800, 3800), rng.uniform(0.2, 1.0) * 1e-7
        arg = (math.pi * fm) ** 2 * (t[None, :] - torch.sqrt(ta * ta + (off / v) ** 2)[:, None]) ** 2
        ev = amp * (1 - 2 * arg) * torch.exp(-arg)
        out[0] += ev * torch.sign(off)[:, None]
        out[1] += ev
    return tuple(np.ascontiguousarray((r.T if c["tx"] else r).cpu().numpy()) for r in out)


def _config(c):
    prec = {"fp32": o.PREC_FP32, "fp16": o.PREC_FP16, "bf16": o.PREC_BF16}[c["prec"]]
    return o.Config(nx=c["nx"], nz=c["nz"], npml=c["npml"], dx=c["dx"], dz=c["dx"], dt=_dt(c), nt=c["nt"],
                    half_order=c["N"], strip_precision=prec, compensated_image=c["comp"],
                    image_align=o.IMAGE_EXACT if c["exact_align"] else o.IMAGE_REFERENCE,
                    gather_layout=o.GATHER_TX if c["tx"] else o.GATHER_XT, max_batch=c["n"], snapshot_every=c["snap"],
                    density=c["density"], gradient=1 if c["kind"] == "gradient" else 0)


def _train_inputs(c, seed):
    """Network parameters, a minibatch of states at rest outside a wavefront
    band, and the loss gradient of its outputs."""
    g = torch.Generator().manual_seed(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n, H, W = c["n"], c["nx"], c["nz"]
    x = torch.randn(n, H, W, N_IN, generator=g)
    r = torch.hypot(torch.arange(H)[:, None] - H / 2.0, torch.arange(W)[None, :] * 1.0)
    ring = torch.stack([torch.exp(-((r - (0.2 + 0.7 * (k + 1) / n) * max(H, W)) / 12.0) ** 2) for k in range(n)])
    x = x * ring[..., None]
    x[x.abs() < 1e-4] = 0.0
    go = torch.randn(n, H, W, N_OUT, generator=g) * ring[..., None] / (n * H * W * N_OUT)
    p = init_params(seed)
    # small seeded biases, so that their gradients are exercised
    return p, x.contiguous().to(dev), go.contiguous().to(dev)


def prepare(case, seed):
    c = case
    if c["kind"] == "train":
        p, x, go = _train_inputs(c, seed)
        out = torch.empty(c["n"], c["nx"], c["nz"], N_OUT, device=x.device)
        return dict(c=c, net=Net(0, p), x=x, go=go, out=out)
    d = _inputs(c, seed)
    rho = d["rho"] if c["density"] or c["kind"] == "gradient" else None
    d["ctx"] = o.Context(_config(c), d["vp"], d["vs"], rho)
    d["c"] = c
    return d


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "train":
        net, st = state["net"], torch.cuda.current_stream().cuda_stream
        n, H, W = c["n"], c["nx"], c["nz"]
        net.forward_dev(n, H, W, state["x"].data_ptr(), state["out"].data_ptr(), st)
        net.zero_grad(st)
        net.backward_dev(state["go"].data_ptr(), st)
        return {"out": state["out"], "grads": net.grads()}
    ctx, w, shots = state["ctx"], state["w"], state["shots"]
    if kind == "forward":
        gx, gz, f = ctx.forward(shots[0], w, fields=bool(c["fields"]))
        return {"gx": gx, "gz": gz, "fields": f}
    if kind == "fo_fwd":
        gx, gz, f = ctx.forward_first_order(shots[0], w, fields=True)
        return {"gx": gx, "gz": gz, "fields": f}
    if kind == "fo_bwd":
        return {"fields": ctx.backward_first_order(shots[0], *state["recs"][0])}
    if kind == "survey":
        imgs = ctx.survey_rtm(shots, state["ap"], w, state["recs"])
    else:
        imgs = ctx.rtm_batch(shots, w, state["recs"])
    out = {"images": imgs, "stack": ctx.stack(reset=True)}
    if kind == "gradient":
        out["gradient"] = ctx.gradient(reset=True)
    return out


# ---- necessary work -------------------------------------------------------------

def work(case):
    c = case
    if c["kind"] == "train":
        P = c["n"] * c["nx"] * c["nz"]
        macs = sum(ci * co * TAPS for ci, co in LAYERS)
        dgrad = sum(ci * co * TAPS for ci, co in LAYERS[1:])
        # input, output, output gradient once; the three hidden activations in
        # 16 bits written once and read by the backward pass
        return {"bytes": P * (4 * (N_IN + 2 * N_OUT) + 3 * 2 * 2 * WIDTH), "flops": 2.0 * P * (2 * macs + dgrad)}
    L, N, nt, n = c["npml"], c["N"], c["nt"], c["n"]
    X, Z = c["nx"] + 2 * L, c["nz"] + 2 * L
    if c["kind"] == "survey":
        X = int(0.525 * c["nx"]) + 2 * L
    cells, inner = X * Z, (X - 2 * L) * c["nz"]
    damped = 2 * L * Z + 2 * L * X
    deriv = 3 * N                                   # N differences, N multiply-adds less one add, one division
    step_f = cells * (12 * deriv + 60)
    if c["kind"] in ("fo_fwd", "fo_bwd"):
        # 12 states read and written, four model fields; records one row
        return {"bytes": nt * (cells * (2 * 48 + 16) + 8 * X), "flops": nt * cells * (12 * deriv + 70.0)}
    # P and S at two levels read, one written, two moduli read; six damping
    # memories per damped cell and axis read and written; one record row
    step_b = 56 * cells + 48 * damped + 8 * X
    if c["kind"] == "forward":
        return {"bytes": nt * (step_b + (8 * cells if c["density"] else 0)), "flops": float(nt * step_f)}
    ring = 4 * N * (X - 2 * L + c["nz"])
    back_b, back_f = step_b, step_f
    if c["snap"]:
        el = 4 if c["prec"] == "fp32" else 2
        acc = 48 if c["comp"] else 24
        img = inner * (2 * 2 * el + 2 * 4 + 16 + acc) / c["snap"]
        tot = 2 * step_b + img
        fl = 2 * step_f + inner * 12 / c["snap"]
    else:
        rec_b = (56 + 24 + 16 + (24 if c["comp"] else 0)) * inner + 32 * ring
        tot = step_b + 32 * ring + back_b + rec_b
        fl = step_f + back_f + inner * (12 * deriv + 60)
    if c["kind"] == "gradient":
        tot += inner * (32 + 12 + 24)
        fl += inner * (8 * deriv + 40)
    return {"bytes": float(n * nt * tot), "flops": float(n * nt * fl)}


# ---- the same in 64 bits ----------------------------------------------------------

class Sim64:
    """The second-order scheme of a batch of shots on one padded grid."""

    def __init__(self, vp, vs, rho, c, dev):
        L, N = c["npml"], c["N"]
        self.L, self.N, self.dev = L, N, dev
        self.X, self.Z = vp.shape
        f32 = lambda v: float(np.float32(v))  # noqa: E731
        self.h, self.dt = f32(c["dx"]), f32(_dt(c))
        self.a = WEIGHTS[N]
        self.vp, self.vs = vp, vs
        self.vp2, self.vs2 = vp * vp, vs * vs
        self.b = None
        if rho is not None:
            self.vp2, self.vs2 = self.vp2 * rho, self.vs2 * rho
            b = 1.0 / rho
            bx, bz = b.clone(), b.clone()
            bx[:-1] = 0.5 * (b[:-1] + b[1:])
            bz[:, :-1] = 0.5 * (b[:, :-1] + b[:, 1:])
            self.b = (bx, bz)
        self.ax, self.az = damping64(vp, L)
        i = torch.arange(self.X, device=dev)[:, None]
        j = torch.arange(self.Z, device=dev)[None, :]
        self.live = ((i >= N) & (i < self.X - N) & (j >= N) & (j < self.Z - N)).double()
        self.inner = (i >= L) & (i < self.X - L) & (j >= L) & (j < self.Z - L)
        box = (i >= L - N) & (i < self.X - L + N) & (j >= L - N) & (j < self.Z - L + N)
        deep = (i >= L + N) & (i < self.X - L - N) & (j >= L + N) & (j < self.Z - L - N)
        self.ring = (box & ~deep).reshape(-1).nonzero()[:, 0]

    def zeros(self, n, k):
        return [torch.zeros(n, self.X, self.Z, dtype=torch.float64, device=self.dev) for _ in range(k)]

    def d(self, f, dim, plus):
        return diff64(f, dim, plus, self.a, self.h)

    def s_stage(self, u, F, live):
        ux, uz = u
        exx, ezx = self.d(ux, 1, False), self.d(uz, 1, True)
        exz, ezz = self.d(ux, 2, True), self.d(uz, 2, False)
        if F is None:
            return [self.vp2 * (exx + ezz), self.vs2 * (exz - ezx), self.vs2 * ezx, self.vs2 * ezz, self.vs2 * exx,
                    self.vs2 * exz]
        for m, e, d in ((F[0], exx, self.ax), (F[1], ezz, self.az), (F[2], exz, self.az), (F[3], ezx, self.ax)):
            m.add_((e - m) * d * live, alpha=self.dt)
        fxx, fzz, fxz, fzx = F
        th, om = self.vp2 * (exx + ezz - fxx - fzz), self.vs2 * (exz - ezx - fxz + fzx)
        return [v * live for v in (th, om, self.vs2 * (ezx - fzx), self.vs2 * (ezz - fzz), self.vs2 * (exx - fxx),
                                   self.vs2 * (exz - fxz))]

    def u_stage(self, s, O, now, past, live):
        """New level into `past`."""
        th, om, qzx, qzz, qxx, qxz = s
        tx, wx, B, E = self.d(th, 1, True), self.d(om, 1, False), self.d(qxz, 1, False), self.d(qzz, 1, True)
        tz, wz, A, C = self.d(th, 2, True), self.d(om, 2, False), self.d(qxx, 2, True), self.d(qzx, 2, False)
        if O is not None:
            vals = []
            for m, v, d in zip(O, (C, A, tz, wz, E, B, tx, wx), (self.az,) * 4 + (self.ax,) * 4):
                m.add_((v - m) * d * live, alpha=self.dt)
                vals.append(v - m)
            C, A, tz, wz, E, B, tx, wx = vals
        acc = [tx + C - E, tz + B - A, wz + C - E, B - A - wx]
        if self.b is not None:
            acc = [acc[0] * self.b[0], acc[1] * self.b[1], acc[2] * self.b[0], acc[3] * self.b[1]]
        dt2 = float(np.float32(self.dt) * np.float32(self.dt))
        for p, q, a in zip(past, now, acc):
            p.copy_((2 * q - p + dt2 * a) * live)


def damping64(vp, L):
    """The absorbing profile of a padded Vp (R = 1e-3)."""
    X, Z = vp.shape

    def profile(n):
        k = np.arange(n, dtype=np.float64)
        d = np.where(k < L, L - k, np.where(k > n - L, k - n + L, 0.0))
        return torch.from_numpy((d / L) ** 4).to(vp.device)

    g = math.log10(1e3) * 1.5 / L
    return g * vp * profile(X)[:, None], g * vp * profile(Z)[None, :]


def diff64(f, dim, plus, a, h):
    """Staggered derivative along axis `dim` of [n][X][Z], zero outside."""
    N, n = len(a), f.shape[dim]
    p = torch.nn.functional.pad(f, (0, 0, N, N) if dim == 1 else (N, N))
    acc = torch.zeros_like(f)
    for k in range(1, N + 1):
        hi, lo = (k, 1 - k) if plus else (k - 1, -k)
        acc.add_(p.narrow(dim, N + hi, n) - p.narrow(dim, N + lo, n), alpha=a[k - 1] / h)
    return acc


def _pad64(f, L, dev):
    return torch.from_numpy(np.pad(f.astype(np.float64), L, mode="edge")).to(dev)


def _forward64(c, sim, shots, w, record=True, save=None):
    """Forward run of the shots; `save(t, u_new, s, p_new)` after each step."""
    n, L, dev = len(shots), c["npml"], sim.dev
    now, past, F, O = sim.zeros(n, 4), sim.zeros(n, 4), sim.zeros(n, 4), sim.zeros(n, 8)
    b = torch.arange(n, device=dev)
    sx = torch.tensor([s.sx + L for s in shots], device=dev)
    sz = torch.tensor([s.sz + L for s in shots], device=dev)
    rz = shots[0].rz + L
    wd = w.astype(np.float64)
    gx = torch.zeros(n, c["nt"], sim.X, dtype=torch.float64, device=dev) if record else None
    gz = torch.zeros_like(gx) if record else None
    dt2 = float(np.float32(sim.dt) * np.float32(sim.dt))
    for t in range(c["nt"]):
        s = sim.s_stage((now[0] + now[2], now[1] + now[3]), F, sim.live)
        if not c["force"]:
            s[0][b, sx, sz] += wd[t]
        sim.u_stage(s, O, now, past, sim.live)
        if c["force"]:
            past[1][b, sx, sz] += dt2 * wd[t]
        now, past = past, now
        if record:
            gx[:, t], gz[:, t] = now[0][:, :, rz] + now[2][:, :, rz], now[1][:, :, rz] + now[3][:, :, rz]
        if save:
            save(t, now, s)
    return now, past, gx, gz


def _rtm64(c, vp, vs, rho_formula, shots, w, recs, dev):
    """RTM of shots on one grid: illumination and FWI gradient per shot."""
    sim = Sim64(vp, vs, None, c, dev)
    n, nt, L, N, K = len(shots), c["nt"], c["npml"], c["N"], c["snap"]
    X, Z = sim.X, sim.Z
    strips_u, strips_s, snaps = {}, {}, {}
    want = set()
    if K:
        for t in range(nt - 1, -1, -K):
            want.add(t if (c["exact_align"] or t == nt - 1) else t + 1)

    def save(t, now, s):
        if K:
            if t in want:
                snaps[t] = (now[0].clone(), now[1].clone())
            return
        u = (now[0] + now[2], now[1] + now[3])
        strips_u[t] = torch.stack([v.reshape(n, -1)[:, sim.ring] for v in u])
        strips_s[t] = torch.stack([v.reshape(n, -1)[:, sim.ring] for v in s])

    now, past, _, _ = _forward64(c, sim, shots, w, record=False, save=save)
    # records, time-major, with the direct-wave mute
    inj = torch.zeros(2, n, nt, X, dtype=torch.float64, device=dev)
    tt = torch.arange(nt, device=dev, dtype=torch.float64)[:, None]
    for k, (s, r) in enumerate(zip(shots, recs)):
        keep = 1.0
        if s.mute:
            i = torch.arange(X, device=dev, dtype=torch.float64)
            dist = torch.hypot(i - (s.sx + L), torch.tensor(float(s.rz - s.sz), dtype=torch.float64, device=dev))
            v = float(vp[s.sx + L, s.rz + L])
            keep = (tt >= (2 * s.t0 + dist * sim.h / (sim.dt * v))[None, :]).double()
        for q in range(2):
            a = torch.from_numpy(r[q].astype(np.float64)).to(dev)
            inj[q, k] = (a if c["tx"] else a.T) * keep
    rz = shots[0].rz + L
    rn, rp, F, O = sim.zeros(n, 4), sim.zeros(n, 4), sim.zeros(n, 4), sim.zeros(n, 8)
    il = sim.zeros(n, 1)[0]
    grad = sim.zeros(n, 3) if c["kind"] == "gradient" else None
    b = torch.arange(n, device=dev)
    sx = torch.tensor([s.sx + L for s in shots], device=dev)
    sz = torch.tensor([s.sz + L for s in shots], device=dev)
    wd = w.astype(np.float64)
    inner = sim.inner.double()
    edge = slice(L + N, X - L - N), slice(L + N, Z - L - N)

    def image(px, pz):
        il.add_((px * px + pz * pz) * inner)

    for t in range(nt - 1, -1, -1):
        if grad is not None:
            u = [rn[0] + rn[2], rn[1] + rn[3]]
            for q in range(2):
                u[q][:, L:X - L, rz] = inj[q, :, t, L:X - L]
            sim.u_stage(sim.s_stage(u, F, sim.live), O, rn, rp, sim.live)
            rn, rp = rp, rn
        if K:
            f = t if (c["exact_align"] or t == nt - 1) else t + 1
            if (nt - 1 - t) % K == 0:
                image(*snaps[f])
            continue
        ref_past = t < nt - 1 and not c["exact_align"]
        if grad is not None:
            s4 = past if ref_past else now
            us, ur = (s4[0] + s4[2], s4[1] + s4[3]), (rn[0] + rn[2], rn[1] + rn[3])
            e = [[sim.d(v[0], 1, False), sim.d(v[1], 2, False), sim.d(v[1], 1, True), sim.d(v[0], 2, True)] for v in (us, ur)]
            (sxx, szz, szx, sxz), (rxx, rzz, rzx, rxz) = e
            vs2 = sim.vs2
            gs = vs2 * ((rxz - rzx) * (sxz - szx) + rzx * szx + rzz * szz + rxz * sxz + rxx * sxx)
            for g, v in zip(grad, (-2 * rho_formula * vp * (sxx + szz) * sim.vp2 * (rxx + rzz), -2 * rho_formula * vs * gs,
                                   us[0] ** 2 + us[1] ** 2)):
                g[:, edge[0], edge[1]] += v[:, edge[0], edge[1]]
        if t == nt - 1:
            image(now[0], now[1])
            now, past = past, now
            continue
        src = past if ref_past else now
        image(src[0], src[1])
        u = [now[0] + now[2], now[1] + now[3]]
        slot_u = nt - 2 if t + 1 == nt - 1 else t + 1       # the reference restores these one level late
        for q in range(2):
            u[q].view(n, -1)[:, sim.ring] = strips_u[slot_u][q]
        s = sim.s_stage(u, None, None)
        if t + 1 == nt - 1 and not c["force"]:
            s[0][b, sx, sz] += wd[t + 1]
        for q in range(6):
            s[q].view(n, -1)[:, sim.ring] = strips_s[t + 1][q]
        sim.u_stage(s, None, now, past, inner)
        now, past = past, now
        strips_s.pop(t + 1)
    return il[:, L:-L, L:-L] * (K or 1), grad


def _first_order64(c, vp, vs, shot, w, rec, dev):
    L, N, nt = c["npml"], c["N"], c["nt"]
    X, Z = vp.shape
    a = FO_WEIGHTS6 if N == 6 else WEIGHTS[N]
    h, dt = float(np.float32(c["dx"])), float(np.float32(_dt(c)))
    ax, az = damping64(vp, L)
    live = torch.zeros(X, Z, dtype=torch.float64, device=dev)
    live[N:X - N, N:Z - N] = 1.0
    damp = [(1.0 - 0.5 * dt * d, live / (1.0 + 0.5 * dt * d)) for d in (ax, az)]
    cp, cs = dt * vp * vp, dt * vs * vs
    v = [torch.zeros(1, X, Z, dtype=torch.float64, device=dev) for _ in range(4)]
    s = [torch.zeros(1, X, Z, dtype=torch.float64, device=dev) for _ in range(8)]
    rz, sx, sz = shot.rz + L, shot.sx + L, shot.sz + L
    d = lambda f, dim, plus: diff64(f, dim, plus, a, h)  # noqa: E731
    gx, gz = [torch.zeros(nt, X, dtype=torch.float64, device=dev) for _ in range(2)]
    inj = None
    if rec is not None:
        inj = [torch.from_numpy(r.astype(np.float64)).to(dev) for r in rec]
        inj = [r if c["tx"] else r.T for r in inj]
    for k in range(nt):
        t = k if rec is None else nt - 1 - k
        ux, uz = v[0] + v[2], v[1] + v[3]
        if inj is not None:
            ux[:, L:X - L, rz], uz[:, L:X - L, rz] = inj[0][t, L:X - L], inj[1][t, L:X - L]
        xx, zx, xz, zz = d(ux, 1, False), d(uz, 1, True), d(ux, 2, True), d(uz, 2, False)
        for f, term in enumerate((cp * xx, cp * zz, -cs * zx, cs * xz, cs * xx, cs * xz, cs * zx, cs * zz)):
            keep, scale = damp[f & 1]
            s[f] = (term + keep * s[f]) * scale
        th, om = s[0] + s[1], s[2] + s[3]
        if rec is None:
            th[0, sx, sz] += float(w[t])
        tx, wx, B, E = d(th, 1, True), d(om, 1, False), d(s[5], 1, False), d(s[7], 1, True)
        tz, wz, A, C = d(th, 2, True), d(om, 2, False), d(s[4], 2, True), d(s[6], 2, False)
        for f, q in enumerate((tx + C - E, tz + B - A, wz + C - E, B - A - wx)):
            keep, scale = damp[f & 1]
            v[f] = (keep * v[f] + dt * q) * scale
        if rec is None:
            gx[t], gz[t] = v[0][0, :, rz] + v[2][0, :, rz], v[1][0, :, rz] + v[3][0, :, rz]
    fields = torch.cat([v[0] + v[2], v[1] + v[3], v[0], v[1], v[2], v[3], th, om, s[6], s[7], s[4], s[5], s[0], s[1], s[2], s[3]])
    return gx, gz, fields


def _train64(c, seed):
    p, x, go = _train_inputs(c, seed)
    q, at, ws = torch.from_numpy(p.astype(np.float64)).to(x.device), 0, []
    for ci, co in LAYERS:
        ws.append((q[at:at + co * ci * TAPS].view(co, ci, 5, 5).clone().requires_grad_(True),
                   q[at + co * ci * TAPS:at + co * ci * TAPS + co].clone().requires_grad_(True)))
        at += co * ci * TAPS + co
    y = x.double().permute(0, 3, 1, 2)
    for k, (wt, b) in enumerate(ws):
        y = torch.nn.functional.conv2d(y, wt, b, padding=2)
        y = torch.relu(y) if k < len(ws) - 1 else y
    y = y.permute(0, 2, 3, 1)
    g = torch.autograd.grad(y, [v for pair in ws for v in pair], go.double())
    return {"out": y.detach().contiguous(), "grads": torch.cat([v.reshape(-1) for v in g]).cpu().numpy()}


def exact(case, seed):
    c = case
    if c["kind"] == "train":
        return _train64(c, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    L, nt, kind, n = c["npml"], c["nt"], c["kind"], c["n"]
    X, Z = c["nx"] + 2 * L, c["nz"] + 2 * L
    runs = {"forward": 1, "fo_fwd": 1, "fo_bwd": 1}.get(kind, 2 if c["snap"] else 4)
    if nt * runs * (1.8e-3 + 2.5e-9 * n * X * Z) > 20:       # seconds of the loops below
        return None
    if kind == "survey":                                     # one grid per shot
        return None
    d = _inputs(c, seed)
    vp, vs = _pad64(d["vp"], L, dev), _pad64(d["vs"], L, dev)
    flip = (lambda g: g if c["tx"] else g.transpose(-1, -2))
    if kind == "forward":
        sim = Sim64(vp, vs, _pad64(d["rho"], L, dev) if c["density"] else None, c, dev)
        now, _, gx, gz = _forward64(c, sim, d["shots"], d["w"])
        f = torch.cat([now[0] + now[2], now[1] + now[3], *now]) if c["fields"] else None
        return {"gx": flip(gx[0]).contiguous(), "gz": flip(gz[0]).contiguous(), "fields": f}
    if kind in ("fo_fwd", "fo_bwd"):
        rec = d["recs"][0] if kind == "fo_bwd" else None
        gx, gz, f = _first_order64(c, vp, vs, d["shots"][0], d["w"], rec, dev)
        return {"fields": f} if rec is not None else {"gx": flip(gx).contiguous(), "gz": flip(gz).contiguous(), "fields": f}
    rho = _pad64(d["rho"], L, dev) if kind == "gradient" else None
    il, grad = _rtm64(c, vp, vs, rho, d["shots"], d["w"], d["recs"], dev)
    # Images are quotients of sums that are round-off-sized in badly lit corners
    # (and, without snapshots, of a backward reconstruction that amplifies
    # round-off): 32-bit ones are percents off these, whoever computes them,
    # so only the illumination and the gradient are given.
    out = {"images": [(None, None)] * n, "stack": (None, None, il.sum(0))}
    if grad is not None:
        out["gradient"] = tuple(g[:, L:-L, L:-L].sum(0) for g in grad)
    return out
