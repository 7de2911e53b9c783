"""The engine's work as its users run it: what is timed, on which inputs, and
what the results are in 64 bits.

Every case goes through a public entry point of ``seis_b200``: the single-shot
calls of ``fd`` (host arrays in, host arrays out), the one-call ``batch``, a
``Plan`` kept across calls, the ``Lsrtm`` solver and the vector operations.
Models are seeded layers with Gaussian anomalies over a smooth background,
wavelets Ricker with a delay of 1.5 periods, gathers sums of hyperbolic
events; the Courant number stays at 0.3 or below, where the scheme's absorbing
boundary is stable.  The step counts of the batched and the large cases are
cut so that one pass takes a fraction of a second: every step costs the same.
"""
import math

import numpy as np
import torch

from seis_b200 import _lib as S
from seis_b200 import fd

_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = S.Context(0)
    return _ctx


def listed():
    return [
        # the smallest call: a test-size shot, where latency and launches count
        dict(name="modeling_small", op="modeling", nx=96, nz=64, pml=12, nt=200, fr=30.0,
             dt=1e-3, dx=10.0),
        # one shot of the 201 x 201 configuration in full: the plain single-shot call
        dict(name="modeling_201", op="modeling", nx=201, nz=201, pml=40, nt=2000, fr=15.0,
             dt=1e-3, dx=10.0),
        # Born of one shot of the 737 x 240 model in full
        dict(name="born_737", op="born", nx=737, nz=240, pml=40, nt=4000, fr=20.0, dt=1e-3,
             dx=12.5),
        # reference RTM of the same shot in full (source pass, reconstruction, receiver
        # field, imaging every step)
        dict(name="rtm_737", op="rtm", nx=737, nz=240, pml=40, nt=4000, fr=20.0, dt=1e-3,
             dx=12.5),
        # source illumination of a survey's shots of uneven aperture in one call
        dict(name="illum_batch", op="illum_batch", nx=737, nz=240, pml=40, nt=500, fr=20.0,
             dt=1e-3, dx=12.5, shots=16, nmin=300),
        # modeling of several full-aperture shots on a kept plan, a new velocity every call
        dict(name="modeling_plan_1200", op="modeling_plan", nx=1200, nz=400, pml=40, nt=500,
             fr=20.0, dt=8e-4, dx=10.0, shots=8, nmin=1200, exact=True),
        # the batched RTM survey (uneven apertures) on a kept plan, new gathers every call
        dict(name="rtm_plan_737", op="rtm_plan", nx=737, nz=240, pml=40, nt=500, fr=20.0,
             dt=1e-3, dx=12.5, shots=16, nmin=300),
        # Born of the largest survey's shots, the forward half of its LSRTM iteration
        dict(name="born_plan_4000", op="born_plan", nx=4000, nz=1000, pml=40, nt=200, fr=25.0,
             dt=5e-4, dx=5.0, shots=8, nmin=1000, exact=False),
        # exact adjoint with FP32 snapshots of every step (the operator of the dot-product
        # test), new gathers every call
        dict(name="adjoint_plan_1200", op="adjoint_plan", nx=1200, nz=400, pml=40, nt=400,
             fr=20.0, dt=8e-4, dx=10.0, shots=4, nmin=1200, every=1, dtype="f32", ckpt=0),
        # the other half of the largest survey's iteration: FP16 snapshots every 4 steps,
        # recomputed from source-field checkpoints
        dict(name="adjoint_plan_4000", op="adjoint_plan", nx=4000, nz=1000, pml=40, nt=200,
             fr=25.0, dt=5e-4, dx=5.0, shots=6, nmin=1000, every=4, dtype="f16", ckpt=128),
        # a whole solver call: reset and one CG iteration of LSRTM, model and residuals out
        dict(name="lsrtm_1200", op="lsrtm", nx=1200, nz=400, pml=40, nt=400, fr=20.0, dt=8e-4,
             dx=10.0, shots=8, nmin=1200, every=4, dtype="f16", ckpt=0),
        # the solver's vector operations on a model of the largest survey
        dict(name="vec_4000x1000", op="vec", n=4000 * 1000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["modeling", "born", "rtm", "illum_batch", "modeling_plan", "rtm_plan",
                     "born_plan", "adjoint_plan", "lsrtm", "vec"])
    if op == "vec":
        return dict(op=op, n=_log(rng, 6000, 4000000))
    c = dict(op=op, pml=rng.choice([12, 20, 30, 40]))
    if op in ("modeling", "born", "rtm"):
        c.update(nx=_log(rng, 96, 737), nz=rng.randint(64, 240), nt=_log(rng, 200, 2000))
    else:
        big = op in ("born_plan", "adjoint_plan") and rng.random() < 0.4
        nx = _log(rng, 1200, 3600) if big else _log(rng, 300, 1200)
        c.update(nx=nx, nz=rng.randint(400, 1000) if big else rng.randint(150, 400),
                 nt=rng.randint(100, 200) if big else _log(rng, 100, 400),
                 shots=rng.randint(1, 5 if big else 8), nmin=max(100, nx // 3))
    c.update(fr=rng.choice([15.0, 20.0, 25.0, 30.0]), dx=rng.choice([5.0, 10.0, 12.5]))
    c["dt"] = round(0.3 * c["dx"] / 4500.0, 7)  # a Courant number of 0.3 at 4500 m/s
    c["fr"] = max(c["fr"], round(1.5 / (200 * c["dt"]), 1))  # at most 200 steps of delay
    if op in ("modeling_plan", "born_plan"):
        c["exact"] = rng.random() < 0.5
    if op in ("adjoint_plan", "lsrtm"):
        c["every"] = rng.choice([1, 2, 4])
        c["dtype"] = rng.choice(["f32", "bf16", "f16"])
        c["ckpt"] = rng.choice([0, 0, 64, 128])
    return c


# ------------------------------------------------------------------ inputs
def _ndel(c):
    return int(math.ceil(1.5 / (c["fr"] * c["dt"]) - 1e-9))


def _wavelet(c):
    """Ricker wavelet of NT samples, delayed by 1.5 periods."""
    t = (np.arange(c["nt"] + _ndel(c)) - _ndel(c)) * c["dt"]
    a = (math.pi * c["fr"] * t) ** 2
    return ((1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _models(c, gen):
    """(background, perturbation) [nx][nz] float32 on the GPU: layers with
    anomalies, 1500 m/s up to a Courant number of 0.3, and their smooth part."""
    nx, nz, dev = c["nx"], c["nz"], "cuda"
    vmax = min(4500.0, 0.3 * c["dx"] / c["dt"])
    nlay = 20
    vals = torch.sort(torch.rand(nlay, generator=gen, device=dev))[0] * (vmax - 1500.0) + 1500.0
    lay = (torch.arange(nz, device=dev) * nlay // nz).clamp(max=nlay - 1)
    v = vals[lay][None, :].repeat(nx, 1)
    X = torch.arange(nx, device=dev, dtype=torch.float32)[:, None]
    Z = torch.arange(nz, device=dev, dtype=torch.float32)[None, :]
    for a in torch.rand(10, 4, generator=gen, device=dev).tolist():
        r = 5.0 + 15.0 * a[2]
        v = v + math.copysign(300.0, a[3] - 0.5) * torch.exp(
            -((X - a[0] * nx) ** 2 + (Z - a[1] * nz) ** 2) / (2.0 * r * r))
    v = v.clamp(1500.0, vmax)
    k = 21
    p = torch.nn.functional.pad(v[None, None], (k // 2,) * 4, mode="replicate")
    v0 = torch.nn.functional.avg_pool2d(p, k, stride=1)[0, 0]
    return v0.contiguous(), (v - v0).contiguous()


def _gather(c, s, gen):
    """Hyperbolic events around the source and some noise, [nx][nt] on the GPU."""
    nt, dt, dev = c["nt"], c["dt"], "cuda"
    t = torch.arange(nt, device=dev, dtype=torch.float32)[None, :] * dt
    x = (torch.arange(s.nx, device=dev, dtype=torch.float32) - s.sx)[:, None] * c["dx"]
    out = 0.05 * torch.randn(s.nx, nt, generator=gen, device=dev)
    for a in torch.rand(6, 3, generator=gen, device=dev).tolist():
        t0 = (0.1 + 0.8 * a[0]) * nt * dt
        q = (math.pi * c["fr"] * (t - torch.sqrt(t0 * t0 + (x / (1800.0 + 2000.0 * a[1])) ** 2))) ** 2
        out += (0.5 + a[2]) * (1.0 - 2.0 * q) * torch.exp(-q)
    return out


def _shots(c):
    """[(first column, width)] of the survey's apertures (its geometry: the same
    for every seed)."""
    n, nmin = c.get("shots", 1), c.get("nmin", c["nx"])
    out = []
    for a, b in np.random.default_rng(3).random((n, 2)):
        w = nmin + int(a * (c["nx"] - nmin + 0.999))
        out.append((int(b * (c["nx"] - w + 0.999)), w))
    return out


def _shot(c, nx, k, n):
    sx = int((k + 0.5) * nx / n) if n > 1 else nx // 2
    return S.Shot(nx=nx, nz=c["nz"], pml=c["pml"], nt=c["nt"], ndel=_ndel(c), sx=sx, sz=2,
                  dt=c["dt"], dx=c["dx"], dz=c["dx"], gz=np.full(nx, 2, np.int32))


def _inputs(c, seed):
    """Everything a case's inputs are made of, the same for prepare and exact."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    if c["op"] == "vec":
        a, b, x, y = (torch.randn(c["n"], generator=gen, device="cuda") for _ in range(4))
        return dict(a=a, b=b, x=x, y=y)
    v0, dv = _models(c, gen)
    ap = _shots(c)
    d = dict(v0=v0, dv=dv, wav=_wavelet(c), ap=ap,
             shots=[_shot(c, w, k, len(ap)) for k, (_, w) in enumerate(ap)])
    if c["op"] in ("rtm", "rtm_plan", "adjoint_plan", "lsrtm"):
        d["rec"] = [_gather(c, s, gen) for s in d["shots"]]
    d["vel"] = [v0[x:x + w].contiguous() for x, w in ap]
    d["dvs"] = [dv[x:x + w].contiguous() for x, w in ap]
    return d


_SNAP = {"f32": S.SNAP_F32, "bf16": S.SNAP_BF16, "f16": S.SNAP_F16}


def prepare(case, seed):
    c, ctx = case, _context()
    d = _inputs(c, seed)
    op = c["op"]
    st = dict(case=c, op=op, ctx=ctx)
    if op == "vec":
        st.update(d)
        return st
    sh = d["shots"]
    if op in ("modeling", "born", "rtm", "illum_batch"):
        st.update(shots=sh, wav=d["wav"], vel=[v.cpu().numpy() for v in d["vel"]])
        if op == "born":
            st["dv"] = d["dvs"][0].cpu().numpy()
        if op == "rtm":
            st["rec"] = d["rec"][0].cpu().numpy()
        return st
    if op == "lsrtm":
        L = S.Lsrtm(ctx, c["nx"], c["nz"], sh, x0=[x for x, _ in d["ap"]], snap_every=c["every"],
                    snap_dtype=_SNAP[c["dtype"]], checkpoint_every=c["ckpt"])
        L.set_background(d["v0"].cpu().numpy(), d["wav"])
        for k, r in enumerate(d["rec"]):
            L.set_data(k, r.cpu().numpy())
        st["solver"] = L
        return st
    kind = {"modeling_plan": S.OP_MODELING, "rtm_plan": S.OP_RTM, "born_plan": S.OP_BORN,
            "adjoint_plan": S.OP_BORN_ADJOINT}[op]
    p = S.Plan(ctx, kind, sh)
    if op in ("modeling_plan", "born_plan"):
        p.set_exact(c["exact"])
    if op == "adjoint_plan":
        p.set_snapshots(c["every"], _SNAP[c["dtype"]])
        if c["ckpt"]:
            p.set_checkpoints(c["ckpt"])
    for k in range(len(sh)):
        p.set(k, S.IN_WAVELET, d["wav"])
        if op != "modeling_plan":
            p.set_device(k, S.IN_VEL, d["vel"][k].data_ptr())
    p.sync()
    st["plan"] = p
    # the inputs that change from call to call, on the GPU
    what, arrs = {"modeling_plan": (S.IN_VEL, d["vel"]), "born_plan": (S.IN_DV, d["dvs"])}.get(
        op, (S.IN_GATHER, d.get("rec")))
    st.update(what=what, arrays=arrs,
              out=S.OUT_GATHER if op in ("modeling_plan", "born_plan") else S.OUT_IMAGE)
    return st


def run(state):
    op, ctx = state["op"], state["ctx"]
    if op == "vec":
        n = state["a"].numel()
        dot = S.vec_dot(ctx, state["a"].data_ptr(), state["b"].data_ptr(), n)
        S.vec_axpby(ctx, state["y"].data_ptr(), state["x"].data_ptr(), 0.75, 0.5, n)
        return dict(dot=dot, y=state["y"])
    if op == "lsrtm":
        L = state["solver"]
        r0 = L.reset()
        r1 = L.iterate(1)
        return dict(rr=np.array([r0, r1[0]]), model=L.model())
    if op in ("modeling", "born", "rtm"):
        s = state["shots"][0]
        a = (s.dt, s.dx, s.dz, s.nt, s.ndel, s.nx, s.nz, s.pml, s.sx, s.sz, s.gz, state["wav"],
             state["vel"][0])
        if op == "modeling":
            return fd.modeling(*a, ctx=ctx)
        if op == "born":
            return fd.forward(*a, state["dv"], ctx=ctx)
        return fd.adjoint(*a, state["rec"], ctx=ctx)
    if op == "illum_batch":
        return S.batch(ctx, S.OP_ILLUM, state["shots"], [state["wav"]] * len(state["shots"]),
                       state["vel"])
    p = state["plan"]
    for k, a in enumerate(state["arrays"]):
        p.set_device(k, state["what"], a.data_ptr())
    p.run()
    return [p.get(k, state["out"]) for k in range(len(state["arrays"]))]


# -------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once; the arithmetic of the time
    steps: per padded cell and field, the two 8th-order second differences (34
    operations) and their combination (8)."""
    c = case
    if c["op"] == "vec":
        return {"bytes": 4.0 * c["n"] * 5, "flops": 5.0 * c["n"]}
    n, nmin, NT = c.get("shots", 1), c.get("nmin", c["nx"]), c["nt"] + _ndel(c)
    nx = 0.5 * (nmin + c["nx"])  # the mean aperture of the survey
    cells = n * (nx + 2 * c["pml"]) * (c["nz"] + 2 * c["pml"])
    model, data = n * nx * c["nz"], n * nx * c["nt"]
    op = c["op"].replace("_plan", "").replace("_batch", "")
    ck = 1 if c.get("ckpt") else 0
    # field steps, input and output words, further operations per model cell
    steps, words, more = {
        "modeling": (NT, model + data, 0),
        "born": (2 * NT, 2 * model + data, 8 * NT),
        "rtm": (NT + 2 * c["nt"], 2 * model + data, 130 * c["nt"]),
        "illum": (NT, 2 * model, 2 * NT),
        # the source field of a fixed background is kept (or recomputed from checkpoints)
        "adjoint": ((1 + ck) * NT, 2 * model + data, 4 * NT // c.get("every", 1)),
        "lsrtm": ((4 + 2 * ck) * NT, 3 * model + 4 * data,
                  8 * NT + 8 * NT // c.get("every", 1)),
    }[op]
    return {"bytes": 4.0 * words, "flops": 42.0 * cells * steps + more * model}


# ----------------------------------------------------------- 64-bit results
class _Grid:
    """The time step of one shot in 64 bits: a leapfrog update (8th order in
    space, 2nd order in the three rings along the edge, an extrapolated frame)
    blended on the pad with a one-way update toward the edge."""

    def __init__(self, c, vel):
        f = lambda v: float(np.float32(v))  # noqa: E731
        self.dt, self.dx, pml = f(c["dt"]), f(c["dx"]), c["pml"]
        dt, dx = self.dt, self.dx
        self.pml, (self.nx, self.nz) = pml, vel.shape
        v = torch.nn.functional.pad(vel.double()[None, None], (pml,) * 4, mode="replicate")[0, 0]
        self.v, self.NX, self.NZ = v, *v.shape
        self.vt2 = (v * dt) ** 2
        self.cof = self.vt2 / (dx * dx)
        self.vel3 = 2.0 / v ** 3
        self.m = (slice(pml, pml + self.nx), slice(pml, pml + self.nz))
        NX, NZ, dev = self.NX, self.NZ, v.device
        X = torch.arange(NX, device=dev)[:, None].expand(NX, NZ)
        Z = torch.arange(NZ, device=dev)[None, :].expand(NX, NZ)
        dl, dr = pml - X, X - (pml + self.nx - 1)
        du, dd = pml - Z, Z - (pml + self.nz - 1)
        distx, distz = torch.maximum(dl, dr).clamp(min=0), torch.maximum(du, dd).clamp(min=0)
        ring = torch.maximum(distx, distz)
        sx = torch.where(dl > 0, 1, torch.where(dr > 0, -1, 0))
        sz = torch.where(du > 0, 1, torch.where(dd > 0, -1, 0))
        flat = (X * NZ + Z).reshape(-1)
        strip = ((ring > 0) & (distx != distz)).reshape(-1)
        corner = ((ring > 0) & (distx == distz)).reshape(-1)
        vert = (distz > distx).reshape(-1)  # top or bottom strip: one-way along z
        w = 1.0 - torch.where(distx > 0, distx, distz).double() / max(pml, 1)
        w = w.reshape(-1)
        inner = torch.where(vert, sz.reshape(-1), sx.reshape(-1) * NZ)
        along = torch.where(vert, NZ, 1)
        self.S, self.C = flat[strip], flat[corner]
        self.Si, self.St = (flat + inner)[strip], along[strip]
        vs = v.reshape(-1)[self.S]
        a1, a2, a3 = 1.0 / dx / 2.0 / dt, 1.0 / 2.0 / dt / dt / vs, vs / 4.0 / dx / dx
        d = a1 + a2
        self.al, self.be, self.ga = (a1 - a2 - 2.0 * a3) / d, a3 / d, 2.0 * a2 / d
        self.ws = w[self.S]
        self.Cz = self.C + sz.reshape(-1)[self.C]
        self.Cx = self.C + NZ * sx.reshape(-1)[self.C]
        k3 = math.sqrt(2.0) / v.reshape(-1)[self.C] / dt
        self.c1, self.c3 = (1.0 / dx) / (2.0 / dx + k3), k3 / (2.0 / dx + k3)
        self.wc = w[self.C]

    def zeros(self):
        return torch.zeros_like(self.v)

    def twoway(self, c, p):
        """2 c - p + (v dt)^2 lap c, and the frame."""
        T = [-1.0 / 560, 8.0 / 315, -0.2, 1.6, -205.0 / 72]
        k = self.cof
        u = 2.0 * c - p
        lo = c[1:-1, :-2] + c[1:-1, 2:] + c[:-2, 1:-1] + c[2:, 1:-1] - 4.0 * c[1:-1, 1:-1]
        n, m = self.NX - 8, self.NZ - 8
        if n > 0 and m > 0:
            i = c[4:-4, 4:-4]
            hi = 2.0 * T[4] * i
            for o in range(1, 5):
                t = T[4 - o]
                hi = hi + t * (c[4 - o:4 - o + n, 4:-4] + c[4 + o:4 + o + n, 4:-4]
                               + c[4:-4, 4 - o:4 - o + m] + c[4:-4, 4 + o:4 + o + m])
            lo = lo.clone()
            lo[3:-3, 3:-3] = hi
        u[1:-1, 1:-1] = u[1:-1, 1:-1] + k[1:-1, 1:-1] * lo
        d = lambda q, a, b, e: q * (a + e - 2.0 * b)  # noqa: E731
        # along the edge rows and columns
        u[1:-1, 0] = u[1:-1, 0] + d(k[1:-1, 0], c[:-2, 0], c[1:-1, 0], c[2:, 0])
        u[1:-1, -1] = u[1:-1, -1] + d(k[1:-1, -1], c[:-2, -1], c[1:-1, -1], c[2:, -1])
        u[0, 1:-1] = u[0, 1:-1] + d(k[0, 1:-1], c[0, :-2], c[0, 1:-1], c[0, 2:])
        u[-1, 1:-1] = u[-1, 1:-1] + d(k[-1, 1:-1], c[-1, :-2], c[-1, 1:-1], c[-1, 2:])
        # across them, extrapolated from inside
        u[:, 0] = u[:, 0] + 2.0 * d(k[:, 1], c[:, 0], c[:, 1], c[:, 2]) - d(k[:, 2], c[:, 1], c[:, 2], c[:, 3])
        u[:, -1] = u[:, -1] + 2.0 * d(k[:, -2], c[:, -1], c[:, -2], c[:, -3]) - d(k[:, -3], c[:, -2], c[:, -3], c[:, -4])
        u[0] = u[0] + 2.0 * d(k[1], c[0], c[1], c[2]) - d(k[2], c[1], c[2], c[3])
        u[-1] = u[-1] + 2.0 * d(k[-2], c[-1], c[-2], c[-3]) - d(k[-3], c[-2], c[-3], c[-4])
        return u

    def absorb(self, u, c, p):
        u, c, p = u.reshape(-1), c.reshape(-1), p.reshape(-1)
        s, i, t = self.S, self.Si, self.St
        one = (self.al * (u[i] + p[s]) + self.be * (u[i + t] + u[i - t] + p[s + t] + p[s - t])
               + self.ga * (c[s] + c[i]) - p[i])
        cor = self.c1 * (u[self.Cz] + u[self.Cx]) + self.c3 * c[self.C]
        o = u.clone()
        o[s] = self.ws * u[s] + (1.0 - self.ws) * one
        o[self.C] = self.wc * u[self.C] + (1.0 - self.wc) * cor
        return o.reshape(self.NX, self.NZ)


def _src(g, s):
    return s.sx + g.pml, s.sz + g.pml


def _rows(g, s, dev):
    return torch.arange(g.nx, device=dev) + g.pml, torch.as_tensor(s.gz, device=dev).long() + g.pml


def _forward64(c, vel, s, wav, dv=None, keep=None):
    """Gather [nx][nt] (of the scattered field when dv is given); keep: called
    with (step, previous, current, new field)."""
    g = _Grid(c, vel)
    a = [g.zeros(), g.zeros()]
    b = [g.zeros(), g.zeros()]
    w = wav.astype(np.float64)
    rx, rz = _rows(g, s, vel.device)
    rec = torch.zeros(g.nx, s.nt, dtype=torch.float64, device=vel.device)
    q = None if dv is None else (g.vt2 * g.vel3)[g.m] * dv.double()
    ix, iz = _src(g, s)
    for it in range(s.NT):
        u = g.twoway(a[1], a[0])
        if it >= 1:
            u[ix, iz] += g.vt2[ix, iz] * float(w[it - 1])
        new = g.absorb(u, a[1], a[0])
        out = new
        if dv is not None:
            ub = g.twoway(b[1], b[0])
            lap = (new + a[0] - 2.0 * a[1])[g.m] / (g.dt * g.dt)
            ub[g.m] += q * lap
            out = g.absorb(ub, b[1], b[0])
            b = [b[1], out]
        if it >= s.ndel:
            rec[:, it - s.ndel] = out[rx, rz]
        if keep is not None:
            keep(g, it, a[0], a[1], new)
        a = [a[1], new]
    return rec


def _hilbert64(n, dev):
    """Matrix of the 61-tap Hamming-tapered Hilbert filter over n samples."""
    H = torch.zeros(n, n, dtype=torch.float64)
    i = np.arange(n)
    for k in range(1, 31, 2):
        t = (0.54 + 0.46 * math.cos(3.1415926 * k / 30)) * 2.0 / (3.1415926 * k)
        if k < n:
            H[i[k:] - k, i[k:]] = t  # out[j] = sum_i in[i] h[j - i]
            H[i[k:], i[k:] - k] = -t
    return H.to(dev)


def _rtm64(c, vel, s, wav, rec):
    """Image of the reference RTM: the source field rebuilt backwards from its
    four boundary layers, the receiver field beside it, correlated and
    filtered with the Hilbert term every step."""
    layers = []

    def edge(g, x):
        m = x[g.m]
        return [t.clone() for t in (m[:, :4], m[:, -4:], m[:4], m[-4:])]

    def keep(g, it, p, cu, n):
        if it >= s.ndel:
            layers.append(edge(g, n))

    _forward64(c, vel, s, wav, keep=keep)
    g = _Grid(c, vel)
    H = _hilbert64(g.NZ, vel.device)
    a, b = [g.zeros(), g.zeros()], [g.zeros(), g.zeros()]
    img = torch.zeros(g.nx, g.nz, dtype=torch.float64, device=vel.device)
    rx, rz = _rows(g, s, vel.device)
    r64 = rec.double()
    ix, iz = _src(g, s)
    w = wav.astype(np.float64)
    for it in range(s.NT - 1, s.ndel - 1, -1):
        if it - 1 > 0:
            a[0][ix, iz] -= g.vt2[ix, iz] * float(w[it - 1])
        m = a[1][g.m]
        top, bot, lef, rig = layers[it - s.ndel]
        m[:, :4], m[:, -4:], m[:4], m[-4:] = top, bot, lef, rig
        na = g.absorb(g.twoway(a[1], a[0]), a[1], a[0])
        u = g.twoway(b[1], b[0])
        u[rx, rz] += r64[:, it - s.ndel] * g.vt2[rx, rz]
        nb = g.absorb(u, b[1], b[0])
        U = ((a[0] + na - 2.0 * a[1]) / (g.dt * g.dt) * g.vel3)[g.pml:g.pml + g.nx]
        R = nb[g.pml:g.pml + g.nx]
        z = g.m[1]
        img += 1.5 * (U * R)[:, z] - 0.5 * ((U @ H) * (R @ H))[:, z]
        a, b = [a[1], na], [b[1], nb]
    return img


def _illum64(c, vel, s, wav):
    out = torch.zeros(vel.shape, dtype=torch.float64, device=vel.device)

    def keep(g, it, p, cu, n):
        if it > s.ndel:
            out.add_(n[g.m] ** 2)

    _forward64(c, vel, s, wav, keep=keep)
    return out


def _weights(NT, every):
    """Steps whose source term is imaged and their trapezoid weights."""
    K = NT - 1
    t = sorted(set(range(0, K + 1, every)) | {K})
    w = {}
    for j, k in enumerate(t):
        lo = t[j - 1] if j else k
        hi = t[j + 1] if j + 1 < len(t) else k
        w[k] = 0.5 * (hi - lo + (j == 0) + (j + 1 == len(t)))
    return {k: 1.0 for k in t} if every == 1 else w


def _source64(c, vel, s, wav):
    laps = {}
    wt = _weights(s.NT, c["every"])

    def keep(g, it, p, cu, n):
        if it in wt:
            laps[it] = (n + p - 2.0 * cu)[g.m] / (g.dt * g.dt)

    _forward64(c, vel, s, wav, keep=keep)
    return laps


def _adjoint64(c, vel, s, laps, rec):
    """Transpose of the Born operator, one reverse step as the vector-Jacobian
    product of the (linear) forward step."""
    g = _Grid(c, vel)
    wt = _weights(s.NT, c["every"])
    rx, rz = _rows(g, s, vel.device)
    r64 = rec.double()
    with torch.enable_grad():  # the step is linear: its graph at zero serves every step
        cu, p, q = (g.zeros().requires_grad_() for _ in range(3))
        new = g.absorb(g.twoway(cu, p) + q, cu, p)
    grad = torch.zeros(g.nx, g.nz, dtype=torch.float64, device=vel.device)
    ln, lc = g.zeros(), g.zeros()  # cotangents of the new and of the current field
    for k in range(s.NT - 1, -1, -1):
        if k >= s.ndel:
            ln = ln.clone()
            ln[rx, rz] += r64[:, k - s.ndel]
        gc, gp, gq = torch.autograd.grad(new, (cu, p, q), grad_outputs=ln, retain_graph=True)
        if k in wt:
            grad += wt[k] * laps[k] * gq[g.m]
        ln, lc = lc + gc, gp
    return grad * (g.vt2 * g.vel3)[g.m]


def exact(case, seed):
    c = case
    d = _inputs(c, seed)
    op = c["op"]
    if op == "vec":
        a, b, x, y = (d[k].double() for k in "abxy")
        # the product is the operation's FP32 one, the sum is in FP64
        return dict(dot=float((a * b).sum()), y=0.75 * x + 0.5 * y)
    sh, vel, wav = d["shots"], d["vel"], d["wav"]
    n = range(len(sh))
    with torch.no_grad():
        if op in ("modeling", "modeling_plan"):
            out = [_forward64(c, vel[k], sh[k], wav) for k in n]
        elif op in ("born", "born_plan"):
            out = [_forward64(c, vel[k], sh[k], wav, d["dvs"][k]) for k in n]
        elif op in ("rtm", "rtm_plan"):
            out = [_rtm64(c, vel[k], sh[k], wav, d["rec"][k]) for k in n]
        elif op == "illum_batch":
            out = [_illum64(c, vel[k], sh[k], wav) for k in n]
        elif op == "adjoint_plan":
            out = []
            for k in n:
                laps = _source64(c, vel[k], sh[k], wav)
                out.append(_adjoint64(c, vel[k], sh[k], laps, d["rec"][k]))
        else:
            return _lsrtm64(c, d)
    return out[0] if op in ("modeling", "born", "rtm") else out


def _lsrtm64(c, d):
    """One iteration of CGLS from a zero model."""
    sh, vel, wav, ap = d["shots"], d["vel"], d["wav"], d["ap"]

    def back(rs):
        s = torch.zeros(c["nx"], c["nz"], dtype=torch.float64, device="cuda")
        for k, (x, w) in enumerate(ap):
            s[x:x + w] += _adjoint64(c, vel[k], sh[k], _source64(c, vel[k], sh[k], wav), rs[k])
        return s

    r = [t.double() for t in d["rec"]]
    s = back(r)
    q = [_forward64(c, vel[k], sh[k], wav, s[x:x + w]) for k, (x, w) in enumerate(ap)]
    alpha = float((s * s).sum()) / sum(float((t * t).sum()) for t in q)
    rr = [sum(float((t * t).sum()) for t in r),
          sum(float(((t - alpha * u) ** 2).sum()) for t, u in zip(r, q))]
    return dict(rr=np.array(rr), model=alpha * s)
