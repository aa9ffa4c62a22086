"""Workloads of the library, each one call (or a short sequence of calls) of
its public entry points as a user's program makes them, with the sizes such
programs use.

listed()              the standing cases, smallest to largest work
draw(rng)             one more case of the same ranges
prepare(case, seed)   inputs on the GPU, and the plan or codec a program keeps
run(state)            one pass, outputs whole
work(case)            bytes and operations a pass cannot do without
exact(case, seed)     the outputs in 64-bit plain torch, without the library

What `work` counts: for 3D propagation, whose wavefields cannot stay on the
chip, every step's reads and writes of state and model once; for 2D
propagation, whose wavefields can, the model in and the results out, and the
operations of the updates.
"""
import math

import numpy as np
import torch

import geophysics_gb300 as geo

DEV = "cuda"
PI_GUI = 3.141592653          # the GUI and GPU programs' literal
PI_MPI = 3.1415926535898      # the MPI program's
C8 = [float(np.float32(c)) for c in (1.196289, -0.0797526, 0.009570313, -0.0006975447)]


def listed():
    return [
        # a quick look at a small model, GUI grid: launches and set-up count
        dict(name="fd2d_small", kind="fd2d", nx=101, nz=121, npd=20, nt=300, variant="gpu", sv=1),
        # forward modelling of one 2D shot with the CPU program's arithmetic
        dict(name="fd2d_401", kind="fd2d", nx=401, nz=401, npd=50, nt=2000, variant="cpu", sv=0),
        # one 2D shot over a whole line, the GPU program's arithmetic
        dict(name="fd2d_line", kind="fd2d", nx=2401, nz=601, npd=50, nt=500, variant="gpu", sv=1),
        # 2D TTI shot at the TTI program's own size
        dict(name="tti2d_600", kind="tti2d", nx=600, nz=300, npd=50, nt=801),
        # one shot of the 2D GPU RTM program with its angle gathers
        dict(name="rtm2d_gpu", kind="rtm2d_gpu", nx=1700, nz=601, npd=50, nt=600, tti=0, ns=1),
        # batched 2D RTM of shots with uneven aperture windows
        dict(name="rtm2d_batch", kind="rtm2d_batch", nx=2401, nz=601, npd=50, nt=500, ns=16, mode="exact", adcig=0),
        # an odd small 3D model, one call, the reference's arithmetic
        dict(name="fd3d_odd", kind="fd3d", nx=121, ny=93, nz=107, npd=20, nt=200, mode="exact", plan=0),
        # 3D modelling of repeated shots on one plan, fast form, 200 x 200 receivers
        dict(name="fd3d_400", kind="fd3d", nx=400, ny=400, nz=400, npd=40, nt=120, mode="fast", plan=1),
        # 3D TTI modelling on one plan
        dict(name="tti3d_300", kind="tti3d", nx=300, ny=300, nz=200, npd=40, nt=80),
        # 3D RTM of one shot with stored source snapshots
        dict(name="rtm3d", kind="rtm3d", nx=176, ny=160, nz=144, npd=20, nt=400, mode="fast", method="snapshot"),
        # encode and decode of one 3D snapshot
        dict(name="codec_snapshot", kind="codec", nx=512, ny=512, nz=384),
        # loss and gradients of one training batch of the codec
        dict(name="codec_grad", kind="codec_grad", nb=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fd2d", "fd2d", "tti2d", "rtm2d_gpu", "rtm2d_batch", "fd3d", "fd3d", "tti3d", "rtm3d", "codec",
                       "codec_grad"])
    if kind == "fd2d":
        nx, nz = _log(rng, 60, 2400), _log(rng, 60, 600)
        pts = (nx + 100) * (nz + 100)
        return dict(kind=kind, nx=nx, nz=nz, npd=rng.choice([20, 31, 50]), nt=min(2000, max(200, int(5e8 / pts))),
                    variant=rng.choice(["cpu", "gpu"]), sv=rng.choice([0, 1]))
    if kind == "tti2d":
        return dict(kind=kind, nx=_log(rng, 101, 1200), nz=_log(rng, 90, 500), npd=rng.choice([25, 50]),
                    nt=rng.randint(200, 800))
    if kind == "rtm2d_gpu":
        return dict(kind=kind, nx=_log(rng, 301, 1700), nz=_log(rng, 201, 601), npd=50, nt=rng.randint(400, 600),
                    tti=rng.choice([0, 1]), ns=1)
    if kind == "rtm2d_batch":
        return dict(kind=kind, nx=rng.randint(1601, 2401), nz=rng.randint(301, 601), npd=rng.choice([30, 50]),
                    nt=rng.randint(300, 500), ns=rng.randint(3, 16), mode=rng.choice(["exact", "exact", "fast"]),
                    adcig=rng.choice([0, 0, 1]))
    if kind == "fd3d":
        nx, ny, nz = (_log(rng, 60, 380) for _ in range(3))
        npd = rng.choice([16, 20, 40])
        pts = (nx + 2 * npd) * (ny + 2 * npd) * (nz + 2 * npd)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, npd=npd, nt=min(240, max(60, int(9e9 / pts))),
                    mode=rng.choice(["fast", "exact"]), plan=rng.choice([0, 1, 1]))
    if kind == "tti3d":
        nx, ny, nz = (_log(rng, 80, 300) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, npd=rng.choice([20, 40]), nt=rng.randint(40, 80))
    if kind == "rtm3d":
        nx, ny, nz = (_log(rng, 64, 160) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, npd=20, nt=rng.randint(260, 400),
                    mode=rng.choice(["fast", "exact"]), method=rng.choice(["boundary", "snapshot", "checkpoint"]))
    if kind == "codec":
        return dict(kind=kind, nx=_log(rng, 64, 512), ny=_log(rng, 64, 512), nz=_log(rng, 64, 384))
    return dict(kind=kind, nb=128 * rng.randint(1, 8))


# ------------------------------------------------------------------ inputs
def _field(shape, corr, g):
    """Gaussian random field of correlation `corr` cells, scaled to [0, 1]."""
    n = torch.randn(shape, generator=g, device=DEV)
    s, filt = corr / 2.0, 0.0
    for k, m in enumerate(shape):
        f = (torch.fft.rfftfreq if k == len(shape) - 1 else torch.fft.fftfreq)(m, device=DEV)
        filt = filt + f.reshape([-1 if q == k else 1 for q in range(len(shape))]) ** 2
    f = torch.fft.irfftn(torch.fft.rfftn(n) * torch.exp(-2 * math.pi ** 2 * s * s * filt), s=shape)
    return (f - f.min()) / (f.max() - f.min())


def _model(shape, g):
    """Velocity 2000-4000 m/s: a smooth random field plus four dipping
    interfaces, the shallow ones reflecting within a short run; eps and
    del <= eps follow it.  z last."""
    v = 2000 + 1400 * _field(shape, 40.0, g)
    nz = shape[-1]
    z = torch.arange(nz, device=DEV).float()
    x = torch.arange(shape[-2], device=DEV).float()[:, None] - shape[-2] / 2
    for k, (z0, a) in enumerate(((0.04, 0.002), (0.075, -0.002), (0.15, 0.01), (0.4, -0.03))):
        v = v + 150 * (z > z0 * nz + a * x + 3 * k).float()
    r = (v - 2000) / 2000
    return v.contiguous(), (0.3 * r).contiguous(), (0.15 * r).contiguous()


def _inputs(case, seed):
    """Everything drawn from the seed: the model, angles, volume or blocks."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + 17)
    k = case["kind"]
    if k in ("fd2d", "tti2d", "rtm2d_gpu", "rtm2d_batch"):
        shape = (case["nx"], case["nz"])
    elif k in ("codec", "fd3d", "tti3d", "rtm3d"):
        shape = (case["ny"], case["nx"], case["nz"])
    if k == "codec":
        # a band-limited wavefield: strong near the source, weak far from it
        f = _field(shape, 8.0, g) - 0.5
        return ((f * torch.exp(-6 * _field(shape, 80.0, g))).contiguous(),)
    if k == "codec_grad":
        b = torch.randn((case["nb"], 16, 16, 16), generator=g, device=DEV)
        b = torch.nn.functional.avg_pool3d(b[:, None], 5, stride=1, padding=2)[:, 0]
        return ((b * torch.exp(torch.randn((case["nb"], 1, 1, 1), generator=g, device=DEV)))
                .reshape(case["nb"], 4096).contiguous(),)
    m = _model(shape, g)
    if k == "tti2d" or case.get("tti"):
        m += ((5 + 40 * _field(shape, 60.0, g)).contiguous(),)
    if k == "tti3d":
        m += ((45 * _field(shape, 60.0, g)).contiguous(), (360 * _field(shape, 60.0, g)).contiguous())
    return m


def _kw(case):
    """The arguments of the case's call."""
    c, k = case, case["kind"]
    if k == "fd2d":
        return dict(npd=c["npd"], nt=c["nt"], dx=10.0, dz=10.0, dt=1e-3, favg=20.0, fs=c["nx"] // 2, zs=5,
                    variant=c["variant"], sv=c["sv"], rec_iz=c["npd"] + 4)
    if k == "tti2d":
        return dict(npd=c["npd"], nt=c["nt"], dx=5.0, dz=5.0, dt=5e-4, favg=40.0, fs=c["nx"] // 3, zs=c["nz"] // 2)
    if k == "rtm2d_gpu":
        return dict(npml=c["npd"], nt=c["nt"], dx=5.0, dz=5.0, dt=5e-4, favg=20.0, ns=c["ns"], fs=c["nx"] // 2, zs=1)
    if k == "rtm2d_batch":
        rng = np.random.default_rng(c["ns"])
        half = rng.integers(200, min(600, c["nx"] // 4), c["ns"])
        xs = np.round(np.linspace(c["nx"] // 4 + 1, c["nx"] - c["nx"] // 4, c["ns"])).astype(int)
        return dict(npd=c["npd"], nt=c["nt"], dx=10.0, dz=10.0, dt_ms=1.0, favg=20.0, pfac=10.0, zs=5,
                    shot_x=xs, shot_nxs=2 * half + 1, mode=c["mode"], adcig=bool(c["adcig"]))
    kw = dict(npd=c["npd"], nt=c["nt"], dx=10.0, dy=10.0, dz=10.0, dt=8e-4, favg=15.0, fsx=c["nx"] // 2,
              fsy=c["ny"] // 2, fsz=1)
    if k == "tti3d":
        return dict(kw, mode="fast")
    if k == "rtm3d":
        return dict(kw, mode=c["mode"], method=c["method"], snap_every=4, sv=1, illum=True)
    if c["plan"]:  # every second surface node records
        kw.update(drx=2, nrx=(c["nx"] + 1) // 2, dry=2, nry=(c["ny"] + 1) // 2)
    return dict(kw, mode=c["mode"], rec_iz=c["npd"])


def prepare(case, seed):
    st = dict(case=case, x=_inputs(case, seed), kw=None)
    k = case["kind"]
    if k in ("codec", "codec_grad"):
        st["codec"] = geo.Codec(seed=1)
        st["codec"].set_params(torch.cat([t.reshape(-1) for t in _codec_params(seed)]).cpu().numpy())
        return st
    st["kw"] = _kw(case)
    if k == "tti3d" or (k == "fd3d" and case["plan"]):
        plan = geo.FD3DPlan(nx=case["nx"], ny=case["ny"], nz=case["nz"], **st["kw"])
        plan.set_model(*st["x"][:3])
        if k == "tti3d":
            plan.set_tilt(*st["x"][3:])
        st["plan"] = plan
    return st


def run(st):
    case, x, kw = st["case"], st["x"], st["kw"]
    k = case["kind"]
    if k == "fd2d":
        return geo.fd2d_shot(*x, **kw)
    if k == "tti2d":
        return geo.tti2d_shot(*x, **kw)
    if k == "rtm2d_gpu":
        return (geo.rtm2d_tti if case["tti"] else geo.rtm2d_gpu)(*x, **kw)
    if k == "rtm2d_batch":
        return geo.rtm2d_batch(*x, **kw)
    if k == "rtm3d":
        return geo.rtm3d(*x, **kw)
    if k == "codec":
        return st["codec"].roundtrip(x[0])
    if k == "codec_grad":
        return st["codec"].eval(x[0], grad=True)
    if "plan" in st:
        return st["plan"].run_shot(0, device=DEV)
    return geo.fd3d_shot(*x, **kw)


def work(case):
    c, k = case, case["kind"]
    if k == "codec":
        n = c["nx"] * c["ny"] * c["nz"]
        return {"bytes": 8 * n, "flops": 2.0 * n / 4096 * _codec_macs()}
    if k == "codec_grad":
        p = sum(n * k + n for n, k, _, _ in _NET)
        return {"bytes": 4 * (2 * 4096 * c["nb"] + 2 * p), "flops": 6.0 * c["nb"] * _codec_macs()}
    pts = lambda n: n + 2 * c["npd"] - 8
    nt = c["nt"]
    if k in ("fd2d", "tti2d"):
        up = pts(c["nx"]) * pts(c["nz"]) * nt
        return {"bytes": 4 * ((3 if k == "fd2d" else 4) * c["nx"] * c["nz"] + nt * c["nx"]),
                "flops": float(up) * (69 if k == "fd2d" else 130)}
    if k == "rtm2d_gpu":
        up = 3 * pts(c["nx"]) * pts(c["nz"]) * nt * c["ns"]
        na = 65 if c["tti"] else 70
        return {"bytes": 4 * (c["nx"] * c["nz"] * (6 + na) + nt * c["nx"]), "flops": float(up) * (130 if c["tti"] else 69)}
    if k == "rtm2d_batch":
        w = _kw(c)["shot_nxs"]
        up = sum(3.0 * pts(int(a)) * pts(c["nz"]) * nt for a in w)
        return {"bytes": 4 * c["nx"] * c["nz"] * (4 + (90 if c["adcig"] else 0)), "flops": up * 69}
    box, tot = c["nx"] * c["ny"] * c["nz"], pts(c["nx"]) * pts(c["ny"]) * pts(c["nz"])
    if k == "tti3d":   # u,v,w,P,Q in and out, three model and four angle arrays
        return {"bytes": 68 * tot * nt, "flops": 190.0 * tot * nt}
    # u,v,w,P,Q in and out and three model arrays inside, the split parts in the sponge
    step = 52 * box + 84 * (tot - box)
    props = 1 if k == "fd3d" else {"boundary": 3, "snapshot": 2, "checkpoint": 3}[c["method"]]
    return {"bytes": step * props * nt, "flops": 100.0 * tot * props * nt}


# ------------------------------------------------- 64-bit plain evaluation
_NET = [(16, 8, 512, 1), (64, 128, 64, 1), (256, 512, 8, 1), (512, 2048, 1, 0),
        (2048, 512, 1, 1), (512, 256, 8, 1), (128, 64, 64, 1), (8, 16, 512, 0)]


def _codec_macs():
    return sum(n * k * r for n, k, r, _ in _NET)


def _codec_params(seed):
    """Weights as a program restores them: He-normal, small biases."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 3)
    out = []
    for n, k, _, act in _NET:
        out.append(torch.randn((n, k), generator=g, device=DEV) * math.sqrt((2.0 if act else 1.0) / k))
        out.append(torch.randn((n,), generator=g, device=DEV) * 0.02)
    return out


def _codec_net(wb, xn):
    """Normalised blocks (nb, 4096) -> reconstruction."""
    a = xn
    for l, (n, k, rows, act) in enumerate(_NET):
        a = a.reshape(-1, k) @ wb[2 * l].T + wb[2 * l + 1]
        if act:
            a = torch.nn.functional.leaky_relu(a, 0.1)
    return a.reshape(-1, 4096)


def _morton():
    m = np.arange(4096)
    z, x, y = (sum(((m >> (3 * l + s)) & 1) << l for l in range(4)) for s in range(3))
    return torch.from_numpy(z + 16 * x + 256 * y).to(DEV)


def _exact_codec(case, x, seed):
    wb = [t.double() for t in _codec_params(seed)]
    if case["kind"] == "codec_grad":
        b = x[0].double()
        xn = b / b.abs().amax(1, keepdim=True)
        for t in wb:
            t.requires_grad_(True)
        rec = _codec_net(wb, xn)
        loss = ((rec - xn) ** 2).mean()
        loss.backward()
        return rec.detach(), float(loss), torch.cat([t.grad.reshape(-1) for t in wb])
    v = x[0].double()
    ny, nx, nz = v.shape
    p = [-ny % 16, -nx % 16, -nz % 16]
    v = torch.nn.functional.pad(v, (0, p[2], 0, p[1], 0, p[0]))
    Y, X, Z = v.shape
    mo = _morton()
    out = torch.empty_like(v)
    for y in range(0, Y, 16):  # a slab of blocks at a time
        b = v[y:y + 16].reshape(16, X // 16, 16, Z // 16, 16).permute(1, 3, 0, 2, 4).reshape(-1, 4096)
        m = b[:, mo]
        s = m.abs().amax(1, keepdim=True)
        r = _codec_net(wb, m / torch.where(s > 0, s, torch.ones_like(s))) * s
        nat = torch.empty_like(r)
        nat[:, mo] = r
        out[y:y + 16] = nat.reshape(X // 16, Z // 16, 16, 16, 16).permute(2, 0, 3, 1, 4).reshape(16, X, Z)
    return out[:ny, :nx, :nz].contiguous()


def _pad(a, npd):
    return torch.nn.functional.pad(a[None, None].double(), (npd,) * (2 * a.dim()), mode="replicate")[0, 0].contiguous()


def _d(a, ax, nd, fwd):
    """8-tap staggered difference along spatial axis `ax` (negative), on the
    updated points: 4 cells in from every edge."""
    for k in range(1, nd + 1):
        if -k != ax:
            a = a.narrow(-k, 4, a.shape[-k] - 8)
    n = a.shape[ax] - 8
    r = None
    for m in range(4):
        t = a.narrow(ax, 4 + m + (1 if fwd else 0), n) - a.narrow(ax, 4 - m - (0 if fwd else 1), n)
        r = t.mul_(C8[m]) if r is None else r.add_(t, alpha=C8[m])
    return r


def _profiles(form, n, npd, dt, d0):
    """coff1, coff2, acoff1, acoff2 along one axis (form: cpu, gpu, mpi, ttirtm)."""
    f32 = np.float32
    out = np.ones((4, n + 2 * npd), np.float32)
    dd = float(f32(f32(dt) * f32(d0)))
    for i in list(range(npd)) + list(range(npd + n, n + 2 * npd)):
        if i < npd:
            qh, qi = (npd - 0.5 - i) / npd, (npd - i) / npd
        else:
            qh, qi = (0.5 + i - n - npd) / npd, (i - n - npd + (0 if form in ("gpu", "ttirtm") else 1)) / npd
        if form == "ttirtm":
            qh = qi
        h, a = dd * qh * qh / 2, dd * qi * qi / 2
        c1, a1 = f32(1 / (1 + h)), f32(1 / (1 + a))
        out[:, i] = (c1, f32(float(c1) * (1 - h)), a1, f32(float(c1 if form == "cpu" else a1) * (1 - a)))
    return torch.from_numpy(out).to(DEV).double()


def _amps(nt, dt, favg, pfac, mpi):
    """Ricker amplitude of each step, time a float advanced by additions."""
    f32 = np.float32
    pi = PI_MPI if mpi else PI_GUI
    dt, td = f32(dt), f32(1.0 / float(f32(favg)))
    t, out = (f32(0) if mpi else dt), []
    for _ in range(nt):
        if t <= f32(2) * td:
            x = f32(favg) * f32(t - td)
            xx = float(f32(x * x))
            out.append(float(f32(pfac) * f32((1 - 2 * pi * pi * xx) * math.exp(-(pi * pi * xx)))))
        else:
            out.append(None)
        t = f32(t + dt)
    return out


def _taper(arrs, centre, R, r, pi, cpu):
    """SV suppression: eps and del to zero around the source cell."""
    nd = arrs[0].dim()
    r2 = 0
    for k in range(nd):
        q = torch.arange(arrs[0].shape[k], device=DEV) - centre[k]
        r2 = r2 + (q * q).reshape([-1 if j == k else 1 for j in range(nd)])
    rad = r2.double().sqrt() if cpu else r2.float().sqrt().double()
    g = 0.5 * (1 - torch.cos(pi * ((rad - (R / 4.0 if cpu else r)) * 4.0 / (R * 3.0 - 1))))
    g = torch.where(r2 <= (R * R // 16 if cpu else r * r), torch.zeros_like(g), g)
    g = torch.where(r2 <= R * R, g, torch.ones_like(g))
    return [a * g for a in arrs]


class _Prop:
    """The time step in 64 bits: VTI with split sponge parts, or TTI with the
    product sponge; 2D (x, z) or 3D (y, x, z)."""

    def __init__(self, form, x, npd, h, dt, src=None, sv=None, tilt=None, lead=()):
        self.nd = nd = x[0].dim()
        self.form, self.npd = form, npd
        v, e, d = (_pad(a, npd) for a in x[:3])
        n = v.shape
        f32 = np.float32
        self.r = [float(f32(f32(dt) / f32(s))) for s in h]          # dt/h, axes outermost first
        if form in ("cpu", "mpi"):
            d0 = f32(3.0 * float(x[0].max()) * math.log(100000.0) / (2.0 * npd * float(f32(h[0]))))
        else:
            hm = sum(float(f32(s)) for s in h) / nd
            vc = float(v.reshape(-1)[v.numel() // 2])
            d0 = f32((3.0 if form == "ttirtm" else 10.0) * vc * math.log(100000.0) / (2.0 * npd * hm))
        self.prof = []
        for k in range(nd):
            p = _profiles(form, x[0].shape[k], npd, dt, d0)[:, 4:-4]
            self.prof.append([q.reshape([-1 if j == k else 1 for j in range(nd)]) for q in p])
        if sv:
            e, d = _taper([e, d], sv[0], sv[1], sv[2], PI_MPI if form == "mpi" else PI_GUI, form in ("cpu", "mpi"))
        I = tuple(slice(4, -4) for _ in range(nd))
        c2 = v[I] ** 2
        self.A, self.B, self.C = c2 * (1 + 2 * e[I]), c2 * torch.sqrt(1 + 2 * d[I]), c2
        self.tilt = None
        if tilt is not None:
            t = [_pad(a.double() * (math.pi / 180), npd)[I] for a in tilt]
            self.tilt = (torch.cos(t[0]), torch.sin(t[0])) + ((torch.cos(t[1]), torch.sin(t[1])) if nd == 3 else ())
        self.I = (Ellipsis,) + I
        self.src = src
        self.new_state(lead, n)

    def new_state(self, lead=(), n=None):
        n = n or self.P.shape[-self.nd:]
        z = lambda s: torch.zeros(tuple(lead) + tuple(s), device=DEV, dtype=torch.float64)
        self.P, self.Q = z(n), z(n)
        self.vel = [z(n) for _ in range(self.nd)]
        # the 2D TTI program's split pairs share their damping: one sum each
        parts = 2 * self.nd if self.tilt is None else 2 if self.nd == 2 else 0
        self.split = [z([k - 8 for k in n]) for _ in range(parts)]

    def step(self, amp=None):
        nd, I, r, pf = self.nd, self.I, self.r, self.prof
        gauss = self.form in ("cpu", "mpi")
        point = amp is not None and not gauss
        if point:   # reaches the velocities only
            keep = self.P[self.src].clone(), self.Q[self.src].clone()
            self.P[self.src] += amp
            self.Q[self.src] += amp
        P, Q = self.P, self.Q
        if self.tilt is None:
            for k in range(nd):
                g = _d(Q if k == nd - 1 else P, k - nd, nd, True)
                w = self.vel[k][I]
                w.mul_(pf[k][1]).sub_(g.mul_(pf[k][0] * r[k]))
            D = [_d(self.vel[k], k - nd, nd, False).mul_(r[k]) for k in range(nd)]
            S = self.split
            for k in range(nd):
                mp, mq = (self.B, self.C) if k == nd - 1 else (self.A, self.B)
                a1, a2 = pf[k][2], pf[k][3]
                S[k].mul_(a2).sub_(a1 * mp * D[k])
                S[nd + k].mul_(a2).sub_(a1 * mq * D[k])
            P[I] = sum(S[1:nd], S[0])
            Q[I] = sum(S[nd + 1:], S[nd])
        else:
            k1, k2, j1, j2 = pf[0]
            for q in pf[1:]:
                k1, k2, j1, j2 = k1 * q[0], k2 * q[1], j1 * q[2], j2 * q[3]
            f = lambda a, ax, fw: _d(a, ax, nd, fw).mul_(r[ax + nd])
            ct, st = self.tilt[:2]
            if nd == 2:
                g = [ct * f(P, -2, True) - st * f(P, -1, True), st * f(Q, -2, True) + ct * f(Q, -1, True)]
            else:
                cp, sp = self.tilt[2:]
                Px, Py, Pz = f(P, -2, True), f(P, -3, True), f(P, -1, True)
                # velocities stored as (v, u, w): axes y, x, z
                g = [cp * Py - sp * Px, ct * cp * Px + ct * sp * Py - st * Pz,
                     st * cp * f(Q, -2, True) + st * sp * f(Q, -3, True) + ct * f(Q, -1, True)]
            for w, gg in zip(self.vel, g):
                w[I] = k2 * w[I] - k1 * gg
            if nd == 2:
                u, w = self.vel
                a = ct * f(u, -2, False) - st * f(u, -1, False)
                b = st * f(w, -2, False) + ct * f(w, -1, False)
            else:
                vv, u, w = self.vel
                a = ct * cp * f(u, -2, False) + ct * sp * f(u, -3, False) - st * f(u, -1, False)
                a = a + cp * f(vv, -3, False) - sp * f(vv, -2, False)
                b = st * cp * f(w, -2, False) + st * sp * f(w, -3, False) + ct * f(w, -1, False)
            if point:
                P[self.src], Q[self.src] = keep
            p0, q0 = self.split or (P[I], Q[I])
            P[I] = j2 * p0 - j1 * (self.A * a + self.B * b)
            Q[I] = j2 * q0 - j1 * (self.B * a + self.C * b)
            if self.split:
                self.split = [P[I].clone(), Q[I].clone()]
        if gauss and amp is not None:
            k = torch.arange(-3, 4, device=DEV).double()
            s = amp * torch.exp(-k[:, None] ** 2 - k[None] ** 2)
            cx, cz = self.src[-2], self.src[-1]
            for F in (P, Q):
                F[..., cx - 3:cx + 4, cz - 3:cz + 4] += s


def _exact_shot(case, x, kw):
    npd, nt, nd = case["npd"], case["nt"], x[0].dim()
    form = kw.get("variant", "gpu")
    if nd == 2:
        src = (int(kw["fs"] + 0.5) + npd - 1, int(kw["zs"] + 0.5) + npd - 1)
        cen = src if form == "cpu" else (src[0] + 1, src[1] + 1)
        h = (kw["dx"], kw["dz"])
        sx, sy = slice(npd, npd + case["nx"]), None
    else:
        src = tuple(s + npd - 1 for s in (kw["fsy"], kw["fsx"], kw["fsz"]))
        cen, h = src, (kw["dy"], kw["dx"], kw["dz"])
        step = 2 if case.get("plan") else 1
        sy, sx = (slice(npd, npd + case[k], step) for k in ("ny", "nx"))
    sv = (cen, 15, 4) if kw.get("sv") else None
    p = _Prop(form, x, npd, h, kw["dt"], src, sv, x[3:] or None)
    scale = 2.0 if form == "cpu" else 1.0
    iz = kw.get("rec_iz", npd)
    rec = []
    for a in _amps(nt, kw["dt"], kw["favg"], 10.0, False):
        p.step(a)
        rec.append(scale * (p.P[sx, iz] if nd == 2 else p.P[sy, sx, iz]))
    return torch.stack(rec, -1)


def _mute(nx, nt, dt, favg, dx, dz, fs, zs, mu_v, tt, ms=None):
    """(first, end) of the muted samples of each trace of a surface record;
    ms: the step in milliseconds, for the program that divides by it."""
    f32 = np.float32
    dt, dx, dz = f32(dt), f32(dx), f32(dz)
    mx, mz = dx * np.abs(np.arange(nx) - fs).astype(np.float32), dz * f32(zs)
    t0 = np.sqrt((mx.astype(np.float64) ** 2 + float(mz) ** 2).astype(np.float32)) / f32(mu_v)
    i0 = (t0 / dt if ms is None else t0 / f32(ms) * f32(1000)).astype(np.int64)
    return i0 - tt + 1, i0 + int(2.0 / float(dt * f32(favg))) + tt


def _lap(a):
    """Adjoint first-difference Laplacian."""
    out = torch.zeros_like(a)
    for k in range(a.dim()):
        n = a.shape[k]
        f = a.narrow(k, 1, n - 1) - a.narrow(k, 0, n - 1)
        out.narrow(k, 1, n - 1).add_(f)
        out.narrow(k, 0, n - 1).sub_(f)
    return out


def _exact_rtm2d_gpu(case, x, kw):
    nx, nz, npd, nt = case["nx"], case["nz"], case["npd"], case["nt"]
    tti = bool(case["tti"])
    fs, zs = kw["fs"], kw["zs"]
    src = (fs + npd - 1, zs + npd - 1)
    R, r = (15, 4) if tti else (18, 7)
    tilt = x[3:] or None
    form = "ttirtm" if tti else "gpu"
    p = _Prop(form, x, npd, (kw["dx"], kw["dz"]), kw["dt"], src, ((fs + npd, zs + npd), R, r), tilt)
    b = _Prop(form, x, npd, (kw["dx"], kw["dz"]), kw["dt"], src, None, tilt)
    X, Z = slice(npd, npd + nx), slice(npd, npd + nz)
    ring = [(X, npd - 1), (X, npd + nz + 1), (npd - 1, Z), (npd + nx + 1, Z)]
    ill = torch.zeros((nx, nz), device=DEV, dtype=torch.float64)
    rec, saved = [], []
    tiny = 2.0 ** -150   # below this a 32-bit sum is zero
    for a in _amps(nt, kw["dt"], kw["favg"], 10.0, False):
        p.step(a)
        rec.append(p.P[X, npd].clone())
        saved.append([(p.P[q].clone(), p.Q[q].clone()) for q in ring])
        ill += p.P[X, Z] ** 2 + p.Q[X, Z] ** 2
        ill = torch.where(ill <= tiny, torch.ones_like(ill), ill)
    rec = torch.stack(rec, -1)
    v00, e00 = float(x[0][0, 0]), float(x[1][0, 0])
    mu_v = v00 * math.sqrt(1 + 2 * e00)
    if tti:
        mu_v = v00 * (1 + (math.sqrt(1 + 2 * e00) - 1) * math.cos(math.radians(float(x[3][0, 0]))))
    lo, hi = _mute(nx, nt, kw["dt"], kw["favg"], kw["dx"], kw["dz"], fs, zs, mu_v, 30 if tti else 20)
    flat = rec.reshape(-1)
    cap = nt if tti else (nt + 511) // 512 * 512   # the VTI program's launch covers samples past nt
    for ix in range(nx):
        flat[ix * nt + max(int(lo[ix]), 0):ix * nt + max(min(int(hi[ix]), cap), 0)] = 0
    # source and receiver fields together: index 0, 1 of a leading axis
    b.new_state((2,))
    b.P[0], b.Q[0] = p.P, p.Q
    for q, s in zip(b.vel, p.vel):
        q[0] = s
    for q, s in zip(b.split, p.split):
        q[0] = s
    mig = torch.zeros_like(ill)
    for it in range(nt - 1, -1, -1):
        for q, (sp, sq) in zip(ring, saved[it]):
            b.P[0][q], b.Q[0][q] = sp, sq
        b.P[1][X, npd] = rec[:, it]
        b.Q[1][X, npd] = rec[:, it]
        b.step()
        mig += b.P[0][X, Z] * b.P[1][X, Z]
    mig = mig / ill
    out = dict(mig_lap=_lap(mig), illum=ill, adcigs=None)   # gathers are binned: no 64-bit value
    if not tti:
        out["stk_lap"] = None
    out["shots"] = rec[None]
    return out


def _exact_rtm2d_batch(case, x, kw):
    nx, nz, npd, nt = case["nx"], case["nz"], case["npd"], case["nt"]
    dt = float(np.float32(kw["dt_ms"]) / np.float32(1000))
    zs, amps = kw["zs"], _amps(nt, dt, kw["favg"], kw["pfac"], True)
    full = torch.zeros((nx, nz), device=DEV, dtype=torch.float64)
    Z = slice(npd, npd + nz)
    for k, nxs in zip(kw["shot_x"], kw["shot_nxs"]):
        k, nxs = int(k), int(nxs)
        o = k - nxs // 2
        cols = torch.clamp(torch.arange(nxs, device=DEV) + o, max=nx - 1)
        w = [a[cols] for a in x]
        src = (nxs // 2 + npd, zs + npd - 1)
        X = slice(npd, npd + nxs)
        p = _Prop("mpi", w, npd, (kw["dx"], kw["dz"]), dt, src, (src, 15, 4))
        edge = [(X, npd), (X, npd + nz - 1), (npd, Z), (npd + nxs - 1, Z)]
        saved, rec = [], []
        for a in amps:
            p.step(a)
            saved.append([(p.P[q].clone(), p.Q[q].clone()) for q in edge])
            rec.append((saved[-1][0][0].clone(), saved[-1][0][1].clone()))
        mu_v = float(w[0][1, 1]) * math.sqrt(1 + 2 * float(w[1][1, 1]))
        _, hi = _mute(nxs, nt, dt, kw["favg"], kw["dx"], kw["dz"], nxs // 2 + 1, zs, mu_v, 285, kw["dt_ms"])
        keep = torch.from_numpy(np.arange(nt)[:, None] >= hi[None]).to(DEV).double()
        b = _Prop("mpi", w, npd, (kw["dx"], kw["dz"]), dt, src, None, None, (2,))
        mig = torch.zeros((nxs, nz), device=DEV, dtype=torch.float64)
        ill = torch.zeros_like(mig)
        for it in range(nt - 1, -1, -1):
            for q, (sp, sq) in zip(edge, saved[it]):
                b.P[0][q], b.Q[0][q] = sp, sq
            b.P[1][X, npd], b.Q[1][X, npd] = rec[it][0] * keep[it], rec[it][1] * keep[it]
            b.step()
            s = b.P[0][X, Z]
            ill += s * s
            ill = torch.where(ill <= 2.0 ** -150, torch.ones_like(ill), ill)
            mig += b.P[1][X, Z] * s
        full[o - 1:o - 1 + nxs] += mig / ill
    img = _lap(full)
    return (img, None) if case["adcig"] else img


def _exact_rtm3d(case, x, kw):
    nx, ny, nz, npd, nt = (case[k] for k in ("nx", "ny", "nz", "npd", "nt"))
    src = tuple(s + npd - 1 for s in (kw["fsy"], kw["fsx"], kw["fsz"]))
    p = _Prop("gpu", x, npd, (kw["dy"], kw["dx"], kw["dz"]), kw["dt"], src, (src, 15, 4))
    Y, X, Z = (slice(npd, npd + n) for n in (ny, nx, nz))
    ring = [(Y, X, npd - 1), (Y, X, npd + nz), (Y, npd - 1, Z), (Y, npd + nx, Z), (npd - 1, X, Z), (npd + ny, X, Z)]
    boundary = case["method"] == "boundary"
    k = kw["snap_every"]
    ill = torch.zeros((ny, nx, nz), device=DEV, dtype=torch.float64)
    rec, saved = [], {}
    for it, a in enumerate(_amps(nt, kw["dt"], kw["favg"], 10.0, False)):
        p.step(a)
        rec.append(p.P[Y, X, npd] + p.Q[Y, X, npd])
        if boundary:
            saved[it] = [(p.P[q].clone(), p.Q[q].clone()) for q in ring]
        elif it % k == k - 1:
            saved[it] = p.P[Y, X, Z].clone()
        ill += p.P[Y, X, Z] ** 2 + p.Q[Y, X, Z] ** 2
    f32 = np.float32
    gx = f32(kw["dx"]) * np.abs(np.arange(nx) - kw["fsx"]).astype(np.float32)
    gy = f32(kw["dy"]) * np.abs(np.arange(ny) - kw["fsy"]).astype(np.float32)
    off = np.sqrt((gx.astype(float)[None] ** 2 + gy.astype(float)[:, None] ** 2 +
                   float(f32(kw["dz"]) * kw["fsz"]) ** 2).astype(np.float32))
    t0 = off / f32(float(x[0][0, 0, 0]) * math.sqrt(1 + 2 * float(x[1][0, 0, 0])))
    i0 = (t0 / f32(kw["dt"])).astype(np.int64)
    lo, hi = i0 - 70, i0 + int(2.0 / float(f32(kw["dt"]) * f32(kw["favg"]))) + 70
    sv = [t.clone() for t in [p.P, p.Q] + p.vel + p.split]
    lo, hi = torch.from_numpy(lo).to(DEV), torch.from_numpy(hi).to(DEV)
    g = p
    if boundary:
        s = _Prop("gpu", x, npd, (kw["dy"], kw["dx"], kw["dz"]), kw["dt"], src, (src, 15, 4))
        s.P, s.Q, s.vel, s.split = sv[0], sv[1], sv[2:5], sv[5:]
    g.new_state()
    mig = torch.zeros_like(ill)
    for it in range(nt - 1, -1, -1):
        if boundary:
            for q, (a, b) in zip(ring, saved[it]):
                s.P[q], s.Q[q] = a, b
            s.step()
        r = torch.where((it > lo) & (it < hi), torch.zeros_like(rec[it]), rec[it])
        g.P[Y, X, npd - 1] = r
        g.Q[Y, X, npd - 1] = r
        g.step()
        gp = g.P[Y, X, Z]
        ill += gp * gp + g.Q[Y, X, Z] ** 2
        if boundary:
            mig += s.P[Y, X, Z] * gp
        elif it % k == k - 1:
            mig += k * saved[it] * gp
    if boundary:   # stepping from the restored ring amplifies rounding: no 64-bit image to compare with
        return None, None, ill
    mig = torch.where(ill > 2.0 ** -150, mig / ill, mig)
    return mig, _lap(mig), ill


def exact(case, seed):
    x = _inputs(case, seed)
    k = case["kind"]
    with torch.no_grad() if k != "codec_grad" else torch.enable_grad():
        if k in ("codec", "codec_grad"):
            return _exact_codec(case, x, seed)
        kw = _kw(case)
        if k == "rtm2d_gpu":
            return _exact_rtm2d_gpu(case, x, kw)
        if k == "rtm2d_batch":
            return _exact_rtm2d_batch(case, x, kw)
        if k == "rtm3d":
            return _exact_rtm3d(case, x, kw)
        return _exact_shot(case, x, kw)
