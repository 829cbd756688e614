"""Performance cases of the VTI modeling and gradient library.

Every case is one call (or one resident-plan call) that a user's program makes
through ``vtib200``: 2D traces, gradient and migration; 3D traces, gradient,
migration, offset gathers, the Gauss-Newton product and the batched survey.
Inputs are made from a seed: a layered VTI model (v 1500..4500 m/s) with a
smooth random perturbation, a Ricker wavelet, a receiver line or grid, and
field-like observed traces (direct, reflected and refracted arrivals).

``exact`` restates each path in 64-bit torch from the published scheme.
"""
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parents[1] / "thesis-source-code_b200"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import vtib200 as V  # noqa: E402

C8 = (-2.84722222222, 1.6, -0.2, 0.02539682539, -0.00178571428)
W_X, W_Z = 0.6666666666, 0.3333333333  # recording / injection weights
H = 4                                  # half width of the stencil
D3, DT3, ST3 = 12.5, 1e-3, 4           # 3D spacing, time step, trace step (4 ms)
D2, DT2, ST2 = 10.0, 1e-3, 2           # 2D spacing, time step, trace step (2 ms)


def listed():
    return [
        # a quick look at a 2 km line: the smallest call, one shot
        dict(name="synth2d_201x101", kind="synth2d", nx=201, nz=101, nt=1000, pad=30, ns=1),
        # a served modeling request at the wide end (8 km line), three shots
        dict(name="synth2d_801x401", kind="synth2d", nx=801, nz=401, nt=1000, pad=30, ns=3),
        # 2D inversion: the benchmark's 2D grid, one shot's gradient
        dict(name="grad2d_401x201", kind="grad2d", nx=401, nz=201, nt=1000, pad=30),
        # 2D migration of two shots, odd sizes
        dict(name="rtm2d_377x183", kind="rtm2d", nx=377, nz=183, nt=900, pad=30, ns=2),
        # a served 3D modeling request at the small end
        dict(name="model3d_128x128x128", kind="model3d", nx=128, ny=128, nz=128, nt=1000, pad=16),
        # a small 3D gradient through the one-call host form (the drop-in's)
        dict(name="grad3d_host_110x97x83", kind="grad3d_host", nx=110, ny=97, nz=83, nt=514,
             pad=12),
        # a shot window of a 3D survey, odd sizes, resident plan
        dict(name="grad3d_251x203x150", kind="grad3d", nx=251, ny=203, nz=150, nt=400, pad=24),
        # the benchmark's 3D gradient grid (its first 400 samples)
        dict(name="grad3d_400x400x200", kind="grad3d", nx=400, ny=400, nz=200, nt=400, pad=40),
        # 3D migration of one shot
        dict(name="rtm3d_256x224x128", kind="rtm3d", nx=256, ny=224, nz=128, nt=400, pad=24),
        # 3D offset gathers with the drop-in's 32 lags on each side
        dict(name="odcig3d_150x120x80", kind="odcig3d", nx=150, ny=120, nz=80, nt=300, pad=12,
             nlag=32),
        # one Gauss-Newton product and gradient (inner step of a truncated Newton inversion)
        dict(name="gnhv3d_200x180x120", kind="gnhv3d", nx=200, ny=180, nz=120, nt=300, pad=20),
        # a survey of windows on one model, all shots in one call
        dict(name="batch3d_6x256x256x100", kind="batch3d", nx=256, ny=256, nz=100, nt=258,
             pad=16, ns=6, amin=96, amax=224),
    ]


def _side(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm; odd as often as even."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["synth2d", "synth2d", "grad2d", "rtm2d", "model3d", "grad3d_host",
                       "grad3d", "grad3d", "rtm3d", "odcig3d", "gnhv3d", "batch3d"])
    if kind in ("synth2d", "grad2d", "rtm2d"):
        c = dict(kind=kind, nx=_side(rng, 150, 801), nz=_side(rng, 90, 401),
                 nt=_side(rng, 400, 1200), pad=rng.choice([20, 30, 40]))
        if kind != "grad2d":
            c["ns"] = rng.randint(1, 3)
        return c
    lo, hi = {"model3d": (96, 300), "grad3d_host": (72, 160), "grad3d": (128, 320),
              "rtm3d": (128, 300), "odcig3d": (100, 160), "gnhv3d": (96, 220),
              "batch3d": (192, 280)}[kind]
    pad = rng.choice([12, 16, 24])
    c = dict(kind=kind, nx=_side(rng, lo, hi), ny=_side(rng, lo, hi),
             nz=_side(rng, 64, 160 if hi > 160 else 100), nt=_side(rng, 160, 500), pad=pad)
    if kind == "odcig3d":
        c["nlag"] = rng.randint(8, 32)
    if kind == "batch3d":
        c.update(ns=rng.randint(2, 6), amin=96, amax=min(c["nx"], c["ny"]), nt=_side(rng, 130, 260))
    return c


# ------------------------------------------------------------------- inputs
def _ricker(nt, dt, freq):
    a = (np.pi * freq * (np.arange(nt) * dt - 1.2 / freq)) ** 2
    return ((1 - 2 * a) * np.exp(-a)).astype(np.float32)


def _smooth_noise(shape, seed, cells, dev):
    """Unit-range smooth random field: coarse noise, linearly interpolated."""
    gen = torch.Generator("cpu").manual_seed(seed)
    coarse = [max(3, n // cells + 2) for n in shape]
    t = torch.rand([1, 1] + coarse, generator=gen) * 2 - 1
    mode = "bilinear" if len(shape) == 2 else "trilinear"
    return torch.nn.functional.interpolate(t.to(dev), size=list(shape), mode=mode,
                                           align_corners=True)[0, 0]


def _model(shape, pad, seed, dev="cuda"):
    """c11, c13, c33 (float32, z slowest) of a 5-layer VTI model with a +-6 %
    smooth perturbation; the pad repeats the layer at its edge."""
    rng = np.random.default_rng(seed)
    nz = shape[0]
    inter = np.sort(rng.uniform(0.1, 0.9, 4)) * (nz - 2 * pad)
    k = np.searchsorted(inter, np.clip(np.arange(nz) - pad, 0, nz - 2 * pad - 1), side="right")
    lay = lambda a: torch.tensor(np.asarray(a, np.float32)[k], device=dev).view(  # noqa: E731
        [-1] + [1] * (len(shape) - 1))
    v = lay([1500, 2250, 3000, 3750, 4500]) * (1 + 0.06 * _smooth_noise(shape, seed + 1, 16, dev))
    eps = (lay([0, .05, .1, .15, .2]) * (1 + 0.1 * _smooth_noise(shape, seed + 2, 16, dev)))
    dl = 0.5 * eps
    c33 = v * v
    return [t.contiguous() for t in (c33 * (1 + 2 * eps), c33 * torch.sqrt(1 + 2 * dl), c33)]


def _events(case, seed, off, dt, vol):
    """Field-like traces (receivers x samples) at offsets `off` (m): direct
    wave, two reflections and a refraction with random strengths; amplitudes
    of a point source of cell volume `vol`."""
    rng = np.random.default_rng(seed + 7)
    nnt = (case["nt"] - 1) // (ST3 if "ny" in case else ST2) + 1
    t = np.arange(nnt) * dt
    r = np.maximum(off, 12.5)[:, None]
    freq = 12.0
    out = np.zeros((off.size, nnt), dtype=np.float32)
    for v0, tau, s in ((1500.0, 0.0, 1.0), (1900.0, rng.uniform(.2, .4), .5 * rng.uniform(.5, 1)),
                       (2400.0, rng.uniform(.5, .8), .3 * rng.uniform(.5, 1)),
                       (3500.0, rng.uniform(.1, .3), .1 * rng.uniform(.5, 1))):
        arr = np.sqrt(tau * tau + (r / v0) ** 2) + 1.2 / freq
        a = (np.pi * freq * (t[None, :] - arr)) ** 2
        amp = s * vol / (4 * np.pi * v0 * v0 * np.sqrt(r * r + (tau * v0) ** 2))
        out += (amp * (1 - 2 * a) * np.exp(-a)).astype(np.float32)
    out[:, 0] = 0  # sample 0 lies before the source
    return out


def _in3(case, seed):
    """Everything a 3D case starts from, made from the seed alone."""
    nx, ny, nz, pad = case["nx"], case["ny"], case["nz"], case["pad"]
    rng = np.random.default_rng(seed)
    c = _model((nz, ny, nx), pad, seed)
    # random boundary: the pad's stiffnesses lowered by random factors
    mask = torch.ones((nz, ny, nx), dtype=torch.bool, device="cuda")
    mask[pad:nz - pad, pad:ny - pad, pad:nx - pad] = False
    gen = torch.Generator("cuda").manual_seed(seed + 3)
    low = 1 - 0.4 * torch.rand((nz, ny, nx), generator=gen, device="cuda")
    cr = [torch.where(mask, k * low, k) for k in c]
    sx, sy = nx // 2 + int(rng.integers(-3, 4)), ny // 2 + int(rng.integers(-3, 4))
    zr = pad + 2
    rx, ry = np.meshgrid(np.arange(H, nx - H, 2), np.arange(H, ny - H, 2))
    rx, ry = rx.reshape(-1), ry.reshape(-1)
    rec = np.zeros((rx.size, 4), np.float32)
    rec[:, 0], rec[:, 1], rec[:, 2], rec[:, 3] = (rx + .25) * D3, (ry + .25) * D3, (zr + .25) * D3, 1
    sou = np.array([(sx + .25) * D3, (sy + .25) * D3, (zr + .25) * D3, rx.size, 0], np.float32)
    off = D3 * np.hypot(rx - sx, ry - sy)
    data = _events(case, seed, off, ST3 * DT3, D3 ** 3)
    return dict(c=c, cr=cr, mask=mask, src=(zr, sy, sx), rx=rx, ry=ry, zr=zr, rec=rec, sou=sou,
                data=data, wav=_ricker(case["nt"], DT3, 12.0))


def _geom3(case):
    return V.geom3d(case["nx"], case["ny"], case["nz"], case["nt"], case["pad"], D3, D3, D3, DT3,
                    ST3 * DT3)


def _in2(case, seed):
    nx, nz, pad, ns = case["nx"], case["nz"], case["pad"], case.get("ns", 1)
    rng = np.random.default_rng(seed)
    c = _model((nz + 2 * pad, nx + 2 * pad), pad, seed, "cpu")
    sx = [int(pad + nx * (k + .5) / ns + rng.integers(-5, 6)) for k in range(ns)]
    per = nx // ns  # each shot is recorded by its own part of the line
    rloc = np.zeros((per * ns, 2), np.int32)
    rloc[:, 0] = np.concatenate([pad + k * per + np.arange(per) for k in range(ns)])
    rloc[:, 1] = pad + 2
    sloc = np.array([[sx[k], pad + 2, per, k * per] for k in range(ns)], np.int32)
    off = np.concatenate([D2 * np.abs(rloc[k * per:(k + 1) * per, 0] - sx[k]) for k in range(ns)])
    data = np.ascontiguousarray(_events(case, seed, off, ST2 * DT2, 40 * D2 ** 2).T)
    return dict(c=[k.numpy().reshape(-1) for k in c], sloc=sloc, rloc=rloc, data=data,
                wav=_ricker(case["nt"], DT2, 15.0))


_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = V.Context(0)
    return _ctx


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    if kind in ("synth2d", "grad2d", "rtm2d"):
        s = _in2(case, seed)
        s["g"] = V.geom2d(case["nx"], case["nz"], case["nt"], case["pad"], D2, D2, DT2, ST2 * DT2)
        s["taper"] = V.init_taper2d(case["nx"], case["nz"], case["pad"])
        return dict(s, kind=kind, ctx=ctx)
    i = _in3(case, seed)
    g, n = _geom3(case), case["nx"] * case["ny"] * case["nz"]
    s = dict(kind=kind, ctx=ctx, g=g, sou=i["sou"], rec=i["rec"], wav=i["wav"])
    if kind == "grad3d_host":
        lists = lambda m: torch.cat([k[i["mask"]] for k in m]).cpu().numpy()  # noqa: E731
        return dict(s, cij=torch.cat([k.view(-1) for k in i["c"]]).cpu().numpy(),
                    padb=lists(i["c"]), randb=lists(i["cr"]), data=i["data"].reshape(-1))
    if kind == "gnhv3d":
        c = [k.cpu().numpy().reshape(-1) for k in i["c"]]
        return dict(s, c=c, dc=_perturbation(i, case, seed).cpu().numpy().reshape(-1),
                    data=i["data"].reshape(-1))
    if kind == "batch3d":
        wins, sou, rec, data = _survey(case, seed)
        b = V.Batch3d(ctx, g, V.OPT_FULL_STEPS)
        b.set_model(*[k.data_ptr() for k in i["c"]], mem=V.MEM_DEVICE)
        b.set_wavelet(i["wav"])
        b.set_receivers(rec)
        b.set_shots(sou, wins, seed=seed & 0xffff)
        return dict(kind=kind, batch=b, data=torch.tensor(data.reshape(-1), device="cuda"),
                    fg=torch.zeros(1 + 3 * n, device="cuda"))
    plan = V.Plan3d(ctx, g, V.OPT_FULL_STEPS)
    lists = lambda m: torch.cat([k[i["mask"]] for k in m])  # noqa: E731
    padb, randb = (lists(i["c"]), lists(i["cr"])) if kind != "model3d" else (None, None)
    torch.cuda.synchronize()
    plan.set_model(*[k.data_ptr() for k in i["c"]], None if padb is None else padb.data_ptr(),
                   None if randb is None else randb.data_ptr(), mem=V.MEM_DEVICE)
    plan.set_wavelet(i["wav"])
    plan.set_receivers(i["rec"])
    s["plan"] = plan
    s["data"] = torch.tensor(i["data"].reshape(-1), device="cuda")
    if kind == "odcig3d":
        s["nlag"] = case["nlag"]
    if kind == "model3d":
        s["out"] = torch.zeros_like(s["data"])
    if kind == "grad3d":
        s["fg"] = torch.zeros(1 + 3 * n, device="cuda")
    if kind == "rtm3d":
        s["image"] = torch.zeros(n, device="cuda")
    return s


def run(s):
    kind = s["kind"]
    if kind == "synth2d":
        return V.synthetic_f(s["ctx"], s["g"], *s["c"], s["wav"], s["sloc"], s["rloc"], s["taper"])
    if kind == "grad2d":
        return V.objFuncGradient_f(s["ctx"], s["g"], s["data"], *s["c"], s["wav"], s["sloc"],
                                   s["rloc"], s["taper"])
    if kind == "rtm2d":
        return V.rtm_f(s["ctx"], s["g"], s["data"], *s["c"], s["wav"], s["sloc"], s["rloc"],
                       s["taper"])
    if kind == "grad3d_host":
        return V.objFuncGradientCij3d_f(s["ctx"], s["g"], s["sou"], [0], s["rec"], s["wav"],
                                        s["cij"], s["padb"], s["randb"], s["data"])
    if kind == "gnhv3d":
        o = V.gnhv_exact(s["ctx"], s["g"], *s["c"], s["wav"], s["sou"], s["rec"], dc=s["dc"],
                         dobs=s["data"])
        return [o[k] for k in ("hv", "grad", "traces", "born", "misfit")]
    if kind == "batch3d":
        _, mis = s["batch"].gradient(s["data"].data_ptr(), V.MEM_DEVICE, s["fg"].data_ptr(),
                                     V.MEM_DEVICE)
        return s["fg"], mis
    plan, dev = s["plan"], V.MEM_DEVICE
    if kind == "model3d":
        plan.model_data(s["sou"], [0], out=s["out"].data_ptr(), mem=dev)
        return s["out"]
    if kind == "grad3d":
        _, mis = plan.gradient(s["sou"], [0], s["data"].data_ptr(), dev, s["fg"].data_ptr(), dev)
        return s["fg"], mis
    if kind == "rtm3d":
        plan.rtm(s["sou"], [0], s["data"].data_ptr(), dev, s["image"].data_ptr(), dev)
        return s["image"]
    return plan.odcig(s["sou"], [0], s["data"].data_ptr(), s["nlag"], data_mem=dev)


# Extra inputs of single kinds.
def _perturbation(i, case, seed):
    """Model perturbation dc (3, nz, ny, nx): 3 % smooth random field, zero in the pad."""
    shape = (case["nz"], case["ny"], case["nx"])
    return torch.stack([torch.where(i["mask"], 0, 0.03 * k * _smooth_noise(shape, seed + 20 + j, 8,
                                                                          "cuda"))
                        for j, k in enumerate(i["c"])])


def _survey(case, seed):
    """Windows, sources, receivers and traces of a batched survey."""
    rng = np.random.default_rng(seed + 11)
    nx, ny, pad, wins, sou, rec, data, first = case["nx"], case["ny"], case["pad"], [], [], [], [], 0
    zr = pad + 2
    for _ in range(case["ns"]):
        ax, ay = (int(rng.integers(case["amin"], min(case["amax"], m) + 1)) for m in (nx, ny))
        x0, y0 = int(rng.integers(0, nx - ax + 1)), int(rng.integers(0, ny - ay + 1))
        sx, sy = x0 + ax // 2, y0 + ay // 2
        rx, ry = np.meshgrid(np.arange(x0 + pad, x0 + ax - pad, 2),
                             np.arange(y0 + pad, y0 + ay - pad, 2))
        rx, ry = rx.reshape(-1), ry.reshape(-1)
        r = np.zeros((rx.size, 4), np.float32)
        r[:, 0], r[:, 1], r[:, 2], r[:, 3] = (rx + .25) * D3, (ry + .25) * D3, (zr + .25) * D3, 1
        wins.append((x0, y0, ax, ay))
        rec.append(r)
        sou.append([(sx + .25) * D3, (sy + .25) * D3, (zr + .25) * D3, rx.size, first])
        data.append(_events(case, seed, D3 * np.hypot(rx - sx, ry - sy), ST3 * DT3, D3 ** 3))
        first += rx.size
    return wins, np.array(sou, np.float32), np.concatenate(rec), np.concatenate(data)


# --------------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass. 3D: per level, every field, model and
    image volume that a level needs read and written once (volumes exceed the
    caches); 2D: inputs and outputs once (a shot's state fits on chip)."""
    kind, nt = case["kind"], case["nt"]
    if kind in ("synth2d", "grad2d", "rtm2d"):
        n = (case["nx"] + 2 * case["pad"]) * (case["nz"] + 2 * case["pad"])
        rows, ns = (nt - 1) // ST2 + 1, case.get("ns", 1)
        io = 4 * (4 * n + rows * case["nx"])
        f = {"synth2d": 40, "grad2d": 40 + 55, "rtm2d": 40 + 46}[kind]
        return {"bytes": io + {"synth2d": 0, "grad2d": 12 * n, "rtm2d": 4 * n}[kind],
                "flops": float(f) * n * nt * ns}
    n = (case["nx"] - 8) * (case["ny"] - 8) * case["nz"]
    if kind == "batch3d":
        n = case["ns"] * ((case["amin"] + case["amax"]) // 2) ** 2 * case["nz"]
    nr = case["nx"] * case["ny"] // 4
    lev = {"model3d": 36, "grad3d": 156, "grad3d_host": 156, "batch3d": 156, "rtm3d": 36 + 68,
           "odcig3d": 36 + 68, "gnhv3d": 72 + 36 + 2 * 84}[kind]
    fl = {"model3d": 54, "grad3d": 224, "grad3d_host": 224, "batch3d": 224, "rtm3d": 170,
          "odcig3d": 170 + 2 * (2 * case.get("nlag", 0) + 1), "gnhv3d": 420}[kind]
    out = {"model3d": 0, "rtm3d": 1, "odcig3d": 2 * case.get("nlag", 0) + 1, "gnhv3d": 12}.get(kind, 6)
    return {"bytes": float(lev) * n * nt + 4.0 * n * out + 4.0 * nr * (nt // ST3),
            "flops": float(fl) * n * nt}


def tolerance(case):
    """Relative errors of FP32 leapfrog runs of a few hundred to a thousand
    levels, about four times what the paths measure against ``exact`` over the
    listed and a few drawn cases: traces up to 9e-6; Born traces, dominated by
    the cancelling near field of the source, 2.4e-4; gradients and images
    around 2e-5 here and, where the image sum cancels near the source, 2e-4
    from one operation order to another."""
    kind = case["kind"]
    if kind in ("synth2d", "model3d"):
        return {"rel": 5e-5, "max": 2e-3}
    if kind == "gnhv3d":
        return {"rel": 1e-3, "max": 4e-2}
    return {"rel": 4e-4, "max": 2e-2}


# -------------------------------------------------------------------- exact
def _f(x):
    """The float32 value a call passes, as a Python float."""
    return float(np.float32(x))


class _Grid3:
    """64-bit 3D operators on (nz, ny, nx) tensors with a zero 4-cell x/y frame."""

    def __init__(self, case, wav):
        self.nz, self.ny, self.nx, self.pad = case["nz"], case["ny"], case["nx"], case["pad"]
        self.dt2, self.i2 = _f(DT3) ** 2, 1 / _f(D3) ** 2
        self.w = [float(v) for v in wav]
        prof = [torch.tensor([self._damp(i, n) for i in range(n)], dtype=torch.float64,
                             device="cuda") for n in (self.nz, self.ny, self.nx)]
        self.d = (prof[0][:, None, None] * prof[1][None, :, None] * prof[2][None, None, :])
        self.dc = self.core(self.d)
        z = torch.arange(self.nz, device="cuda")
        # planes z-k of the 4-plane block above are already damped
        self.above = [((z[k:] - k) // 4 < z[k:] // 4).view(-1, 1, 1) for k in range(5)]

    def _damp(self, i, n):
        dist = self.pad - i if i < self.pad else (i - n + self.pad if i > n - self.pad else 0)
        return float(np.float32(.95 + (1. - .95) * np.cos(3.14159265359 * dist / self.pad)))

    def zeros(self):
        return torch.zeros((self.nz, self.ny, self.nx), dtype=torch.float64, device="cuda")

    def core(self, u):
        return u[:, H:-H, H:-H]

    def lxy(self, u):
        a = self.core(u) * (2 * C8[0] * self.i2)
        for k in range(1, 5):
            f = C8[k] * self.i2
            a.add_(u[:, H:-H, H + k:self.nx - H + k], alpha=f)
            a.add_(u[:, H:-H, H - k:self.nx - H - k], alpha=f)
            a.add_(u[:, H + k:self.ny - H + k, H:-H], alpha=f)
            a.add_(u[:, H - k:self.ny - H - k, H:-H], alpha=f)
        return a

    def lz(self, q, sponge):
        q = self.core(q)
        a = q * (C8[0] * self.i2)
        qd = q * self.dc if sponge else None
        for k in range(1, 5):
            f = C8[k] * self.i2
            a[:-k].add_(q[k:], alpha=f)
            up = torch.where(self.above[k], qd[:-k], q[:-k]) if sponge else q[:-k]
            a[k:].add_(up, alpha=f)
        return a

    def step(self, cur, prev, c, sponge, src=None, amp=0.0, lap=None):
        """next over prev (in place); returns the unscaled Laplacian pair."""
        h, z = lap or (self.lxy(cur[0]), self.lz(cur[1], sponge))
        for f, (a, b) in enumerate(((c[0], c[1]), (c[1], c[2]))):
            n = (a * h).addcmul_(b, z).mul_(self.dt2).add_(self.core(cur[f]), alpha=2)
            p = self.core(prev[f])
            n.sub_(p * self.dc if sponge else p)
            if src is not None:
                n[src[0], src[1] - H, src[2] - H] += amp
            p.copy_(n.mul_(self.dc) if sponge else n)
        return h, z

    def forward(self, c, src, last, sponge, each=None):
        """Levels 1..last; returns (level last, level last-1)."""
        cur, prev = [self.zeros(), self.zeros()], [self.zeros(), self.zeros()]
        for u in cur:
            u[src] = self.dt2 * self.w[0]
        for it in range(2, last + 1):
            self.step(cur, prev, c, sponge, src, self.dt2 * self.w[it - 1])
            cur, prev = prev, cur
            if each:
                each(it, cur)
        return cur, prev


def _backward3(G, case, c, i, cur, prev, last, r, image):
    """The adjoint sweep: source field (cur = level last-1, prev = level last)
    stepped back, adjoint driven by the traces r; image(h, z, sc, lc) per level."""
    nt, nnt = case["nt"], r.shape[1]
    la, lb = [G.zeros(), G.zeros()], [G.zeros(), G.zeros()]
    at = (torch.full((len(i["rx"]),), i["zr"], device="cuda"), torch.tensor(i["ry"], device="cuda"),
          torch.tensor(i["rx"], device="cuda"))
    for u, w in zip(la, (W_X, W_Z)):
        u[at] = w * G.dt2 * r[:, nnt - 1]
    for k in range(last - 1):
        it = nt - 3 - k
        lap = G.lxy(cur[0]), G.lz(cur[1], False)
        image(lap, cur, la)
        G.step(cur, prev, c, False, i["src"], G.dt2 * G.w[it + 1], lap)
        G.step(la, lb, c, True)
        f = float(np.float32(it + 1) / np.float32(ST3))
        i0 = int(f)
        v = r[:, nnt - 1] if i0 >= nnt - 1 else (1 - (f - i0)) * r[:, i0] + (f - i0) * r[:, i0 + 1]
        for u, w in zip(lb, (W_X, W_Z)):
            u[at] += G.d[at] * (w * G.dt2) * v
        cur, prev, la, lb = prev, cur, lb, la


def _exact3(case, seed):
    kind, nt = case["kind"], case["nt"]
    i = _in3(case, seed)
    G = _Grid3(case, i["wav"])
    last = nt - 1 if kind != "grad3d_host" else 1 + 64 * ((nt - 2) // 64)
    nnt = (nt - 1) // ST3 + 1
    rx, ry = (torch.tensor(k, device="cuda") for k in (i["rx"], i["ry"]))
    data = torch.tensor(i["data"], device="cuda").double()
    c = [G.core(k.double()).contiguous() for k in i["c"]]
    if kind == "gnhv3d":
        return _exact_gn(case, seed, i, G, c, rx, ry, data, last)
    cr = [G.core(k.double()).contiguous() for k in i["cr"]]
    tr = torch.zeros((rx.numel(), nnt), dtype=torch.float64, device="cuda")

    def record(it, cur):
        if it % ST3 == 0 and it // ST3 < nnt:
            tr[:, it // ST3] = W_X * cur[0][i["zr"], ry, rx] + W_Z * cur[1][i["zr"], ry, rx]

    if kind in ("model3d", "grad3d", "grad3d_host"):
        G.forward(c, i["src"], last, True, record)
    if kind == "model3d":
        return tr.view(-1)
    cur, prev = G.forward(cr, i["src"], last, False)
    if kind.startswith("grad3d"):
        r = tr - data
        g = [G.zeros() for _ in range(3)]

        def image(lap, sc, lc):
            lx, lz = G.core(lc[0]), G.core(lc[1])
            G.core(g[0]).addcmul_(lx, lap[0])
            G.core(g[1]).addcmul_(lz, lap[0]).addcmul_(lx, lap[1])
            G.core(g[2]).addcmul_(lz, lap[1])

        _backward3(G, case, cr, i, prev, cur, last, r, image)
        mis = float((r * r).sum()) / 2
        fg = torch.cat([torch.tensor([mis], dtype=torch.float64, device="cuda")]
                       + [k.view(-1) for k in g])
        return (fg if kind == "grad3d" else fg.cpu().numpy()), mis
    nlag = case.get("nlag", 0)
    out = [G.zeros() for _ in range(2 * nlag + 1)]
    lo, nx = max(H, nlag), case["nx"]

    def image(lap, sc, lc):
        s = G.core(W_X * sc[0] + W_Z * sc[1])[:, :, lo - H:nx - lo - H]
        rr = (W_X * lc[0] + W_Z * lc[1]) * G.d
        for j in range(2 * nlag + 1):
            h = j - nlag
            out[j][:, H:-H, lo:nx - lo].addcmul_(s, rr[:, H:-H, lo + h:nx - lo + h])

    _backward3(G, case, cr, i, prev, cur, last, data, image)
    if kind == "rtm3d":
        return out[0].view(-1)
    return torch.stack(out).view(2 * nlag + 1, -1).cpu().numpy()


def _exact_gn(case, seed, i, G, c, rx, ry, data, last):
    """Exact-mode forward, Born and adjoint levels: centred damping."""
    dc = [G.core(k.double()).contiguous() for k in _perturbation(i, case, seed)]
    nnt, z0 = data.shape[1], i["zr"]
    k1, k2 = G.dc * G.dt2, 2 * G.dc - 1
    a, ap, b, bp = ([G.zeros(), G.zeros()] for _ in range(4))
    for u in a:
        u[i["src"]] = G.dt2 * G.w[0]
    tr, born = (torch.zeros((rx.numel(), nnt), dtype=torch.float64, device="cuda") for _ in "ab")
    laps = {}
    for t in range(2, last + 1):
        h, z = laps[t - 1] = G.lxy(a[0]), G.lz(a[1], False)
        hb, zb = G.lxy(b[0]), G.lz(b[1], False)
        for f in range(2):
            n = k1 * (c[f] * h + c[f + 1] * z) + 2 * G.dc * G.core(a[f]) - k2 * G.core(ap[f])
            s = i["src"]
            n[s[0], s[1] - H, s[2] - H] += G.d[s] * G.dt2 * G.w[t - 1]
            m = k1 * (c[f] * hb + c[f + 1] * zb + dc[f] * h + dc[f + 1] * z)
            m += 2 * G.dc * G.core(b[f]) - k2 * G.core(bp[f])
            G.core(ap[f]).copy_(n)
            G.core(bp[f]).copy_(m)
        a, ap, b, bp = ap, a, bp, b
        if t % ST3 == 0 and t // ST3 < nnt:
            for to, u in ((tr, a), (born, b)):
                to[:, t // ST3] = W_X * u[0][z0, ry, rx] + W_Z * u[1][z0, ry, rx]
    del a, ap, b, bp
    r, imgs = tr - data, []
    for res in (r, born):
        mu, mp = [G.zeros(), G.zeros()], [G.zeros(), G.zeros()]
        g = [G.zeros() for _ in range(3)]
        w = [G.zeros(), G.zeros()]
        for t in range(last, 1, -1):
            for f in range(2):
                G.core(w[f]).copy_(c[f] * G.core(mu[0]) + c[f + 1] * G.core(mu[1]))
            back = G.lxy(w[0]), G.lz(w[1], False)
            for f in range(2):
                G.core(mp[f]).copy_(k1 * back[f] + 2 * G.dc * G.core(mu[f]) - k2 * G.core(mp[f]))
                if t % ST3 == 0 and t // ST3 < nnt:
                    mp[f][z0, ry, rx] += G.d[z0, ry, rx] * (W_X, W_Z)[f] * res[:, t // ST3]
            mu, mp = mp, mu
            h, z = laps[t - 1]
            mx, mz = G.core(mu[0]) * G.dt2, G.core(mu[1]) * G.dt2
            G.core(g[0]).addcmul_(mx, h)
            G.core(g[1]).addcmul_(mx, z).addcmul_(mz, h)
            G.core(g[2]).addcmul_(mz, z)
        imgs.append(torch.stack(g).view(-1).cpu().numpy())
    return [imgs[1], imgs[0], tr.view(-1).cpu().numpy(), born.view(-1).cpu().numpy(),
            float((r * r).sum()) / 2]


class _Grid2:
    """64-bit 2D operators on (nnz, nnx) tensors, zero 4-cell frame."""

    def __init__(self, case):
        self.nnx, self.nnz = case["nx"] + 2 * case["pad"], case["nz"] + 2 * case["pad"]
        self.dt2, self.i2 = _f(DT2) ** 2, 1 / _f(D2) ** 2
        t = torch.ones((self.nnz, self.nnx), dtype=torch.float64, device="cuda")
        npad = case["pad"]
        for i in range(npad):
            f = _f(np.float32(.95) + (1. - np.float64(np.float32(.95)))
                   * np.cos(float(np.float32(np.pi)) * np.float32(npad - 1 - i) / npad))
            t[:, i] *= f
            t[:, self.nnx - 1 - i] *= f
            t[i] *= f
            t[self.nnz - 1 - i] *= f
        self.taper, self.t = t, self.core(t)

    def zeros(self):
        return torch.zeros((self.nnz, self.nnx), dtype=torch.float64, device="cuda")

    def core(self, u):
        return u[H:-H, H:-H]

    def lap(self, p, q):
        """(Dxx p, Dzz q) on the update region."""
        a, b = self.core(p) * (C8[0] * self.i2), self.core(q) * (C8[0] * self.i2)
        for k in range(1, 5):
            f = C8[k] * self.i2
            a.add_(p[H:-H, H + k:self.nnx - H + k], alpha=f)
            a.add_(p[H:-H, H - k:self.nnx - H - k], alpha=f)
            b.add_(q[H + k:self.nnz - H + k, H:-H], alpha=f)
            b.add_(q[H - k:self.nnz - H - k, H:-H], alpha=f)
        return a, b

    def step(self, cur, prev, c, lap, src=None, amp=0.0, dipole=False):
        """Forward form C D (c given) or the update with lap as is (c None)."""
        for f in range(2):
            s = lap[f] if c is None else c[f] * lap[0] + c[f + 1] * lap[1]
            n = self.dt2 * s + 2 * self.core(cur[f]) - self.t * self.core(prev[f])
            if src is not None:
                n[src[1] - H, src[0] - H] += amp
                if dipole:
                    n[src[1] + 1 - H, src[0] - H] -= amp
            self.core(prev[f]).copy_(n * self.t)


def _pairs(nt, r):
    """Which two stored levels of D(sigma) each adjoint level is imaged with:
    the reference's rotation of its checkpoint buffers for a first shot."""
    host = [None] * ((nt - 1) // r + 1)
    dq, da, db, ha, hb = 1, None, None, None, None
    for it in range(2, nt):
        dq = it
        if it % r == 0:
            da = dq if it != nt - 1 else da
            if it > r and it // r - 1 < len(host):
                host[it // r - 1] = ha
        if it % r == 1 and it != nt - r:
            ha = da
    if len(host) >= 3:
        hb = host[len(host) - 3]
    f = (nt - 2.) / r
    out = [(da, dq, f - int(f))]
    for it in range(nt - 3, -1, -1):
        if it % r == 0:
            ha, hb = hb, ha
            db = ha
            hb = host[it // r - 2] if it >= 2 * r else hb
        if (it + 1) % r == 0:
            db, dq, da = dq, da, db
        out.append((da, dq, it / r - it // r))
    return out


def _exact2(case, seed):
    kind, nt = case["kind"], case["nt"]
    i = _in2(case, seed)
    G = _Grid2(case)
    c = [G.core(torch.tensor(k, device="cuda").view(G.nnz, G.nnx).double()).contiguous()
         for k in i["c"]]
    wav = [float(v) for v in i["wav"]]
    rows, nr = (nt - 1) // ST2 + 1, len(i["rloc"])
    rx, rz = (torch.tensor(i["rloc"][:, k], device="cuda").long() for k in (0, 1))
    tr = torch.zeros((rows, nr), dtype=torch.float64, device="cuda")
    data = torch.tensor(i["data"], device="cuda").double()
    img = [G.zeros() for _ in range(3)]
    for sx, sz, nri, ir0 in i["sloc"].tolist():
        x, z = rx[ir0:ir0 + nri], rz[ir0:ir0 + nri]
        cur, prev = [G.zeros(), G.zeros()], [G.zeros(), G.zeros()]
        dip = kind == "rtm2d"
        for u in cur:
            u[sz, sx] = G.dt2 * wav[0] * (1 if kind == "grad2d" else float(G.taper[sz, sx]))
            if dip:
                u[sz + 1, sx] = -G.dt2 * wav[0] * float(G.taper[sz + 1, sx])
        kept, slices = {}, {}
        pairs = _pairs(nt, ST2) if kind == "grad2d" else []
        need = {k for p in pairs for k in p[:2]}
        for it in range(2, nt):
            lap = G.lap(*cur)
            if it - 1 in need:
                kept[it - 1] = lap
            G.step(cur, prev, c, lap, (sx, sz), G.dt2 * wav[it - 1], dip)
            cur, prev = prev, cur
            if it % ST2 == 0:
                if dip:
                    slices[it // ST2] = 0.5 * (cur[0] + cur[1])
                else:
                    tr[it // ST2, ir0:ir0 + nri] = 0.5 * (cur[0][z, x] + cur[1][z, x])
        if kind == "synth2d":
            continue
        if nt - 1 in need:
            kept[nt - 1] = G.lap(*cur)
        d = data[:, ir0:ir0 + nri] if dip else tr - data
        cur, prev = [G.zeros(), G.zeros()], [G.zeros(), G.zeros()]

        def inject(u, v, scaled):
            t = G.taper[z, x] if scaled else 1.0
            for w in u:
                w.index_put_((z, x), v * t, accumulate=True)
                if dip:
                    w.index_put_((z + 1, x), -v * G.taper[z + 1, x], accumulate=True)

        inject(cur, G.dt2 * 0.5 * d[rows - 1], dip)
        b0, b1 = d[rows - 1], torch.zeros_like(d[0])
        zero = torch.zeros_like(cur[0])
        f = (nt - 2.) / ST2
        s0, s1, fs = int(f), min(int(f) + 1, rows), f - int(f)
        for n, it in enumerate(range(nt - 3, -2, -1)):  # images level it+1, makes level it
            if kind == "grad2d":
                ka, kb, fw = pairs[n]
                dp, dq = ((1 - fw) * kept[ka][k] * 1.0 if ka is not None else 0 for k in (0, 1))
                dp, dq = (v + (fw * kept[kb][k] if kb is not None else 0)
                          for k, v in enumerate((dp, dq)))
                p, q = G.core(cur[0]), G.core(cur[1])
                for u, v in zip(img, (p * dp, p * dq + q * dp, q * dq)):
                    G.core(u).add_(v)
            else:
                s = (1 - fs) * slices.get(s0, zero) + fs * slices.get(s1, zero)
                G.core(img[0]).add_(G.core(0.5 * (cur[0] + cur[1]) * s))
            if it < 0:
                break
            if kind == "grad2d":
                w = [G.zeros(), G.zeros()]
                for k in range(2):
                    G.core(w[k]).copy_(c[k] * G.core(cur[0]) + c[k + 1] * G.core(cur[1]))
                    # the frame of the adjoint is zero except for seeded receivers
                G.step(cur, prev, None, G.lap(*w))
            else:
                G.step(cur, prev, c, G.lap(*cur))
            f = (it + 1.) / ST2
            if (it + 2) % ST2 == 0:
                b0, b1 = d[int(f)], b0
            fi = f - int(f)
            inject(prev, G.dt2 * 0.5 * ((1 - fi) * b0 + fi * b1), True)
            cur, prev = prev, cur
            if (it + 1) % ST2 == 0:
                s0, s1 = it // ST2, s0
            fs = it / ST2 - it // ST2
    if kind == "synth2d":
        return tr.cpu().numpy()
    if kind == "rtm2d":
        return img[0].view(-1).cpu().numpy()
    r = tr - data
    return tuple(k.view(-1).cpu().numpy() for k in img) + (0.5 * float((r * r).sum()),)


def exact(case, seed):
    if case["kind"] == "batch3d":  # its random boundaries are the library's own
        return None
    with torch.no_grad():
        if "ny" not in case:
            return _exact2(case, seed)
        return _exact3(case, seed)
