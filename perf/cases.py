"""Timed cases of the propagators and of the U-Net convolution.

A propagation case is one call of ``PropTorch`` as a modelling or inversion
program makes it: either a forward run that makes records (``grad`` false) or
one gradient of the L2 misfit against observed records (``grad`` true), which
runs the forward, the adjoint and the imaging.  A convolution case is one
3x3 layer of the U-Net preconditioner, forward and backward.

Grid sizes, layer widths, orders and shot counts are those of the repository's
benchmark workloads and tests; the time axes are shorter than a survey's (the
cost of a step does not depend on their length).  Models are layered with a
smooth anomaly, wavelets are Ricker pulses, and observed records are pulses
with the moveout and amplitude of direct and reflected arrivals.
"""
from __future__ import annotations

import math
from fractions import Fraction

import numpy as np
import torch
import torch.nn.functional as F

import sweep_b200 as sb
from sweep_b200 import unet

DEVICE = "cuda"

# Per equation: the class, number of space axes and of models, the Courant
# number dt v_max / h of the time step, and the rate in cell-steps per second
# by which a drawn case's cost is bounded.
EQS = {
    "acoustic2d": dict(cls=sb.Acoustic, nd=2, models=1, courant=0.40, rate=30e9),
    "acoustic3d": dict(cls=sb.Acoustic3D, nd=3, models=1, courant=0.36, rate=25e9),
    "elastic2d": dict(cls=sb.Elastic, nd=2, models=3, courant=0.40, rate=9e9),
    "elastic3d": dict(cls=sb.Elastic3D, nd=3, models=3, courant=0.34, rate=4e9),
    "vti2d": dict(cls=sb.AcousticVTI1st, nd=2, models=4, courant=0.36, rate=11e9),
    "vti3d": dict(cls=sb.AcousticVTI1st3D, nd=3, models=4, courant=0.32, rate=8e9),
}


def _case(name, eq, order, shape, nt, shots, nrec, abcn, grad=True, strips="fp32", chunks=0, free=False, wgrad=False):
    nz, ny, nx = shape if len(shape) == 3 else (shape[0], 1, shape[1])
    c = {"kind": "prop", "eq": eq, "order": order, "nz": nz, "ny": ny, "nx": nx, "nt": nt, "shots": shots,
         "nrec": nrec, "abcn": abcn, "grad": grad, "strips": strips, "chunks": chunks, "free": free, "wgrad": wgrad}
    return dict(c, name=name) if name else c


def _conv_case(name, n, h, w, cin, cout):
    c = {"kind": "conv", "n": n, "h": h, "w": w, "cin": cin, "cout": cout}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a single small shot, where the latency of a step counts (the 96 x 128 two-layer workload)
        _case("acoustic2d_one_shot", "acoustic2d", 8, (96, 128), 800, 1, 1, 20),
        # records of a few shots on a small odd grid at the default order and layer width; the smallest call
        _case("acoustic2d_records_o4", "acoustic2d", 4, (151, 203), 400, 4, 101, 50, grad=False),
        # the 32-shot survey gradient
        _case("acoustic2d_survey", "acoustic2d", 8, (256, 768), 256, 32, 384, 40),
        # the same grid at the equations' default order, with the wavelet's gradient
        _case("acoustic2d_survey_o4", "acoustic2d", 4, (256, 768), 256, 16, 384, 40, wgrad=True),
        # the 3-D survey gradient, one group of three shots; the largest call
        _case("acoustic3d_survey", "acoustic3d", 8, (256, 256, 256), 64, 3, 4096, 24),
        # an odd 3-D grid at the default order
        _case("acoustic3d_o4", "acoustic3d", 4, (101, 119, 141), 160, 2, 529, 20),
        # the elastic survey gradient
        _case("elastic2d_survey", "elastic2d", 8, (400, 1200), 128, 16, 600, 40),
        # land data: a traction-free top face, odd grid, default order
        _case("elastic2d_free_o4", "elastic2d", 4, (187, 331), 300, 8, 165, 30, free=True),
        # the 3-D elastic survey gradient, two of its shots
        _case("elastic3d_survey", "elastic3d", 8, (128, 128, 128), 48, 2, 1024, 16),
        # the VTI survey gradient on the elastic grid at the default order
        _case("vti2d_survey_o4", "vti2d", 4, (400, 1200), 96, 16, 600, 40),
        # the 3-D VTI survey gradient at the default order
        _case("vti3d_survey_o4", "vti3d", 4, (128, 128, 128), 64, 4, 1024, 16),
        # the U-Net's second level in training: 16 inputs of 128 x 384, 64 channels at half resolution
        _conv_case("unet_conv_64", 16, 64, 192, 64, 64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(c):
    m = c["order"] // 2
    e = 2 * (c["abcn"] + m)
    top = c["abcn"] if c["free"] else 0
    y = c["ny"] + e if EQS[c["eq"]]["nd"] == 3 else 1
    return (c["nz"] + e - top) * y * (c["nx"] + e)


def draw(rng):
    """One more case: an equation at one of its orders on a grid, shot count
    and time axis of the listed cases' ranges, or a layer of the U-Net."""
    kind = rng.choice(["acoustic2d", "acoustic2d", "acoustic3d", "acoustic3d", "elastic2d", "elastic2d",
                       "elastic3d", "vti2d", "vti3d", "conv"])
    if kind == "conv":
        level = rng.randrange(4)
        base = 32 << level
        cin, cout = rng.choice([(base, base), (base, base), (3 * base if level < 3 else base // 2, base),
                                (8 if level == 0 else base // 2, base)])
        return _conv_case("", rng.randint(2, 16), 128 >> level, 8 * rng.randint(12, 48) >> level, cin, cout)
    q = EQS[kind]
    order = rng.choice([4, 8] if kind != "vti2d" and kind != "vti3d" else [4, 4, 8])
    if rng.random() < 0.2:
        order = rng.choice([2, 6] if kind == "elastic3d" else [2, 6, 10, 12])
    if q["nd"] == 2:
        shape = (_log(rng, 60, 400), _log(rng, 90, 1200))
        shots, nrec, abcn, nt = _log(rng, 1, 32), _log(rng, 1, 600), rng.choice([20, 30, 40, 50]), rng.randint(150, 600)
    else:
        top = 200 if kind == "acoustic3d" else 128
        shape = tuple(_log(rng, 40, top) for _ in range(3))
        shots, nrec, abcn, nt = _log(rng, 1, 4), _log(rng, 1, 4096), rng.choice([10, 16, 20, 24]), rng.randint(80, 200)
    grad = rng.random() < 0.8
    strips, chunks = "fp32", 0
    if grad and ((order == 8 and kind in ("acoustic2d", "acoustic3d", "elastic2d")) or kind == "elastic3d"):
        if rng.random() < 0.25:
            strips = rng.choice(["fp16", "bf16", "int8"])
        elif rng.random() < 0.15:
            chunks = rng.choice([25, 100])
    free = kind in ("acoustic2d", "acoustic3d", "elastic2d", "elastic3d") and rng.random() < 0.2
    wgrad = grad and kind.startswith("acoustic") and rng.random() < 0.2
    c = _case("", kind, order, shape, nt, shots, nrec, abcn, grad, strips, chunks, free, wgrad)
    most = 0.15 * q["rate"]
    while _cells(c) * c["shots"] * c["nt"] > most and c["shots"] > 1:
        c["shots"] -= 1
    c["nt"] = max(80, min(c["nt"], int(most / (_cells(c) * c["shots"]))))
    return c


# ------------------------------------------------------------------ inputs
H = 10.0                      # grid spacing, m
VMIN, VMAX = 1500.0, 4500.0


def _dt(c):
    return EQS[c["eq"]]["courant"] * H / VMAX


def _shape(c):
    return (c["nz"], c["ny"], c["nx"]) if EQS[c["eq"]]["nd"] == 3 else (c["nz"], c["nx"])


def _ricker(t, f):
    a = (math.pi * f * t) ** 2
    return (1.0 - 2.0 * a) * np.exp(-a)


F0 = VMIN / (6.0 * H)         # six cells per shortest dominant wavelength
DELAY = 1.0 / F0


def _models(c, rng):
    """Layers of rising velocity with an undulating depth and a smooth
    anomaly; the equation's other models follow from the velocity."""
    shape = _shape(c)
    nz = shape[0]
    grid = [torch.arange(n, dtype=torch.float64, device=DEVICE) for n in shape]
    z, x = grid[0], grid[-1]
    lat = 6.0 * torch.sin(2 * math.pi * rng.uniform(0.5, 2.0) * x / shape[-1] + rng.uniform(0, 6.0))
    if len(shape) == 3:
        lat = lat[None, :] + 4.0 * torch.sin(2 * math.pi * rng.uniform(0.5, 2.0) * grid[1] / shape[1])[:, None]
    vp = torch.full(shape, VMIN, dtype=torch.float64, device=DEVICE)
    depths = np.sort(rng.uniform(0.1, 0.95, 8)) * nz
    for d in depths:
        arg = (z.view((-1,) + (1,) * (len(shape) - 1)) + 0.05 * lat[None] * math.sqrt(nz) - d) / 3.0
        vp += rng.uniform(0.6, 1.0) * (0.8 * (VMAX - VMIN) / 8) * torch.sigmoid(arg)
    r2 = torch.zeros((1,) * len(shape), dtype=torch.float64, device=DEVICE)
    for a, g in enumerate(grid):
        view = [1] * len(shape)
        view[a] = -1
        r2 = r2 + ((g - rng.uniform(0.35, 0.65) * shape[a]) / (0.12 * shape[a])).view(view) ** 2
    vp += rng.uniform(0.05, 0.15) * (VMAX - VMIN) * torch.exp(-0.5 * r2)
    vp = vp.clamp(VMIN, VMAX)
    rho = 310.0 * vp ** 0.25
    if c["eq"].startswith("elastic"):
        out = [vp, vp / 1.73, rho]
    elif c["eq"].startswith("vti"):
        eps = 0.05 + 0.15 * (vp - VMIN) / (VMAX - VMIN)
        out = [vp, eps, 0.5 * eps, rho]
    else:
        out = [vp]
    return [m.to(torch.float32) for m in out]


def _geometry(c, rng):
    """Sources spread along the surface, each with a spread of receivers
    around it that its waves reach; coordinates are (x[, y], z)."""
    shape = _shape(c)
    B, n = c["shots"], c["nrec"]
    reach = max(8, int(0.3 * EQS[c["eq"]]["courant"] * c["nt"]), int(n ** (1.0 / (len(shape) - 1))))
    src, rec = [], []
    for size in (shape[-1],) if len(shape) == 2 else (shape[-1], shape[1]):
        s = np.sort(rng.integers(2, size - 2, B)) if not src else rng.integers(2, size - 2, B)
        lo, hi = np.maximum(0, s - reach), np.minimum(size - 1, s + reach)
        r = lo[:, None] + np.floor(rng.random((B, n)) * (hi - lo + 1)[:, None]).astype(np.int64)
        src.append(s)
        rec.append(np.sort(r, axis=1) if not rec else r)
    src.append(np.full(B, 3))
    rec.append(np.full((B, n), 2))
    return np.stack(src, -1).astype(np.int64), np.stack(rec, -1).astype(np.int64)


def _inputs(c, seed):
    rng = np.random.default_rng(seed)
    models = _models(c, rng)
    src, rec = _geometry(c, rng)
    t = np.arange(c["nt"]) * _dt(c)
    wavelet = _ricker(t - DELAY, F0 * rng.uniform(0.8, 1.0)).astype(np.float32)
    obs = None
    if c["grad"]:
        # a direct arrival and two reflections on every trace
        nf = len(EQS[c["eq"]]["cls"].RECEIVER_FIELDS)
        dist = np.sqrt((((rec - src[:, None, :]) * H) ** 2).sum(-1)) + H
        scale = np.sqrt(H / dist) if len(_shape(c)) == 2 else 0.5 * H / dist
        if not c["eq"].startswith("acoustic"):
            scale = scale / (2200.0 * VMIN)
        tt = torch.from_numpy(t).to(DEVICE)[None, :, None]
        obs = torch.zeros((c["shots"], c["nt"], c["nrec"], nf), dtype=torch.float64, device=DEVICE)
        for k, refl in enumerate((1.0, 0.4, -0.3)):
            depth = 0.0 if k == 0 else rng.uniform(0.02, 0.2) * c["nz"] * H
            v = rng.uniform(VMIN, 1.3 * VMIN)
            at = torch.from_numpy(np.sqrt(dist ** 2 + 4 * depth ** 2) / v + DELAY).to(DEVICE)[:, None, :]
            arg = (math.pi * F0 * (tt - at)) ** 2
            pulse = refl * torch.from_numpy(scale).to(DEVICE)[:, None, :] * (1.0 - 2.0 * arg) * torch.exp(-arg)
            for f in range(nf):
                obs[..., f] += (1.0 if f == nf - 1 else 0.5) * pulse
        obs = obs.to(torch.float32)
    return models, src, rec, torch.from_numpy(wavelet).to(DEVICE), obs


def prepare(case, seed):
    if case["kind"] == "conv":
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        n, h, w, ci, co = (case[k] for k in ("n", "h", "w", "cin", "cout"))
        x = F.gelu(torch.randn((n, h, w, ci), generator=g, device=DEVICE)).to(torch.bfloat16).requires_grad_()
        bound = math.sqrt(6.0 / (9 * ci))
        wt = ((torch.rand((co, 3, 3, ci), generator=g, device=DEVICE) * 2 - 1) * bound).requires_grad_()
        b = (0.1 * torch.randn(co, generator=g, device=DEVICE)).requires_grad_()
        gout = torch.randn((n, h, w, co), generator=g, device=DEVICE) * (1.0 / (h * w))
        return {"case": case, "x": x, "w": wt, "b": b, "gout": gout}
    c = case
    models, src, rec, wavelet, obs = _inputs(c, seed)
    memory = sb.Ckpt(chunks=c["chunks"]) if c["chunks"] else sb.BoundarySaving(storage_dtype=c["strips"])
    eq = EQS[c["eq"]]["cls"](spatial_order=c["order"], device=DEVICE)
    solver = sb.PropTorch(eq, shape=_shape(c), dh=H, dt=_dt(c), abcn=c["abcn"], device=DEVICE, memory=memory,
                          free_surface=bool(c["free"]))
    if c["grad"]:
        models = [m.requires_grad_() for m in models]
        wavelet = wavelet.requires_grad_(bool(c["wgrad"]))
    return {"case": case, "solver": solver, "models": models, "src": src, "rec": rec, "wavelet": wavelet, "obs": obs}


def run(state):
    case = state["case"]
    if case["kind"] == "conv":
        x, w, b = state["x"], state["w"], state["b"]
        x.grad = w.grad = b.grad = None
        y = unet.conv3x3(x, w, b)
        y.backward(state["gout"])
        return {"y": y.detach(), "gx": x.grad, "gw": w.grad, "gb": b.grad}
    models, wavelet = state["models"], state["wavelet"]
    if not case["grad"]:
        with torch.no_grad():
            return {"record": state["solver"](wavelet, state["src"], state["rec"], models=models)}
    for m in models:
        m.grad = None
    wavelet.grad = None
    pred = state["solver"](wavelet, state["src"], state["rec"], models=models)
    loss = 0.5 * ((pred - state["obs"]) ** 2).sum()
    loss.backward()
    out = {"record": pred.detach(), "grads": [m.grad for m in models]}
    if case["wgrad"]:
        out["gwavelet"] = wavelet.grad
    return out


# ------------------------------------------------------- work and tolerance
def work(case):
    """Convolution: operands and results once, three products.  Propagation:
    per cell and step of the runtime grid, each field of the state read and
    written once in the forward, and in the reverse the same for the
    reconstructed and for the adjoint fields, and each gradient read and
    written; models and the layers' memories are not counted."""
    if case["kind"] == "conv":
        n, h, w, ci, co = (case[k] for k in ("n", "h", "w", "cin", "cout"))
        px = n * h * w
        by = px * ci * 2 + 9 * ci * co * 4 + px * co * 4        # forward
        by += px * co * 4 + px * ci * 2 + 9 * ci * co * 4        # backward: cotangent, gx, gw
        return {"bytes": by, "flops": 3 * 2 * px * 9 * ci * co}
    q = EQS[case["eq"]]
    nd = q["nd"]
    fields = {"acoustic2d": 1, "acoustic3d": 1, "elastic2d": 5, "elastic3d": 9, "vti2d": 4, "vti3d": 5}[case["eq"]]
    acoustic = case["eq"].startswith("acoustic")
    # leapfrog: two levels read, one written; staggered: each field read and written
    fwd = 3 if acoustic else 2 * fields
    rev = 2 * fwd + 2 * q["models"]
    cells = _cells(case) * case["shots"]
    if acoustic:
        flops = nd * 3 * case["order"]
    else:
        flops = (2 * nd * nd if "elastic" in case["eq"] else 2 * nd) * 2 * case["order"]
    steps = case["nt"]
    by = cells * steps * 4 * (fwd + (rev if case["grad"] else 0))
    return {"bytes": by, "flops": cells * steps * flops * (3 if case["grad"] else 1)}


def tolerance(case):
    """About four times what the float32 runs differ from 64 bits, or by a
    change of the order of the sums; reduced strips add the rounding of their
    codes, which a last-bit difference of a value can flip."""
    if case["kind"] == "conv":
        return {"rel": 1e-2, "max": 0.2}
    if case["strips"] != "fp32":
        return {"rel": {"bf16": 2e-3, "fp16": 2e-4, "int8": 5e-3}[case["strips"]], "max": 0.5}
    return {"rel": 2e-5 if case["eq"].startswith("acoustic") else 1e-4, "max": 4e-3}


# ------------------------------------------------ the same in 64 bits (torch)
def _centred(m, second):
    """Weights k = 1..m of the centred first or second derivative; the second
    derivative's in float32 with the last one closing the sum (the tables of
    the float32 stencils)."""
    out = []
    for k in range(1, m + 1):
        w = Fraction((-1) ** (k + 1) * math.factorial(m) ** 2, math.factorial(m - k) * math.factorial(m + k))
        out.append(2 * w / (k * k) if second else w / k)
    vals = [float(np.float32(float(x))) for x in out]
    if second:
        vals[-1] = float(np.float32(float(2 * sum(out)))) / 2 - sum(vals[:-1])
    return vals


def _staggered(m):
    out = []
    for i in range(1, m + 1):
        w = Fraction((-1) ** (i + 1), 2 * i - 1)
        for n in range(1, m + 1):
            if n != i:
                num = (2 * n - 1) ** 2
                w *= abs(Fraction(num, num - (2 * i - 1) ** 2))
        out.append(float(np.float32(float(w))))
    return out


def _damping(n, m, lo, hi, dt, offset):
    """(a, b) of one axis: a = exp(-(sigma + alpha) dt), b = sigma / (sigma +
    alpha) (a - 1) in a layer of lo / hi cells, zero outside."""
    sigma0 = -3.0 * VMAX_PML * math.log(1e-3) / (2 * max(lo, hi) * H)
    x = np.arange(n) + offset
    frac = np.zeros(n)
    if lo:
        frac = np.maximum(frac, (m + lo - x) / lo)
    if hi:
        frac = np.maximum(frac, (x - (n - 1 - m - hi)) / hi)
    frac = np.clip(frac, 0.0, 1.0)
    sigma, alpha = sigma0 * frac ** 2, math.pi * F_PML * (1.0 - frac)
    a = np.exp(-(sigma + alpha) * dt)
    b = sigma / (sigma + alpha) * (a - 1.0)
    a[frac == 0] = 0.0
    return a, b


VMAX_PML, F_PML = 4500.0, 25.0      # the call's default max_vel and pml_freq


class _Exact:
    """A propagator in 64 bits on the cells that a step updates (the runtime
    grid without its outermost stencil halo, which stays zero): ``step(state,
    models, amplitude)`` is one time step, differentiated by autograd."""

    def __init__(self, c, src, rec):
        self.c, q = c, EQS[c["eq"]]
        self.nd, self.m, self.dt = q["nd"], c["order"] // 2, _dt(c)
        self.src, self.rec = src, rec
        self.shape = _shape(c)
        pads = [(0 if c["free"] and a == 0 else c["abcn"], c["abcn"]) for a in range(self.nd)]
        self.pads = pads
        self.core = tuple(n + lo + hi for n, (lo, hi) in zip(self.shape, pads))
        self.acoustic = c["eq"].startswith("acoustic")
        m = self.m
        self.prof = []
        for a, (lo, hi) in enumerate(pads):
            n = self.core[a] + 2 * m
            view = [1] * (self.nd + 1)
            view[a + 1] = -1

            def put(v):
                return torch.from_numpy(v[m:n - m].astype(np.float32).astype(np.float64)).to(DEVICE).view(view)

            pa, pb = _damping(n, m, lo, hi, self.dt, 0.0)
            pa, pb = pa.astype(np.float32).astype(np.float64), pb.astype(np.float32).astype(np.float64)
            if self.acoustic:
                db = np.gradient(pb, H)
                self.prof.append((put(pa), put(pb), put(db)))
            else:
                ha, hb = _damping(n, m, lo, hi, self.dt, 0.5)
                self.prof.append((put(pa), put(pb), put(ha), put(hb)))
        self.lap, self.grad, self.stag = _centred(m, True), _centred(m, False), _staggered(m)
        # staggered equations damp outside the physical box (3-D elastic: also its outermost cells)
        inner = 1 if c["eq"] == "elastic3d" else 0
        box = torch.ones((1,) + self.core, dtype=torch.float64, device=DEVICE)
        box[(slice(None),) + tuple(slice(lo + inner, n - hi - inner) for n, (lo, hi) in zip(self.core, pads))] = 0.0
        self.layer = box
        at = [torch.arange(c["shots"], device=DEVICE)]
        for a in range(self.nd):
            at.append(torch.from_numpy(self.src[:, self.nd - 1 - a] + pads[a][0]).to(DEVICE))
        self.src_at = tuple(at)
        at = [torch.arange(c["shots"], device=DEVICE)[:, None]]
        for a in range(self.nd):
            at.append(torch.from_numpy(self.rec[:, :, self.nd - 1 - a] + pads[a][0]).to(DEVICE))
        self.rec_at = tuple(at)
        e = c["eq"]
        if self.acoustic:
            self.nfield = 2 + 2 * self.nd
        elif e == "elastic2d":
            self.names, self.nmem, self.out = ["vx", "vz", "sxx", "szz", "sxz"], 8, ["vx", "vz"]
            self.into = ["sxx", "szz"]
        elif e == "elastic3d":
            self.names = ["vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz"]
            self.nmem, self.out, self.into = 18, ["vx", "vy", "vz"], ["sxx", "syy", "szz"]
        else:
            self.names = ["vx", "vz", "sh", "sv"] if self.nd == 2 else ["vx", "vy", "vz", "sh", "sv"]
            self.nmem, self.out, self.into = 2 * self.nd, ["vz"], ["sh", "sv"]

    def zero(self):
        n = self.nfield if self.acoustic else len(self.names) + self.nmem
        z = torch.zeros((self.c["shots"],) + self.core, dtype=torch.float64, device=DEVICE)
        return [z.clone() for _ in range(n)]

    def pad(self, model):
        """A model on the updated cells: its edge values out to the layers."""
        w = []
        for lo, hi in reversed(self.pads):
            w += [lo, hi]
        x = model.to(torch.float64)[None, None]
        return F.pad(x, w, mode="replicate")[0]

    def crop(self, g):
        return g[(0,) + tuple(slice(lo, n - hi) for n, (lo, hi) in zip(self.core, self.pads))]

    def _taps(self, u, axis):
        """u moved by k = -m..m cells along the axis, zero from outside."""
        w = [0, 0] * (self.nd - 1 - axis) + [self.m, self.m]
        p, n = F.pad(u, w), u.shape[axis + 1]
        return lambda k: p.narrow(axis + 1, self.m + k, n)

    def _lap(self, u, axis):
        t = self._taps(u, axis)
        return sum(w * ((t(-k) - u) + (t(k) - u)) for k, w in enumerate(self.lap, 1)) / (H * H)

    def _grad(self, u, axis):
        t = self._taps(u, axis)
        return sum(w * (t(k) - t(-k)) for k, w in enumerate(self.grad, 1)) / H

    def _plus(self, u, axis):
        t = self._taps(u, axis)
        return sum(w * (t(k) - t(1 - k)) for k, w in enumerate(self.stag, 1)) / H

    def _minus(self, u, axis):
        t = self._taps(u, axis)
        return sum(w * (t(k - 1) - t(-k)) for k, w in enumerate(self.stag, 1)) / H

    def derived(self, models):
        """What the steps take of the models."""
        e = self.c["eq"]
        if self.acoustic:
            return [(models[0] * self.dt) ** 2]
        if e.startswith("elastic"):
            vp, vs, rho = models
            mu = rho * vs * vs
            return [self.dt / rho, rho * vp * vp - 2.0 * mu, mu]
        vp, eps, dlt, rho = models
        c33 = rho * vp * vp
        return [self.dt / rho, c33 * (1 + 2 * eps), c33 * torch.sqrt(1 + 2 * dlt), c33]

    def step(self, state, models, amp):
        new = self._acoustic(state, models) if self.acoustic else self._first_order(state, models)
        for f in ([1] if self.acoustic else [self.names.index(n) for n in self.into]):
            new[f] = new[f].index_put(self.src_at, amp, accumulate=True)
        rec = [new[1]] if self.acoustic else [new[self.names.index(n)] for n in self.out]
        return new, torch.stack([r[self.rec_at] for r in rec], -1)

    def _acoustic(self, state, models):
        prev, u = state[:2]
        psi, zeta = list(state[2:2 + self.nd]), list(state[2 + self.nd:])
        w = 0.0
        for a in range(self.nd):
            pa, pb, db = self.prof[a]
            lu, du = self._lap(u, a), self._grad(u, a)
            if self.nd == 2:
                dap = self._grad(pa * psi[a], a)
            else:
                dap = pa * self._grad(psi[a], a) + self._da(a) * psi[a]
            tmp = (1 + pb) * lu + db * du + dap
            w = w + (1 + pb) * tmp + pa * zeta[a]
            psi[a] = pb * du + pa * psi[a]
            zeta[a] = pb * tmp + pa * zeta[a]
        return [u, 2 * u - prev + self.derived(models)[0] * w] + psi + zeta

    def _da(self, axis):
        """d a / d axis; the profile holds its edge values past the cells."""
        pa, m = self.prof[axis][0], self.m
        lo, hi = self.pads[axis]
        n = self.core[axis] + 2 * m
        full = torch.from_numpy(_damping(n, m, lo, hi, self.dt, 0.0)[0].astype(np.float32).astype(np.float64)).to(DEVICE)
        k = n - 2 * m
        d = sum(w * (full[m + i:m + i + k] - full[m - i:m - i + k]) for i, w in enumerate(self.grad, 1)) / H
        return d.view(pa.shape)

    def _first_order(self, state, models):
        """Velocities from the stresses, then the stresses from the new
        velocities; every derivative passes through its layer memory."""
        names, nd = self.names, self.nd
        f = dict(zip(names, state))
        mem = list(state[len(names):])
        buoy, *stiff = self.derived(models)
        count = [0]
        axis = {"x": nd - 1, "y": 1, "z": 0}

        def d(name, ax, plus):
            a = axis[ax]
            g = self._plus(f[name], a) if plus else self._minus(f[name], a)
            pa, pb = self.prof[a][2:] if plus else self.prof[a][:2]
            i = count[0]
            count[0] += 1
            mem[i] = self.layer * (pa * mem[i] + pb * g)
            return g + mem[i]

        if self.c["eq"].startswith("vti"):
            lat = ["x"] if nd == 2 else ["x", "y"]
            for ax in lat:
                f["v" + ax] = f["v" + ax] + buoy * d("sh", ax, True)
            f["vz"] = f["vz"] + buoy * d("sv", "z", True)
            dh = sum(d("v" + ax, ax, False) for ax in lat)
            dz = d("vz", "z", False)
            c11, c13, c33 = stiff
            f["sh"] = f["sh"] + self.dt * (c11 * dh + c13 * dz)
            f["sv"] = f["sv"] + self.dt * (c13 * dh + c33 * dz)
        else:
            axes = ["x", "z"] if nd == 2 else ["x", "y", "z"]
            lam, mu = stiff

            def s(i, j):
                return "s" + "".join(sorted((i, j)))

            new = {}
            for i in axes:
                new["v" + i] = f["v" + i] + buoy * sum(d(s(i, j), j, i == j) for j in axes)
            f.update(new)
            diag = {i: d("v" + i, i, False) for i in axes}
            div = sum(diag.values())
            for i in axes:
                f[s(i, i)] = f[s(i, i)] + self.dt * (lam * div + 2 * mu * diag[i])
            for n, i in enumerate(axes):
                for j in axes[n + 1:]:
                    f[s(i, j)] = f[s(i, j)] + self.dt * mu * (d("v" + i, j, True) + d("v" + j, i, True))
        return [f[n] for n in names] + mem


def _free_elastic(c):
    return c["free"] and c["eq"].startswith("elastic")


def exact(case, seed):
    if case["kind"] == "conv":
        s = prepare(case, seed)
        x, w, b = (s[k].detach().double().requires_grad_() for k in ("x", "w", "b"))
        y = F.conv2d(x.permute(0, 3, 1, 2), w.permute(0, 3, 1, 2), b, padding=1).permute(0, 2, 3, 1)
        gx, gw, gb = torch.autograd.grad(y, (x, w, b), s["gout"].double())
        return {"y": y.detach(), "gx": gx, "gw": gw, "gb": gb}
    # too long in 64 bits, or the image method of a traction-free face
    big = _cells(case) * case["shots"] * case["nt"]
    if _free_elastic(case) or big > (3e9 if case["eq"].startswith("acoustic") else 1.4e9):
        return None
    models, src, rec, wavelet, obs = _inputs(case, seed)
    e = _Exact(case, src, rec)
    full = [e.pad(m) for m in models]
    amp = wavelet.double()[None, :].expand(case["shots"], -1)
    nt = case["nt"]
    every = max(1, int(math.sqrt(nt)))
    with torch.no_grad():
        state, kept, recs = e.zero(), [], []
        for it in range(nt):
            if it % every == 0:
                kept.append([x.clone() for x in state])
            state, r = e.step(state, full, amp[:, it])
            recs.append(r)
    record = torch.stack(recs, 1)
    if not case["grad"]:
        return {"record": record}
    cot = record - obs.double()
    adj = [torch.zeros_like(x) for x in state]
    gm = [torch.zeros_like(m) for m in full]
    gw = torch.zeros(nt, dtype=torch.float64, device=DEVICE)
    del state, recs
    for seg in reversed(range(len(kept))):
        lo, hi = seg * every, min(nt, (seg + 1) * every)
        chain = [kept.pop()]
        with torch.no_grad():
            for it in range(lo, hi - 1):
                chain.append(e.step(chain[-1], full, amp[:, it])[0])
        for it in reversed(range(lo, hi)):
            ins = [x.detach().requires_grad_() for x in chain.pop()]
            ms = [m.detach().requires_grad_() for m in full]
            a = amp[:, it].detach().clone().requires_grad_()
            new, r = e.step(ins, ms, a)
            got = torch.autograd.grad(new + [r], ins + ms + [a], adj + [cot[:, it]], allow_unused=True)
            adj = [torch.zeros_like(x) if g is None else g for g, x in zip(got, ins)]
            for k in range(len(gm)):
                g = got[len(ins) + k]
                if g is not None:
                    gm[k] += g
            gw[it] = got[-1].sum()
            del new, r, ins, got
    out = {"record": record, "grads": [e.crop(g) for g in gm]}
    if case["wgrad"]:
        out["gwavelet"] = gw
    return out
