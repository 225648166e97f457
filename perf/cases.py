"""The work that a user of this framework has it do, as timed cases.

Every case is a frame (or a batch of frames) of a linear array: RF lines of a few dozen
point scatterers plus noise, the imaging grid, the band, window and F-number of a plan, and
one call of a public entry point.  ``listed()`` holds the fixed cases, ``draw(rng)`` one
more of the same ranges, ``prepare`` / ``run`` the call itself, ``work`` what it cannot do
without and ``exact`` its result in 64 bits from plain torch.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from f_number_gb300 import autograd as fauto
from f_number_gb300 import das, f_numbers, windows

C0 = 1540.0
FILL = 0.918          # element width over pitch
DEV = "cuda"


def listed():
    base = {"ne": 128, "na": 11, "nt": 2048, "fs": 20e6, "pitch": 0.3048e-3, "f_lo": 2e6, "f_hi": 7e6,
            "window": "hann", "par": 0.0, "F": "angle_lb", "norm": "on", "t0": 0.0, "f64": False, "stack": False,
            "max_deg": 10.0}

    def c(name, kind, **kw):
        return dict(base, name=name, kind=kind, **kw)

    return [
        # one plane wave into a small region of interest, e.g. a tracking gate: launches and latency count
        c("pw_roi_64el", "plan", ne=64, na=1, nt=1024, nx=48, nz=57, dx=0.1007e-3, dz=0.1009e-3),
        # a single 0 degree plane wave over the whole field (the reference's own call pattern)
        c("pw_single_256", "plan", na=1, nx=256, nz=256, dx=0.1176e-3, dz=0.1569e-3, f_lo=2.25e6, f_hi=6.75e6,
          window="tukey", par=0.5),
        # the headline: 11 compounded angles on 512 x 512 voxels
        c("cpwc_11_512", "plan", nx=512, nz=512, dx=0.06e-3, dz=0.06e-3),
        # fast compounding on a ragged grid, double RF with a start time, boxcar, sums not normalised
        c("cpwc_5_boxcar_f64", "plan", ne=96, na=5, nt=1024, nx=203, nz=321, dx=0.13e-3, dz=0.077e-3,
          window="boxcar", F="constant", norm="off", t0=16.0, f64=True),
        # a long array with many angles (the largest frames of the batch workload)
        c("cpwc_31_192el", "plan", ne=192, na=31, nt=4096, nx=301, nz=451, dx=0.12e-3, dz=0.061e-3,
          window="tukey", par=0.2),
        # one image per angle, kept apart for the caller's own angular weighting
        c("pw_stack_11", "plan", nx=161, nz=224, dx=0.1507e-3, dz=0.1003e-3, stack=True),
        # das_pw on host arrays with the reference's defaults, one angle per call
        c("host_das_pw", "host", na=1, nx=256, nz=384, dx=0.1013e-3, dz=0.0807e-3, window="tukey", par=0.2, f64=True,
          max_deg=5.0),
        # full synthetic aperture, 128 x 128 elements, directivity F-number and boxcar windows
        c("saft_128_boxcar", "saft", na=1, nt=3072, fs=40e6, pitch=0.3e-3, nx=400, nz=400, dx=0.0952e-3,
          dz=0.0927e-3, window="boxcar", F="perrot"),
        # a small probe over its whole band, tapered windows, ragged grid
        c("saft_64_hann_fullband", "saft", ne=64, na=1, nt=1536, fs=40e6, pitch=0.3e-3, nx=151, nz=187,
          dx=0.1103e-3, dz=0.1009e-3, f_lo=0.0, f_hi=0.0, window="hann", t0=8.0),
        # image-sharpness gradients with respect to the spectra and the sound speed
        c("sharpness_grad_11", "sharp", nx=256, nz=256, dx=0.12e-3, dz=0.12e-3),
        # forward and backward of the differentiable beamformer under a torch loss
        c("autograd_5", "autograd", ne=96, na=5, nt=1024, nx=150, nz=203, dx=0.1507e-3, dz=0.1003e-3,
          window="tukey", par=0.5),
        # uneven frames in one graph (shapes from shape_seed)
        c("batch_uneven_6", "batch", frames=6, shape_seed=5, side_lo=128, side_hi=400),
    ]


def draw(rng):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["plan", "plan", "plan", "plan", "host", "saft", "sharp", "autograd", "batch"])
    case = dict(listed()[2], kind=kind)
    del case["name"]
    w = rng.choice(["hann", "boxcar", "tukey", "triangular"])
    case.update(window=w, par=rng.choice([0.2, 0.5]) if w == "tukey" else 0.0,
                F=rng.choice(["angle_lb", "angle_lb", "constant", "perrot"]), norm=rng.choice(["on", "on", "on", "off"]),
                t0=rng.choice([0.0, 0.0, 8.0, 16.0]), f64=rng.random() < 0.25)
    if kind == "batch":
        case.update(frames=rng.randint(4, 8), shape_seed=rng.randint(0, 10 ** 6), side_lo=128, side_hi=320,
                    window="hann", par=0.0, F="angle_lb", norm="on", t0=0.0, f64=False)
        return case
    if kind == "saft":
        case.update(ne=rng.randint(32, 128), na=1, nt=rng.choice([1024, 1536, 2048, 3072]), fs=40e6, pitch=0.3e-3,
                    norm="on", f64=False, f_hi=rng.choice([7e6, 9e6]))
    else:
        case.update(ne=rng.choice([64, 96, 128, 192]) - rng.choice([0, 0, 0, 1, 3]), nt=rng.choice([1024, 2048, 4096]),
                    na=rng.choice([1, 1, 2, 3, 5, 7, 11, 16, 31]))
        if kind == "host":
            case.update(na=1, f64=True, window="tukey", par=0.2, F="angle_lb", norm="on", t0=0.0)
        if kind in ("sharp", "autograd"):
            case.update(na=rng.choice([3, 5, 7, 11]), norm="on", f64=False)
        if kind == "plan":
            case["stack"] = case["na"] > 1 and rng.random() < 0.2
    cap = {"saft": 300, "sharp": 256, "autograd": 220, "host": 400}.get(kind, 512)
    lo = 40 if kind == "plan" else 96
    case.update(nx=logu(lo, cap), nz=logu(lo, cap), max_deg=rng.choice([5.0, 10.0, 15.0]))
    case.update(dx=case["pitch"] * case["ne"] * rng.uniform(0.7, 1.0) / case["nx"],
                dz=rng.uniform(10e-3, 35e-3) / case["nz"])
    # no dearer than the listed frames: at most the headline's voxel, element, sample and angle product
    big = 512 * 512 * 128 * 2048 * 11.0
    while case["nx"] * case["nz"] * case["ne"] * case["nt"] * max(case["na"], 1.0) > big:
        case["nx"] = case["nx"] * 4 // 5
        case["dx"] *= 1.25
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _frames(case):
    """The frames of a batch case, each a plane-wave case of its own."""
    r = random.Random(case["shape_seed"])
    out = []
    for _ in range(case["frames"]):
        side = r.randint(case["side_lo"], case["side_hi"])
        out.append(dict(case, kind="plan", ne=r.choice([64, 96, 128, 192]), na=r.choice([1, 5, 11, 31]),
                        nt=r.choice([1024, 2048, 4096]), nx=side, nz=side, dx=case["pitch"] / 5,
                        dz=case["pitch"] / 5))
    return out


def _grid(case):
    px = (np.arange(case["nx"]) - (case["nx"] - 1) / 2.0) * case["dx"]
    pz = (3e-3 if case["kind"] == "saft" else 5e-3) + np.arange(case["nz"]) * case["dz"]
    return px, pz


def _angles(case):
    if case["na"] == 1:
        return np.array([math.radians(3.0) if case["kind"] == "host" else 0.0])
    return np.deg2rad(np.linspace(-case["max_deg"], case["max_deg"], case["na"]))


def _bounds(case):
    return None if case["f_hi"] == 0.0 else [case["f_lo"], case["f_hi"]]


def _window(case):
    if case["window"] == "tukey":
        return windows.tukey(case["par"])
    return {"hann": windows.hann, "boxcar": windows.boxcar, "triangular": windows.triangular}[case["window"]]()


def _f_number(case):
    if case["F"] == "constant":
        return f_numbers.constant(1.0)
    if case["F"] == "perrot":
        return f_numbers.directivity.perrot(FILL)
    return f_numbers.grating.angle_lb(60.0, 1.5)


def _norm(case):
    from f_number_gb300 import normalizations
    return normalizations.on() if case["norm"] == "on" else normalizations.off()


def _rf(case, seed):
    """[signals.., samples] float32 on the GPU: Gaussian-modulated 5 MHz pulses of 48 point
    scatterers of random amplitude at their two-way delays, plus white noise."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    ne, nt, fs = case["ne"], case["nt"], case["fs"]
    px, pz = _grid(case)
    n = 48
    u = torch.rand(2, n, generator=g, device=DEV)
    amp = torch.randn(n, generator=g, device=DEV)
    xs = px[0] + (px[-1] - px[0]) * u[0]
    zs = pz[0] + (pz[-1] - pz[0]) * u[1]
    ctr = torch.tensor(case["pitch"] * (np.arange(ne) - (ne - 1) / 2.0), device=DEV, dtype=torch.float32)
    d_rx = torch.sqrt((ctr[:, None] - xs) ** 2 + zs ** 2)                       # [E, S]
    if case["kind"] == "saft":
        tau = (d_rx[:, None, :] + d_rx[None, :, :]) / C0                        # [tx, rx, S]
    else:
        th = torch.tensor(_angles(case), device=DEV, dtype=torch.float32)
        ex, ez = -torch.sin(th), torch.cos(th)
        M = (ne - 1) / 2.0 * case["pitch"]
        ref = torch.where(ex >= 0, -M, M)
        d_tx = ex[:, None] * (xs[None, :] - ref[:, None]) + ez[:, None] * zs    # [A, S]
        tau = (d_tx[:, None, :] + d_rx[None, :, :]) / C0                        # [A, E, S]
    t = torch.arange(nt, device=DEV, dtype=torch.float32) / fs
    alpha = (math.pi * 5e6 * 0.6) ** 2 / (4.0 * math.log(2.0))
    rf = torch.randn(tau.shape[0], ne, nt, generator=g, device=DEV) * 0.02
    for s in range(n):
        d = t - tau[..., s, None]
        rf += amp[s] * torch.exp(-alpha * d * d) * torch.cos(2.0 * math.pi * 5e6 * d)
    return rf


def _plan(case):
    px, pz = _grid(case)
    p, w = case["pitch"], FILL * case["pitch"]
    if case["kind"] == "saft":
        return das.SAPlan(px, pz, case["nt"], case["ne"], case["fs"], w, p, C0, _bounds(case), case["t0"],
                          _window(case), _window(case), _f_number(case), _f_number(case), _norm(case), _norm(case))
    return das.PWPlan(px, pz, case["nt"], case["ne"], case["fs"], _angles(case), w, p, C0, _bounds(case), case["t0"],
                      _window(case), _f_number(case), _norm(case), compound=not case["stack"])


def _device_rf(case, seed):
    rf = _rf(case, seed)
    return rf.double() if case["f64"] else rf


def _spectra32(case, seed):
    """Band spectra [E, K, A] complex64 of the case's RF (torch's FFT), an input of the
    differentiable beamformer."""
    g = _geometry(case)
    X = torch.fft.rfft(_rf(case, seed).double(), n=g["N"], dim=-1)[..., g["k_lb"]:g["k_ub"] + 1]
    return X.permute(1, 2, 0).to(torch.complex64).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        fr = _frames(case)
        plans = [_plan(f) for f in fr]
        rfs = [_device_rf(f, seed + 101 * i) for i, f in enumerate(fr)]
        images = [torch.empty((1, p.n_x, p.n_z), dtype=torch.complex64, device=DEV) for p in plans]
        return {"kind": kind, "batch": das.Batch(plans, rfs, images, n_streams=4), "images": images}
    if kind == "host":
        px, pz = _grid(case)
        rf = _rf(case, seed)[0].double().cpu().numpy().T.copy()                  # [N_t, N_el]
        return {"kind": kind, "args": (px, pz, rf, case["fs"], float(_angles(case)[0]), FILL * case["pitch"],
                                       case["pitch"], C0, _bounds(case))}
    if kind == "autograd":
        return {"kind": kind, "plan": _plan(case), "X": _spectra32(case, seed),
                "c": torch.tensor(C0 - 8.0, dtype=torch.float64)}
    return {"kind": kind, "plan": _plan(case), "rf": _device_rf(case, seed)}


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].execute()
        return list(state["images"])
    if kind == "host":
        return das.das_pw(*state["args"])
    if kind == "sharp":
        loss, dc, g = state["plan"].sharpness_grad(state["rf"])
        return [loss, dc, g]
    if kind == "autograd":
        X = state["X"].detach().requires_grad_(True)
        c = state["c"].detach().requires_grad_(True)
        image = fauto.pw_beamform(state["plan"], X, c)
        loss = fauto.sharpness(image)
        loss.backward()
        return [image.detach(), loss.detach(), X.grad, c.grad]
    return state["plan"].execute(state["rf"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    if case["kind"] == "batch":
        parts = [work(f) for f in _frames(case)]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    g = _geometry(case)
    nv, ne, K, na = case["nx"] * case["nz"], case["ne"], g["K"], case["na"]
    # mean number of elements in the aperture, over a coarse sample of voxels and bins
    px, pz = _grid(case)
    x = px[np.linspace(0, px.size - 1, 24).astype(int)][:, None, None]
    z = pz[np.linspace(0, pz.size - 1, 24).astype(int)][None, :, None]
    F = g["F"][np.linspace(0, K - 1, 64).astype(int)][None, None, :]
    half = np.where(F > 1.2e-7, z / (2.0 * np.maximum(F, 1e-12)), 1e9)
    lo = np.maximum(np.ceil(g["M"] + (x - half) / case["pitch"]), 0)
    hi = np.minimum(np.floor(g["M"] + (x + half) / case["pitch"]), ne - 1)
    n = np.maximum(hi - lo + 1, 0)
    rf_item = 8 if case["f64"] else 4
    if case["kind"] == "saft":
        return {"bytes": ne * ne * case["nt"] * rf_item + nv * 8, "flops": 8.0 * nv * K * float((n * n).mean())}
    terms = nv * K * na * float(n.mean())
    spectra = ne * K * na * 8
    if case["kind"] == "sharp":      # image and its derivative, then the adjoint
        return {"bytes": na * ne * case["nt"] * rf_item + spectra, "flops": 24.0 * terms}
    if case["kind"] == "autograd":
        return {"bytes": 2 * spectra + nv * 8, "flops": 24.0 * terms}
    n_img = na if case["stack"] else 1
    return {"bytes": na * ne * case["nt"] * rf_item + n_img * nv * 8, "flops": 8.0 * terms}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _geometry(case):
    """DFT order, band bins and the F-number of every bin (das_pw.m and the CUDA gateways)."""
    ne, fs, p = case["ne"], case["fs"], case["pitch"]
    _, pz = _grid(case)
    M = (ne - 1) / 2.0
    ap = np.float32(p * (ne - 1 - M)) - np.float32(p * (0 - M))     # the gateways' float aperture
    ap2 = float(np.float32(ap * ap))
    z1 = float(pz[1] if pz.size > 1 else pz[0])
    pad = int(math.ceil((math.sqrt(ap2 + z1 * z1) - z1) * fs / C0))
    N = case["nt"] + pad + 1 - (case["nt"] + pad) % 2
    lo, hi = (np.finfo(float).tiny, fs / 2.0) if case["f_hi"] == 0.0 else (case["f_lo"], case["f_hi"])
    k_lb, k_ub = int(math.ceil(lo * N / fs)), int(math.floor(hi * N / fs))
    pl = p * np.arange(k_lb, k_ub + 1) * fs / (N * C0)
    return {"N": N, "k_lb": k_lb, "k_ub": k_ub, "K": k_ub - k_lb + 1, "M": M, "F": _f_values(case["F"], pl)}


def _f_values(name, pl):
    if name == "constant":
        return np.ones_like(pl)
    if name == "perrot":
        thr = 10.0 ** (-3.0 / 20.0)
        return np.array([1.0 / (2.0 * math.tan(_brent(
            lambda a, w=FILL * q: abs(math.cos(a) * float(np.sinc(w * math.sin(a))) - thr)))) for q in pl])
    # grating lobes at least 60 degrees off, F at most 1.5, 10 degrees apart
    thr = math.sin(math.radians(60.0))
    lower, upper = 1.0 / (1.0 + thr), 1.0 / (1.0 / math.sqrt(1.0 + 9.0) + thr)
    F = np.zeros_like(pl)
    mid = (pl > lower) & (pl < upper)
    F[mid] = np.sqrt(1.0 / (1.0 / pl[mid] - thr) ** 2 - 1.0) / 2.0
    F[pl >= upper] = 1.5
    s, opc = math.sin(math.radians(10.0)), 1.0 + math.cos(math.radians(10.0))
    D = np.zeros_like(pl)
    a = (pl >= 0.5) & (pl < 1.0 / opc)
    D[a] = np.sqrt(1.0 / (1.0 / pl[a] - 1.0) ** 2 - 1.0) / 2.0
    b = (pl >= 1.0 / opc) & (pl < 1.0 / s)
    D[b] = (np.sqrt(2.0 * opc * pl[b] ** 2 - 1.0) + opc * s * pl[b] ** 2) / (2.0 - 2.0 * s * s * pl[b] ** 2)
    D[pl >= 1.0 / s] = math.inf
    return np.maximum(F, D)


def _brent(f, a=0.0, b=math.pi / 2.0, tol=1e-4):
    """Brent's minimiser (Algorithms for Minimization without Derivatives, 1973), stopped at
    the tolerance that the directivity F-number's definition uses."""
    gold = 0.5 * (3.0 - math.sqrt(5.0))
    x = w = v = a + gold * (b - a)
    fx = fw = fv = f(x)
    step = prev = 0.0
    for _ in range(500):
        m = 0.5 * (a + b)
        t1 = math.sqrt(np.finfo(float).eps) * abs(x) + tol / 3.0
        if abs(x - m) <= 2.0 * t1 - 0.5 * (b - a):
            break
        parabola = False
        if abs(prev) > t1:
            r, q = (x - w) * (fx - fv), (x - v) * (fx - fw)
            p, q = (x - v) * q - (x - w) * r, 2.0 * (q - r)
            if q > 0.0:
                p = -p
            q = abs(q)
            old, prev = prev, step
            if abs(p) < abs(0.5 * q * old) and q * (a - x) < p < q * (b - x):
                parabola = True
                step = p / q
                if x + step - a < 2.0 * t1 or b - x - step < 2.0 * t1:
                    step = math.copysign(t1, m - x)
        if not parabola:
            prev = (a - x) if x >= m else (b - x)
            step = gold * prev
        u = x + (step if abs(step) >= t1 else math.copysign(t1, step))
        fu = f(u)
        if fu <= fx:
            a, b = (x, b) if u >= x else (a, x)
            v, fv, w, fw, x, fx = w, fw, x, fx, u, fu
        else:
            a, b = (u, b) if u < x else (a, u)
            if fu <= fw or w == x:
                v, fv, w, fw = w, fw, u, fu
            elif fu <= fv or v == x or v == w:
                v, fv = u, fu
    return x


class _Field:
    """A block of voxels in 64 bits: per band bin the weights and receive phasors of all elements."""

    def __init__(self, case, ix, geo, c=C0):
        t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=DEV)
        px, pz = _grid(case)
        self.case, self.geo = case, geo
        nz = pz.size
        self.x = t(np.repeat(px[ix], nz))[:, None]
        self.z = t(np.tile(pz, len(ix)))[:, None]
        ctr = case["pitch"] * (np.arange(case["ne"]) - geo["M"])
        self.ctr = t(ctr)
        self.half_w = 0.5 * FILL * case["pitch"]
        self.dx = self.ctr[None, :] - self.x
        self.adx = self.dx.abs()
        self.left = self.dx < 0
        self.e = torch.arange(case["ne"], device=DEV)[None, :]
        self.Ku = case["fs"] / (geo["N"] * c)
        self.u = self.Ku * torch.sqrt(self.dx ** 2 + self.z ** 2)
        if case["kind"] != "saft":
            th = _angles(case)
            ex, ez = -np.sin(th), np.cos(th)
            ref = np.where(ex >= 0, -geo["M"] * case["pitch"], geo["M"] * case["pitch"])
            self.utx = self.Ku * (t(ex)[None, :] * (self.x - t(ref)[None, :]) + t(ez)[None, :] * self.z)
        self.t0 = case["t0"] / geo["N"]

    def phasors(self, u):
        """e^{2 pi i k u} at the band's first bin and the step to the next."""
        k = float(self.geo["k_lb"])
        return torch.polar(torch.ones_like(u), 2.0 * math.pi * torch.remainder(k * u, 1.0)), \
            torch.polar(torch.ones_like(u), 2.0 * math.pi * u)

    def weights(self, kk):
        """(window values [V, E], normaliser [V, 1]) of band bin kk."""
        F, p, ne, M = self.geo["F"][kk], self.case["pitch"], self.case["ne"], self.geo["M"]
        if F > np.finfo(np.float32).eps:
            h = self.z / (2.0 * F)
            lo = torch.ceil(M + (self.x - h) / p).clamp(0, ne)
            hi = torch.floor(M + (self.x + h) / p).clamp(-1, ne - 1)
        else:
            lo, hi = torch.zeros_like(self.x), torch.full_like(self.x, ne - 1)
        inside = torch.where(self.left, self.e >= lo, self.e <= hi)
        Ll = self.x - (self.ctr[lo.long().clamp(max=ne - 1)] - self.half_w)
        Lr = self.ctr[hi.long().clamp(min=0)] + self.half_w - self.x
        u = self.adx / torch.where(self.left, Ll, Lr)
        inside &= u < 1.0
        name, par = self.case["window"], self.case["par"]
        if name == "boxcar":
            w = torch.ones_like(u)
        elif name == "triangular":
            w = 1.0 - u
        elif name == "hann":
            w = 0.5 + 0.5 * torch.cos(math.pi * u)
        else:
            w = torch.where(u <= 1.0 - par, 1.0, 0.5 + 0.5 * torch.cos(math.pi * (u - 1.0 + par) / par))
        w = torch.where(inside, w, 0.0)
        W = w.sum(1, keepdim=True)
        if self.case["norm"] == "on":
            inv = torch.where(W > 0, 1.0 / W, 0.0)
        else:
            inv = (W > 0).double()
        return w, inv


def _blocks(case):
    """Blocks of whole columns, about 60000 voxels x 128 elements at a time."""
    n = max(1, int(60000 * 128 / (case["nz"] * case["ne"])))
    idx = np.arange(case["nx"])
    return [idx[i:i + n] for i in range(0, case["nx"], n)]


def _spectra64(case, seed):
    """[A, E, K] complex128 of the RF as the gateways round it (float)."""
    g = _geometry(case)
    return torch.fft.rfft(_rf(case, seed).double(), n=g["N"], dim=-1)[..., g["k_lb"]:g["k_ub"] + 1].contiguous()


def _pw_image(case, X, c=C0, derivative=False):
    """Per-angle images [A, nx nz] of spectra X [A, E, K]; with `derivative` also dI/dc of the
    compounded image at fixed apertures."""
    g = _geometry(case)
    Xk = X.permute(2, 1, 0).contiguous()                                    # [K, E, A]
    scale = 2.0 / g["N"]
    images, ders = [], []
    for ix in _blocks(case):
        f = _Field(case, ix, g, c)
        R, r = f.phasors(f.u)
        T, t = f.phasors(f.utx + f.t0)
        acc = torch.zeros(f.x.shape[0], case["na"], dtype=torch.complex128, device=DEV)
        der = torch.zeros(f.x.shape[0], dtype=torch.complex128, device=DEV)
        for kk in range(g["K"]):
            w, inv = f.weights(kk)
            A = R * (w * inv)
            G = A @ Xk[kk]
            acc += T * G
            if derivative:
                H = (A * f.u) @ Xk[kk]
                der += (g["k_lb"] + kk) * (T * (f.utx * G + H)).sum(1)
            R *= r
            T *= t
        images.append(acc.T * scale)
        ders.append(der * scale * (-2j * math.pi / c))
    return torch.cat(images, 1), (torch.cat(ders) if derivative else None)


def _pw_adjoint(case, G, c=C0):
    """dL/dX* [E, K, A] of a cotangent G = dL/dI* [nx nz] of the compounded image."""
    g = _geometry(case)
    out = torch.zeros(g["K"], case["ne"], case["na"], dtype=torch.complex128, device=DEV)
    nz = case["nz"]
    for ix in _blocks(case):
        f = _Field(case, ix, g, c)
        R, r = f.phasors(f.u)
        T, t = f.phasors(f.utx + f.t0)
        Gb = G[int(ix[0]) * nz:(int(ix[-1]) + 1) * nz, None]
        for kk in range(g["K"]):
            w, inv = f.weights(kk)
            out[kk] += (R * (w * inv)).conj().T @ (T.conj() * Gb)
            R *= r
            T *= t
    return out.permute(1, 0, 2).contiguous() * (2.0 / g["N"])


def _sharpness(case, X, c):
    """Loss, dL/dc, dL/dX* and the image of the sharpness loss for spectra X [A, E, K]."""
    img, dI = _pw_image(case, X, c, derivative=True)
    I = img.sum(0)
    p = I.real ** 2 + I.imag ** 2
    s2, s4 = p.sum(), (p * p).sum()
    G = -2.0 * I * (p / s2 ** 2 - s4 / s2 ** 3)
    dc = 2.0 * (G.conj() * dI).real.sum()
    return -s4 / s2 ** 2, dc, _pw_adjoint(case, G, c), I


def _saft_image(case, seed):
    g = _geometry(case)
    X = _spectra64(case, seed)                                              # [T, R, K]
    scale = 2.0 / g["N"]
    k = torch.arange(g["k_lb"], g["k_ub"] + 1, device=DEV, dtype=torch.float64)
    ph = 2.0 * math.pi * torch.remainder(k * case["t0"], float(g["N"])) / g["N"]
    rot = torch.polar(torch.ones_like(ph), ph)
    out = []
    for ix in _blocks(case):
        f = _Field(case, ix, g)
        R, r = f.phasors(f.u)
        acc = torch.zeros(f.x.shape[0], dtype=torch.complex128, device=DEV)
        for kk in range(g["K"]):
            w, inv = f.weights(kk)
            A = R * (w * inv)
            Y = A @ X[:, :, kk].T
            acc += rot[kk] * (A * Y).sum(1)
            R *= r
        out.append(acc * scale)
    return torch.cat(out)


def exact(case, seed):
    kind, shape = case["kind"], (case.get("nx"), case.get("nz"))
    if kind == "batch":
        return [_pw_image(f, _spectra64(f, seed + 101 * i))[0].sum(0).reshape(1, f["nx"], f["nz"])
                for i, f in enumerate(_frames(case))]
    if kind == "saft":
        return _saft_image(case, seed).reshape(1, *shape)
    if kind == "sharp":
        loss, dc, g, _ = _sharpness(case, _spectra64(case, seed), C0)
        return [float(loss), float(dc), g]
    if kind == "autograd":
        c = C0 - 8.0
        X = _spectra32(case, seed).to(torch.complex128).permute(2, 0, 1)
        loss, dc, g, I = _sharpness(case, X, c)
        # torch's complex gradient of a real loss is twice dL/dX*
        return [I.reshape(shape), loss, 2.0 * g, dc]
    img, _ = _pw_image(case, _spectra64(case, seed))
    if kind == "host":
        return img[0].reshape(shape).T.cpu().numpy()
    return img.reshape(-1, *shape) if case["stack"] else img.sum(0).reshape(1, *shape)
