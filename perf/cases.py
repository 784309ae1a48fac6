"""The framework's own work, case by case, for timing and comparing two builds of it.

A case is one call (or the pair of calls that a solver's iteration makes) through the
public Python entry points of msot_gb300, at the sizes of this repository's
configurations and benchmark:

  operator   A, its transpose, or both, on images and sinograms that stay on the GPU
             (single frames while a user moves the probe; batches of frames or
             wavelengths; the SIR model; odd batches and grids)
  l2/l1/tv   a whole non-negative reconstruction, the framework's main call
  frames     the analytic path of a recording: pre-processing, backproject_waveeq, dmas_cf
  unet       the warm-start network: prediction, or loss and gradients

The model (plan) of a geometry is kept between states, as a user's program keeps it
between frames.  `exact` restates every path but the TV solve in FP64 on plain torch.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "mb-rec-msot_gb300"))

C = 1500.0            # speed of sound, m/s
FS = 4e7              # sampling rate
RADIUS = 0.040        # arc radius of every probe here, m
EIR_TAPS = 257
FMIN, FMAX = 1e5, 12e6
LAMBDA_L2, LAMBDA_L1, LAMBDA_TV = 1e-2, 1e-3, 5e-3
RAW_CROP = 3          # samples cropped from the raw recordings of `frames`
WINDOW = (2, 300.0, 200.0)  # order, low, margin at the end (preprocess_raw_data's defaults)

# the two probes of the configurations: (detectors, coverage in degrees, samples)
PROBES = {"arc256": (256, 135.0, 2030), "ring512": (512, 270.0, 4096)}


# --- the cases ---------------------------------------------------------------------------
def listed():
    return [
        # one frame at a time: live view while the probe moves, and a single reconstruction
        {"name": "forward_1x128", "kind": "operator", "dir": "forward", "probe": "arc256",
         "n": 128, "batch": 1, "sir": False},
        {"name": "transpose_1x128", "kind": "operator", "dir": "transpose", "probe": "arc256",
         "n": 128, "batch": 1, "sir": False},
        {"name": "l2_1x128", "kind": "l2", "probe": "arc256", "n": 128, "batch": 1, "iters": 50},
        # the benchmark's batch of 64 frames
        {"name": "forward_64x128", "kind": "operator", "dir": "forward", "probe": "arc256",
         "n": 128, "batch": 64, "sir": False},
        {"name": "transpose_64x128", "kind": "operator", "dir": "transpose", "probe": "arc256",
         "n": 128, "batch": 64, "sir": False},
        {"name": "l2_64x128", "kind": "l2", "probe": "arc256", "n": 128, "batch": 64,
         "iters": 50},
        # the large probe and grid, an odd number of frames: A and A^T of one gradient
        {"name": "gradient_13x400", "kind": "operator", "dir": "both", "probe": "ring512",
         "n": 400, "batch": 13, "sir": False},
        {"name": "l1_4x400", "kind": "l1", "probe": "ring512", "n": 400, "batch": 4,
         "iters": 50},
        # one multispectral stack of 28 wavelengths, TV
        {"name": "tv_28x200", "kind": "tv", "probe": "arc256", "n": 200, "batch": 28,
         "iters": 50},
        # the model with the spatial impulse response
        {"name": "sir_8x128", "kind": "operator", "dir": "both", "probe": "arc256", "n": 128,
         "batch": 8, "sir": True},
        # a recording of 64 frames through the analytic path
        {"name": "frames_64x128", "kind": "frames", "probe": "arc256", "n": 128, "batch": 64},
        # the warm start's prediction for the benchmark's batch
        {"name": "unet_64x128", "kind": "unet", "n": 128, "batch": 64, "backward": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operator", "operator", "operator", "l2", "l1", "tv", "sir", "frames",
                       "unet"])
    # the interpolation radius (fov 25.4 mm) stays below 9 samples from 78 pixels up
    if kind == "unet":
        side = 8 * rng.randint(8, 24)
        most = max(1, 64 * 128 * 128 // (side * side))
        back = rng.random() < 0.5
        return {"kind": "unet", "n": side, "batch": _log_int(rng, 1, most // 4 if back else most),
                "backward": back}
    if kind == "sir":
        n = _log_int(rng, 78, 160)
        most = max(1, 8 * 128 * 128 // (n * n))
        return {"kind": "operator", "dir": rng.choice(["forward", "transpose", "both"]),
                "probe": "arc256", "n": n, "batch": rng.randint(1, most), "sir": True}
    if kind == "frames":
        n = _log_int(rng, 78, 200)
        most = max(1, min(64, 64 * 128 * 128 // (n * n)))
        return {"kind": "frames", "probe": "arc256", "n": n, "batch": _log_int(rng, 1, most)}
    probe = "ring512" if rng.random() < 0.25 else "arc256"
    n = _log_int(rng, 150, 400) if probe == "ring512" else _log_int(rng, 78, 256)
    pairs = n * n * PROBES[probe][0]
    if kind == "operator":
        most = max(1, min(64, 13 * 400 * 400 * 512 // pairs))
        return {"kind": "operator", "dir": rng.choice(["forward", "transpose", "both"]),
                "probe": probe, "n": n, "batch": _log_int(rng, 1, most), "sir": False}
    if kind == "tv":
        n = _log_int(rng, 78, 200)
        most = max(1, min(28, 28 * 200 * 200 // (n * n)))
        return {"kind": "tv", "probe": "arc256", "n": n, "batch": rng.randint(1, most),
                "iters": rng.randint(10, 50)}
    most = max(1, min(64, 4 * 400 * 400 * 512 // pairs))
    return {"kind": kind, "probe": probe, "n": n, "batch": _log_int(rng, 1, most),
            "iters": rng.randint(10, 50)}


# --- states ------------------------------------------------------------------------------
def _axis(n):
    h = 0.2e-3 * 127 / 2
    return np.linspace(-h, h, n)


def _eir():
    """Gaussian-modulated cosine: 5 MHz, 60 % bandwidth at -6 dB, one zero appended."""
    a = -(math.pi * 5e6 * 0.6) ** 2 / (4.0 * math.log(10.0 ** (-6.0 / 20.0)))
    t = (np.arange(256) - 128) / FS
    return np.concatenate([np.exp(-a * t * t) * np.cos(2 * math.pi * 5e6 * t), [0.0]])


def _norm(probe, n, sir):
    """Normalisation factor of a geometry (largest singular value within some per cent),
    given to the model as a program does that has estimated it once."""
    if sir:
        return 250.0
    return float(np.interp(n, *NORMS)) * (1.22 if probe == "ring512" else 1.0)


# grid sizes and the largest singular values of arc256 on them (power iteration)
NORMS = ((78, 100, 128, 150, 200, 256, 400),
         (1.35e-5, 1.81e-5, 2.07e-5, 1.92e-5, 1.45e-5, 1.03e-5, 3.95e-6))


def _detectors(probe):
    D, cover, T = PROBES[probe]
    ang = np.deg2rad((180.0 - cover) / 2.0 + cover / (D - 1) * np.arange(D))
    return RADIUS * np.cos(ang), -RADIUS * np.sin(ang), ang


def _sir_tables(n):
    """(SPMR [NS, 91], start/end 1-based, column of every (detector, pixel)): responses of
    a flat 0.25 mm x 10 mm element (8 x 8 point sources) to a Gaussian pixel on a polar
    grid of 0.1 mm and 1 degree."""
    x = torch.as_tensor(_axis(n), device="cuda")
    xd, zd, ang = (torch.as_tensor(v, device="cuda") for v in _detectors("arc256"))
    dx = x.view(1, -1, 1) - xd.view(-1, 1, 1)
    dz = x.view(1, 1, -1) - zd.view(-1, 1, 1)
    rho = (dx * dx + dz * dz).sqrt()
    cosine = -(dx * torch.cos(ang).view(-1, 1, 1) - dz * torch.sin(ang).view(-1, 1, 1)) / rho
    theta = torch.rad2deg(torch.acos(cosine.clamp(-1, 1)))
    r0 = math.floor(float(rho.min()) * 1e4)
    nr, na = math.ceil(float(rho.max()) * 1e4) - r0 + 1, math.ceil(float(theta.max())) + 1
    idx = (torch.round(rho * 1e4).long() - r0) * na + torch.round(theta).long()
    r = (torch.arange(nr, device="cuda", dtype=torch.float64) + r0) * 1e-4
    a = torch.deg2rad(torch.arange(na, device="cuda", dtype=torch.float64))
    ex = ((torch.arange(8, device="cuda", dtype=torch.float64) + 0.5) / 8 - 0.5) * 0.25e-3
    ey = ((torch.arange(8, device="cuda", dtype=torch.float64) + 0.5) / 8 - 0.5) * 10e-3
    px, pz = r.view(-1, 1) * torch.sin(a), r.view(-1, 1) * torch.cos(a)
    sigma = round((x[1] - x[0]).item() / 2 * 1e6) / 1e6
    k = torch.arange(91, device="cuda", dtype=torch.float64) - 45
    h = torch.zeros(nr, na, 91, device="cuda", dtype=torch.float64)
    for u in ex:
        for v in ey[:4]:  # symmetric in elevation
            dist = ((px - u) ** 2 + pz ** 2 + v * v).sqrt()
            t = k * (C / FS) - (dist - r.view(-1, 1)).unsqueeze(-1)
            h += torch.exp(-t * t / (2 * sigma * sigma)) * (-t) / dist.unsqueeze(-1)
    h = h.view(-1, 91)
    h /= h.abs().max()
    on = h.abs() > 1e-4 * h.abs().amax(1, keepdim=True)
    first = on.int().argmax(1)
    last = 90 - on.flip(1).int().argmax(1)
    se = torch.stack([first, last], 1) + 1
    return (h.cpu().numpy(), se.int().cpu().numpy(),
            (idx + 1).int().reshape(idx.shape[0], -1).cpu().numpy())


@functools.lru_cache(maxsize=2)
def _model(probe, n, most, sir):
    """The model of a geometry, for batches up to ``most``."""
    from msot_gb300 import Discretization, MSOTmodel, Probe
    D, cover, T = PROBES[probe]
    p = Probe(n_det=D, radius=RADIUS, angular_coverage=cover, fs=FS, n_samples=T, delay=0.0,
              eir=_eir(), eir_length=EIR_TAPS)
    x = _axis(n)
    return MSOTmodel(p, Discretization([x[0], x[-1]], n), C, sir, True, 0, FMIN, FMAX,
                     _norm(probe, n, sir), sir_tables=_sir_tables(n) if sir else None,
                     max_batch=most)


@functools.lru_cache(maxsize=2)
def _frames_plan(probe, batch):
    from msot_gb300.analytic import bp_kernel_device
    from msot_gb300.preprocess import Preprocessor
    D, _, T = PROBES[probe]
    prep = Preprocessor(T + RAW_CROP, RAW_CROP, (WINDOW[0], WINDOW[1], T - WINDOW[2]), FS, FMIN,
                        FMAX, max_cols=D * batch)
    return prep, bp_kernel_device(np.arange(1, T + RAW_CROP + 1) / FS)


@functools.lru_cache(maxsize=2)
def _unet(n, batch):
    from msot_gb300.warmstart import UNet
    return UNet(levels=4, base_channels=32, side=n, max_batch=batch, seed=0)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)


def _images(g, batch, n):
    """Disks of 0.3 to 3 mm and two thin vessels on an empty background: [batch, n, n]."""
    u = lambda k: torch.rand(batch, k, 1, 1, generator=g, device="cuda")
    x = torch.as_tensor(_axis(n), device="cuda", dtype=torch.float32)
    X, Z = x.view(1, 1, -1, 1), x.view(1, 1, 1, -1)
    img = torch.zeros(batch, n, n, device="cuda")
    cx, cz, r, a = (2 * u(8) - 1) * 0.01, (2 * u(8) - 1) * 0.01, 3e-4 + 2.7e-3 * u(8), u(8)
    for i in range(8):
        s = slice(i, i + 1)
        img += (((X - cx[:, s]) ** 2 + (Z - cz[:, s]) ** 2 <= r[:, s] ** 2)
                * (0.2 + 0.8 * a[:, s])).squeeze(1)
    px, pz, th = (2 * u(2) - 1) * 0.008, (2 * u(2) - 1) * 0.008, math.pi * u(2)
    for i in range(2):
        s = slice(i, i + 1)
        across = (Z - pz[:, s]) * torch.cos(th[:, s]) - (X - px[:, s]) * torch.sin(th[:, s])
        img += (0.7 * torch.exp(-across ** 2 / (2 * 8.5e-5 ** 2))).squeeze(1)
    return img


def _sinograms(g, batch, probe, crop=0):
    """Recordings of 24 absorbers of 0.1 to 1.5 mm per frame through the EIR's band, with
    1 % noise: [batch, D, T + crop], scaled so that reconstructions are of order one."""
    D, _, T = PROBES[probe]
    T += crop
    u = lambda *s: torch.rand(batch, *s, generator=g, device="cuda")
    xd, zd, _ = (torch.as_tensor(v, device="cuda", dtype=torch.float32) for v in _detectors(probe))
    t = torch.arange(T, device="cuda", dtype=torch.float32) * (C / FS)
    y = torch.zeros(batch, D, T, device="cuda")
    q = u(24, 4)
    for i in range(24):
        cx, cz = (2 * q[:, i, 0] - 1) * 0.011, (2 * q[:, i, 1] - 1) * 0.011
        s = 1e-4 * 15.0 ** q[:, i, 2]
        dist = ((cx.view(-1, 1) - xd) ** 2 + (cz.view(-1, 1) - zd) ** 2).sqrt()
        z = (t - dist.unsqueeze(-1)) / s.view(-1, 1, 1)
        y -= (0.2 + q[:, i, 3]).view(-1, 1, 1) * z * torch.exp(-0.5 * z * z)
    eir = torch.as_tensor(_eir(), device="cuda", dtype=torch.float32)
    m = T + EIR_TAPS
    for w in range(batch):  # frame by frame: the spectra of a whole batch are large
        y[w] = torch.fft.irfft(torch.fft.rfft(y[w], m) * torch.fft.rfft(eir, m),
                               m)[:, EIR_TAPS // 2:EIR_TAPS // 2 + T]
    y /= y.flatten(1).pow(2).mean(1).sqrt().view(-1, 1, 1)
    y += 0.01 * torch.randn(y.shape, generator=g, device="cuda")
    return (y * DATA_RMS).contiguous()


DATA_RMS = 0.002


def _unet_inputs(g, batch, n):
    x = _images(g, batch, n).unsqueeze(1)
    x = x + 0.2 * torch.randn(x.shape, generator=g, device="cuda")
    x = x / x.flatten(1).pow(2).mean(1).sqrt().view(-1, 1, 1, 1)
    return x, 0.1 * torch.randn(x.shape, generator=g, device="cuda")


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    s = dict(case)
    if kind == "unet":
        s["net"] = _unet(case["n"], case["batch"])
        s["x"], s["t"] = _unet_inputs(g, case["batch"], case["n"])
        return s
    if kind == "frames":
        s["prep"], s["K"] = _frames_plan(case["probe"], case["batch"])
        s["axis"] = _axis(case["n"])
        s["raw"] = _sinograms(g, case["batch"], case["probe"], RAW_CROP)
        return s
    s["model"] = _model(case["probe"], case["n"], 16 if case["batch"] <= 16 else 64,
                        case.get("sir", False))
    if kind == "operator":
        if case["dir"] != "transpose":
            s["x"] = _images(g, case["batch"], case["n"])
        if case["dir"] != "forward":
            s["y"] = _sinograms(g, case["batch"], case["probe"])
    else:
        s["y"] = _sinograms(g, case["batch"], case["probe"])
    return s


def run(s):
    from msot_gb300 import (backproject_waveeq, dmas_cf, rec_nn_with_L1_eye_reg,
                            rec_nn_with_L2_reg, rec_nn_with_TV_reg)
    kind = s["kind"]
    if kind == "operator":
        out = {}
        if s["dir"] != "transpose":
            out["sinogram"] = s["model"].forward(s["x"])
        if s["dir"] != "forward":
            out["image"] = s["model"].transpose(s["y"])
        return out
    if kind == "unet":
        if s["backward"]:
            loss, grad = s["net"].gradients(s["x"], s["t"])
            return {"loss": np.float32(loss), "gradient": grad}
        return {"prediction": s["net"].forward(s["x"])}
    if kind == "frames":
        filtered = s["prep"](s["raw"])
        D, cover, _ = PROBES[s["probe"]]
        bp = backproject_waveeq(filtered, s["axis"], s["axis"], C, FS, RAW_CROP, cover, RADIUS,
                                np.array([[1.0]]), s["K"])
        das = dmas_cf(filtered, s["axis"], s["axis"], C, FS, RAW_CROP, cover, RADIUS)
        return {"filtered": filtered, "waveeq": bp, "dmas": list(das)}
    # the l-curve values are sums of FP32 residuals and images: float32 is what they carry
    if kind == "l2":
        rec, e1, e2 = rec_nn_with_L2_reg(s["model"], s["y"], s["iters"], LAMBDA_L2)[:3]
    elif kind == "l1":
        rec, e1, e2 = rec_nn_with_L1_eye_reg(s["model"], s["y"], s["iters"], LAMBDA_L1)[:3]
    else:  # the wavelengths of one stack are one coupled solve, as in the reference
        rec, e1, e2 = rec_nn_with_TV_reg(s["model"], s["y"], s["iters"], LAMBDA_TV,
                                         coupled=True)[:3]
    return {"image": rec, "residual": np.float32(e1), "penalty": np.float32(e2)}


# --- work --------------------------------------------------------------------------------
def work(case):
    n, W = case["n"], case["batch"]
    P = n * n
    if case["kind"] == "unet":
        # 3 x 3 convolutions of a 4-level net with 32 base channels (and its gradients)
        ch, mac = [32, 64, 128, 256], 0
        for l, c in enumerate(ch):
            p = P >> (2 * l)
            mac += 9 * p * c * ((ch[l - 1] if l else 1) + c)
            if l < 3:
                mac += 9 * p * c * (ch[l + 1] + c + c)
        f = 2.0 * W * (mac + 32 * P)
        return {"bytes": 4.0 * (2 * W * P + 4.3e6), "flops": f * (3 if case["backward"] else 1)}
    D, _, T = PROBES[case["probe"]]
    img, sino, pairs = 4.0 * W * P, 4.0 * W * D * T, float(P) * D
    # one application: two multiply-adds per (pixel, detector, frame), the IR convolution
    # as FFTs of the columns (5 N log2 N there and back), the separable prefilter
    conv = W * D * 2 * 5.0 * T * math.log2(2048)
    apply = 4.0 * pairs * W + conv + 4.0 * 29 * P * W
    if case["kind"] == "frames":
        # the filters as FFTs, the time-domain kernel as the dense product that K is
        return {"bytes": 2 * sino + 4.0 * T * T + 5 * img,
                "flops": W * D * (2 * 5.0 * T * 11 + 2.0 * T * T) + 10.0 * pairs * W}
    if case["kind"] == "operator":
        k = 2 if case["dir"] == "both" else 1
        if case["sir"]:
            apply = W * pairs * 2.0 * 30 + conv + 4.0 * 29 * P * W
        return {"bytes": k * (img + sino + 4.0 * pairs), "flops": k * apply}
    # applications of A and A^T of one outer iteration: LSQR (2 steps) 3 + 2, CGS (2 steps)
    # 4 + 4, SpaRSA (2 steps) 3 + 2
    per = {"l2": 5, "l1": 8, "tv": 5}[case["kind"]]
    return {"bytes": sino + img + 4.0 * pairs, "flops": per * case["iters"] * apply}


# --- the same in 64 bits -------------------------------------------------------------------
def _butter_power(w, order, cutoff, high):
    """|H|^2 of the bilinear Butterworth low- or high-pass at the angles w."""
    t = torch.tan(w / 2).abs() / math.tan(cutoff / 2)
    return 1 / (1 + (1 / t if high else t) ** (2 * order))


def _zero_phase(x):
    """Demean and the zero-phase band-pass on the last axis (circular, FFT domain)."""
    n = x.shape[-1]
    w = 2 * math.pi * torch.arange(n, device=x.device, dtype=torch.float64) / n
    h2 = _butter_power(w, 8, 2 * math.pi * FMAX / FS, False)
    h2 = h2 * _butter_power(w, 2, 2 * math.pi * FMIN / FS, True)
    x = x - x.mean(-1, keepdim=True)
    return torch.fft.ifft(torch.fft.fft(x) * h2).real


class _Exact:
    """A and A^T of a case's model in FP64: the interpolation as a sparse matrix."""

    def __init__(self, case):
        self.n, self.probe = case["n"], case["probe"]
        self.D, _, self.T = PROBES[self.probe]
        n, D, T = self.n, self.D, self.T
        f64 = dict(device="cuda", dtype=torch.float64)
        x = torch.as_tensor(_axis(n), **f64)
        xd, zd, _ = (torch.as_tensor(v, **f64) for v in _detectors(self.probe))
        tau = ((x.view(1, -1, 1) - xd.view(-1, 1, 1)) ** 2
               + (x.view(1, 1, -1) - zd.view(-1, 1, 1)) ** 2).sqrt().view(D, -1) / C * FS
        h = (x[1] - x[0]).item()
        self.r = h / (C / FS)
        sigma = round(h / 2 * 1e6) / 1e6
        eir = torch.as_tensor(_eir(), **f64)
        if case.get("sir"):
            ir = eir
        else:
            L = EIR_TAPS
            t = torch.arange(-(L // 2), L // 2 + 1, **f64) / FS
            resp = torch.exp(-(t * C) ** 2 / (2 * sigma ** 2)) * (-t)
            ir = torch.fft.irfft(torch.fft.rfft(eir, 2 * L) * torch.fft.rfft(resp, 2 * L),
                                 2 * L)[L // 2:L // 2 + L]
        ir = _zero_phase(ir) / _norm(self.probe, n, case.get("sir", False))
        self.m = T + EIR_TAPS
        self.irf = torch.fft.rfft(ir, self.m)
        g = torch.exp(-(h * (np.floor(-n / 2) + torch.arange(n, **f64))) ** 2
                      / (2 * sigma ** 2))
        gh = torch.fft.fft(torch.fft.fftshift(g))
        kern = torch.fft.ifft(torch.conj(gh / torch.fft.fft(
            torch.fft.ifft(gh.abs() ** 2).real))).real
        self.pre = torch.fft.fft(kern)
        taps = int(math.floor(2 * self.r)) + 2
        first = torch.ceil(tau - self.r)
        if case.get("sir"):
            self.sir, self.tau, self.first, self.taps = _sir_tables(n), tau, first, taps
            return
        pix = torch.arange(n * n, device="cuda").view(1, -1)
        det = torch.arange(D, device="cuda").view(-1, 1)
        rows, cols, vals = [], [], []
        for k in range(taps):
            w = 1 - (first + k - tau).abs() / self.r
            keep = w > 0
            rows.append((det * T + first.long() + k)[keep].int())
            cols.append(pix.expand(D, -1)[keep].int())
            vals.append(w[keep])
        rows, cols, vals = torch.cat(rows), torch.cat(cols), torch.cat(vals)
        self.S = self._csr(rows, cols, vals, D * T, n * n)
        self.St = self._csr(cols, rows, vals, n * n, D * T)

    @staticmethod
    def _csr(rows, cols, vals, nr, nc):
        order = torch.argsort(rows)
        ptr = torch.zeros(nr + 1, dtype=torch.int64, device="cuda")
        ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=nr), 0)
        return torch.sparse_csr_tensor(ptr.int(), cols[order], vals[order], (nr, nc))

    def _prefilter(self, img, conj):
        p = self.pre.conj() if conj else self.pre
        f = torch.fft.fft2(img) * p.view(-1, 1) * p.view(1, -1)
        return torch.fft.ifft2(f).real

    def _sir_columns(self, d):
        """(first sample, response [P, 90 + taps]) of every pixel for detector d: its column
        (zero outside start .. end) convolved with the tri taps."""
        h, se, idx = self.sir
        h, se = (torch.as_tensor(v, device="cuda") for v in (h, se))
        i = torch.as_tensor(idx[d], device="cuda").long() - 1
        k = torch.arange(1, 92, device="cuda")
        h = h[i] * ((k >= se[i, :1]) & (k <= se[i, 1:]))
        e = torch.zeros(h.shape[0], 90 + self.taps, device="cuda", dtype=torch.float64)
        for j in range(self.taps):
            w = (1 - (self.first[d] + j - self.tau[d]).abs() / self.r).clamp_min(0)
            e[:, j:j + 91] += w.view(-1, 1) * h
        return self.first[d].long() - 45, e

    def _sir_apply(self, v, transpose):
        W, pad = v.shape[0], 256
        out = torch.zeros((W, self.n ** 2) if transpose else (W, self.D, self.T),
                          device="cuda", dtype=torch.float64)
        for d in range(self.D):
            first, e = self._sir_columns(d)
            at = first.view(-1, 1) + torch.arange(e.shape[1], device="cuda") + pad
            for w in range(W):
                if transpose:
                    row = torch.nn.functional.pad(v[w, d], (pad, pad))
                    out[w] += (e * row[at]).sum(1)
                else:
                    col = torch.zeros(self.T + 2 * pad, device="cuda", dtype=torch.float64)
                    col.index_add_(0, at.flatten(), (e * v[w].view(-1, 1)).flatten())
                    out[w, d] = col[pad:pad + self.T]
        return out

    def forward(self, img):
        W, L = img.shape[0], EIR_TAPS
        c = self._prefilter(img, False).reshape(W, -1)
        if hasattr(self, "sir"):
            y = self._sir_apply(c, False)
        else:
            y = (self.S @ c.t().contiguous()).t().reshape(W, self.D, self.T)
        out = torch.empty_like(y, memory_format=torch.contiguous_format)
        for w in range(W):
            f = torch.fft.irfft(torch.fft.rfft(y[w].contiguous(), self.m) * self.irf, self.m)
            out[w] = f[:, L // 2:L // 2 + self.T]
        return out

    def transpose(self, y):
        W, L = y.shape[0], EIR_TAPS
        s = torch.empty_like(y)
        for w in range(W):
            f = torch.fft.rfft(torch.nn.functional.pad(y[w], (L // 2, self.m - self.T - L // 2)))
            s[w] = torch.fft.irfft(f * self.irf.conj(), self.m)[:, :self.T]
        if hasattr(self, "sir"):
            c = self._sir_apply(s, True)
        else:
            c = (self.St @ s.view(W, -1).t().contiguous()).t()
        return self._prefilter(c.reshape(W, self.n, self.n), True)


def _dot(a, b):
    return (a * b).flatten(1).sum(1).view(-1, 1, 1)


def _exact_l2(A, b, iters, beta=1e-3):
    """The splitting of nnls_L2_less with two LSQR steps per iteration, per instance, on
    the stacked system [A; sqrt(lambda) I; sqrt(beta) I]."""
    lam, W, n = LAMBDA_L2, b.shape[0], A.n
    sl, sb = math.sqrt(lam), math.sqrt(beta)
    w = torch.zeros(W, n, n, device="cuda", dtype=torch.float64)
    v = torch.zeros_like(w)
    op = lambda z: (A.forward(z), sl * z, sb * z)
    op_t = lambda u: A.transpose(u[0]) + sl * u[1] + sb * u[2]
    norm = lambda u: sum(_dot(t, t) for t in u).sqrt()
    for _ in range(iters):
        rhs = (b, torch.zeros_like(w), sb * (w + v))
        x = w.clone()
        u = tuple(r - a for r, a in zip(rhs, op(x)))
        bet = norm(u)
        u = tuple(t / bet for t in u)
        c, s, phibar, normr = torch.ones_like(bet), torch.zeros_like(bet), bet, bet
        z = op_t(u)
        alpha = _dot(z, z).sqrt()
        z, d = z / alpha, torch.zeros_like(w)
        for step in range(2):
            u = tuple(a - alpha * t for a, t in zip(op(z), u))
            bet = norm(u)
            u = tuple(t / bet for t in u)
            thet, rhot = -s * alpha, c * alpha
            rho = (rhot * rhot + bet * bet).sqrt()
            c, s = rhot / rho, -bet / rho
            phi, phibar = c * phibar, s * phibar
            d = (z - thet * d) / rho
            x = x + phi * d  # |s| < 1: the residual estimate falls, the last iterate stays
            if step == 0:
                z = op_t(u) - bet * z
                alpha = _dot(z, z).sqrt()
                z = z / alpha
        w = (x - v).clamp_min(0)
        v = v + w - x
    return w


def _exact_l1(A, b, iters):
    """nnls_L1_eye_matrix_less: split Bregman with two CGS steps from zero."""
    op = lambda x: A.transpose(A.forward(x)) + x
    atb = A.transpose(b)
    u, bp = atb.clone(), torch.zeros_like(atb)
    for _ in range(iters):
        d = (u - bp).clamp_min(0)
        rhs = d + bp + atb - LAMBDA_L1
        x, r = torch.zeros_like(rhs), rhs.clone()
        best, least = x.clone(), _dot(rhs, rhs).sqrt()
        rt, rho, q, p = rhs, None, None, None
        for step in range(2):
            last, rho = rho, _dot(rt, r)
            if step == 0:
                t = r.clone()
                p = t.clone()
            else:
                beta = rho / last
                t = r + beta * q
                p = t + beta * (q + beta * p)
            vh = op(p)
            alpha = rho / _dot(rt, vh)
            q = t - alpha * vh
            x = x + alpha * (t + q)
            r = r - alpha * op(t + q)
            size = _dot(r, r).sqrt()
            best = torch.where(size < least, x, best)
            least = torch.minimum(size, least)
        bp, u = bp + d - best, best
    return u


def _nearest(probe, axis, T):
    D, _, _ = PROBES[probe]
    x = torch.as_tensor(axis, device="cuda")
    xd, zd, ang = (torch.as_tensor(v, device="cuda") for v in _detectors(probe))
    dist = ((x.view(1, -1, 1) - xd.view(-1, 1, 1)) ** 2
            + (x.view(1, 1, -1) - zd.view(-1, 1, 1)) ** 2).sqrt()
    v = (dist / C - (1 + RAW_CROP) / FS) * FS + 1
    return torch.floor(v + 0.5).long().view(D, -1) - 1, ang


def _exact_frames(s):
    y = s["raw"].double()[..., RAW_CROP:]
    W, D, T = y.shape
    k = torch.arange(T, device="cuda", dtype=torch.float64)
    lo, hi = math.tan(math.pi * WINDOW[1] / T / 2), math.tan(math.pi * (T - WINDOW[2]) / T / 2)
    om = torch.tan(math.pi * k / T / 2)
    h = 1 / (1 + ((om * om - lo * hi) / ((hi - lo) * om)) ** (2 * WINDOW[0])).sqrt()
    m = y.mean(-1, keepdim=True)
    y = _zero_phase(m + (y - m) * h)
    out = {"filtered": y}
    idx, ang = _nearest(s["probe"], s["axis"], T)
    dt = 1 / FS
    acc = torch.cumsum(0.5 * dt * (y[..., 1:] + y[..., :-1]) / C, -1)
    acc = torch.nn.functional.pad(acc, (1, 0)) / ((k + 1 + RAW_CROP) * dt)
    nt = T + RAW_CROP
    t = torch.arange(1, nt + 1, device="cuda", dtype=torch.float64) / FS
    dl = math.pi / ((nt - 1) / FS)
    lam = dl * torch.arange(1, nt + 1, device="cuda", dtype=torch.float64)
    wl = torch.full_like(lam, dl)
    wl[0] = wl[-1] = dl / 2
    arg = t.view(-1, 1) * lam
    M = (torch.special.bessel_j0(arg) * (wl * lam)) @ torch.special.bessel_y0(arg).t()
    K = (M - M.t())[RAW_CROP:, RAW_CROP:]
    swl = (acc.reshape(-1, T) @ K.t()).view(W, D, T) * dt
    n = len(s["axis"])
    fx = torch.zeros(W, n * n, device="cuda", dtype=torch.float64)
    fz = torch.zeros_like(fx)
    sig = y.float().double()  # dmas_cf takes the FP32 sinogram
    sig = sig / sig.abs().max()
    sums = [torch.zeros_like(fx) for _ in range(4)]
    for d in range(D):
        v = swl[:, d, idx[d]] * dt * C
        fx += v * torch.cos(-ang[d])
        fz += v * torch.sin(-ang[d])
        v = sig[:, d, idx[d]]
        root = v.sign() * v.abs().sqrt()
        for acc_, add in zip(sums, (root * root, root, v, v * v)):
            acc_ += add
    ax = torch.as_tensor(s["axis"], device="cuda")

    def grad(f, dim):
        f = f.transpose(dim, -1)
        g = torch.empty_like(f)
        g[..., 1:-1] = (f[..., 2:] - f[..., :-2]) / (ax[2:] - ax[:-2])
        g[..., 0] = (f[..., 1] - f[..., 0]) / (ax[1] - ax[0])
        g[..., -1] = (f[..., -1] - f[..., -2]) / (ax[-1] - ax[-2])
        return g.transpose(dim, -1)

    out["waveeq"] = (grad(fx.view(W, n, n), 1) + grad(fz.view(W, n, n), 2)).flip(1)
    sos, sqs, num, den = (t.view(W, n, n) for t in sums)
    dmas, cf = 0.5 * (sqs ** 2 - sos), num ** 2 / (1e-6 + D * den)
    out["dmas"] = [dmas * cf, dmas, cf, num]
    return out


def _exact_unet(s):
    """The network in FP64; its 3 x 3 weights are BF16 by definition."""
    F = torch.nn.functional
    p = torch.as_tensor(s["net"].get_params(), device="cuda").double()
    at, leaves = [0], []

    def conv(x, co, k=3):
        ci = x.shape[1]
        n = co * ci * k * k
        w, b = p[at[0]:at[0] + n].view(co, ci, k, k), p[at[0] + n:at[0] + n + co]
        at[0] += n + co
        if k == 3:
            w = w.float().bfloat16().double()
        w, b = w.detach().clone().requires_grad_(), b.detach().clone().requires_grad_()
        leaves.append((w, b))
        return lambda v, w=w, b=b: F.conv2d(v, w, b, padding=k // 2)

    def layers():
        ch = [32, 64, 128, 256]
        probe = lambda c: torch.empty(1, c, 1, 1)
        enc = [(conv(probe(ch[l - 1] if l else 1), ch[l]), conv(probe(ch[l]), ch[l]))
               for l in range(4)]
        dec = {l: (conv(probe(ch[l + 1] + ch[l]), ch[l]), conv(probe(ch[l]), ch[l]))
               for l in (2, 1, 0)}
        return enc, dec, conv(probe(32), 1, 1)

    def net(x):
        skips = []
        for l, (a, b) in enumerate(enc):
            x = F.relu(b(F.relu(a(x))))
            skips.append(x)
            if l < 3:
                x = F.avg_pool2d(x, 2)
        for l in (2, 1, 0):
            u = F.interpolate(x, scale_factor=2, mode="nearest")
            a, b = dec[l]
            x = F.relu(b(F.relu(a(torch.cat([u, skips[l]], 1)))))
        return last(x)

    enc, dec, last = layers()
    x, t = s["x"].double(), s["t"].double()
    if not s["backward"]:
        with torch.no_grad():
            return {"prediction": torch.cat([net(v) for v in x.split(1)])}
    loss = 0.0
    for v, u in zip(x.split(1), t.split(1)):
        part = ((net(v) - u) ** 2).sum() / t.numel()
        part.backward()
        loss += part.item()
    grad = torch.cat([v.grad.flatten() for pair in leaves for v in pair])
    return {"loss": torch.tensor(loss, dtype=torch.float64), "gradient": grad}


def exact(case, seed):
    if case["kind"] == "tv":
        return None  # thousands of small split-Bregman steps: minutes in 64 bits
    s = prepare(case, seed)
    if case["kind"] == "unet":
        return _exact_unet(s)
    if case["kind"] == "frames":
        return _exact_frames(s)
    A = _Exact(case)
    if case["kind"] == "operator":
        out = {}
        if "x" in s:
            out["sinogram"] = A.forward(s["x"].double())
        if "y" in s:
            out["image"] = A.transpose(s["y"].double())
        return out
    b = s["y"].double()
    if case["kind"] == "l2":
        rec = _exact_l2(A, b, case["iters"])
        penalty = rec.pow(2).flatten(1).sum(1)
    else:
        rec = _exact_l1(A, b, case["iters"])
        penalty = rec.abs().flatten(1).sum(1)
    res = (A.forward(rec) - b).pow(2).flatten(1).sum(1)
    return {"image": rec, "residual": res, "penalty": penalty}
