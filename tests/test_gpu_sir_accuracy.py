"""The SIR operators' error against 64 bits on the data they are made for: recordings in
the EIR's band, 256 detectors, responses as smooth as the pixel.  A pixel's taps
cancel within one detector there (white noise shows nothing), and the fewer the pixels,
the more they do."""
import numpy as np
import pytest

from oracle import model as M
from pairs import make_pair, rel

pytestmark = pytest.mark.gpu

D, T, S, NS = 256, 2030, 91, 24


def _pair(n, W):
    """Derivatives of Gaussians as wide as the pixel and up to half as wide again, by the
    pixel's direction from the detector."""
    r = 0.0254 / (n - 1) / 0.0375e-3
    t = np.arange(S) - S // 2
    sig = r / 2 * (1 + 0.5 * np.arange(NS) / NS)
    sir = -t / sig[:, None] * np.exp(-t ** 2 / (2 * sig[:, None] ** 2))
    on = np.abs(sir) > 1e-4 * np.abs(sir).max(1, keepdims=True)
    se = np.stack([on.argmax(1) + 1, S - on[:, ::-1].argmax(1)], 1).astype(np.int32)
    x = np.linspace(-0.0127, 0.0127, n)
    ang = np.linspace(0, 1, D)[:, None, None]
    where = (x[None, :, None] * (1 - ang) + x[None, None, :] * ang) / 0.0127
    idx = (1 + (NS - 1) * np.abs(where).clip(0, 1)).astype(np.int32).reshape(D, -1)
    return make_pair(n=n, n_det=D, n_samples=T, norm=250.0, max_batch=W,
                     sir_tables=(sir, se, idx))


def _recordings(rng, W):
    eir = M.gauss_pulse_eir()
    m = T + eir.size
    y = np.fft.irfft(np.fft.rfft(rng.standard_normal((W, D, T)), m) * np.fft.rfft(eir, m), m)
    return y[..., eir.size // 2:eir.size // 2 + T]


# one image takes the kernel that filters by the tri taps first, more may take composite
# rows: no less exact, but for the scatter of two orders of the same roundings
@pytest.mark.parametrize("n,W", [(50, 3), (60, 8), (60, 64), (78, 8), (80, 3), (100, 8), (128, 8)])
def test_transpose_is_as_exact_in_a_batch(cuda, n, W):
    import torch
    pm, om = _pair(n, W)
    y = np.repeat(_recordings(np.random.default_rng(n), 1), W, 0).astype(np.float32)
    ref = om.transpose(y[:1].astype(np.float64))[0]
    alone = rel(pm.transpose(torch.tensor(y[:1])).cpu().numpy()[0], ref)
    batch = rel(pm.transpose(torch.tensor(y)).cpu().numpy()[W - 1], ref)
    print(f"n {n} W {W}: alone {alone:.2e} batch {batch:.2e}")
    assert batch <= 1.1 * alone


# the bars are the errors of k_sir_fwd (a column in shared memory, atomics) on these images
@pytest.mark.parametrize("n,W,bar", [(78, 4, 7.9e-6), (100, 2, 3.8e-6), (128, 1, 2.2e-6),
                                     (128, 8, 2.6e-6)])
def test_forward_is_as_exact_as_with_atomics(cuda, n, W, bar):
    import torch
    pm, om = _pair(n, W)
    x = np.linspace(-1, 1, n)
    img = np.zeros((W, n, n), dtype=np.float32)
    for cx, cz, r in ((-0.3, 0.2, 0.4), (0.5, 0.5, 0.15), (0.1, -0.6, 0.25), (-0.7, -0.7, 0.05)):
        img += ((x[:, None] - cx) ** 2 + (x[None] - cz) ** 2 <= r * r).astype(np.float32)
    ref = om.forward(img[:1].astype(np.float64))[0]
    err = rel(pm.forward(torch.tensor(img)).cpu().numpy()[W - 1], ref)
    print(f"n {n} W {W}: forward {err:.2e}")
    assert err <= bar
