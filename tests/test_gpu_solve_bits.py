"""The bits of A and of the iterative solves.

A solve amplifies a last bit of its operators to 1e-3 of an image's rms at single
pixels: moving the recordings of 64 frames by at most one ulp moves some pixel by
more than 8e-4 of the rms in one L2 solve of eight, one coupled TV solve of six.  So
a kernel that adds in another order gives other images, however exact it is, and the
digests here pin the order: convolution tiles at multiples of the block, the filter
over the bucket moments as one chain, detector groups of the adjoint, slabs of the
TV prox.  ``python tests/test_gpu_solve_bits.py`` prints them.
"""
import hashlib
import json
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "solve_bits.json")


def _model(n, D, T, W, radius=0.02, fov=0.006):
    from oracle import model as M
    from msot_gb300 import Discretization, MSOTmodel, Probe
    eir = M.gauss_pulse_eir()
    return MSOTmodel(Probe(n_det=D, radius=radius, n_samples=T, eir=eir, eir_length=eir.size),
                     Discretization([-fov, fov], n), 1500.0, False, True, 0, 1e5, 12e6, 2e-5,
                     max_batch=W)


def _images(n, W):
    """Two disks per image: values that need no transcendental function."""
    x = np.linspace(-1.0, 1.0, n)
    img = np.zeros((W, n, n), dtype=np.float32)
    for w in range(W):
        for k in range(2):
            cx, cz, r = ((37 * w + 11 * k) % 17 - 8) / 12, ((23 * w + 5 * k) % 13 - 6) / 9, 0.2
            img[w] += ((x[:, None] - cx) ** 2 + (x[None] - cz) ** 2 <= r * r) * (0.5 + k)
    return img


def _data(model, n, W):
    """Recordings of the disks, with a ripple that is no image's."""
    import torch
    y = model.forward(torch.tensor(_images(n, W)).cuda())
    t = torch.arange(y.numel(), device="cuda").reshape(y.shape)
    return y + y.abs().max() * 0.01 * ((t * 7919 % 1009) - 504).float() / 504


# (what, n, detectors, samples, images)
CASES = [
    ("forward", 70, 37, 1300, 3),      # odd D: column pairs across images
    ("forward", 70, 16, 4096, 9),      # most tiles without input; lanes over instances
    ("forward", 31, 8, 1300, 33),      # r = 8.9; tiles of 32 images and of one
    ("transpose", 400, 8, 1300, 2),    # prefilter of long columns
    ("l2", 64, 64, 1300, 9),
    ("l2", 90, 40, 1300, 2),           # D no multiple of 8 pairs: the unfused update
    ("l1", 64, 64, 1300, 6),
]
TV_CASES = [
    ("tv", 48, 32, 1300, 5),           # coupled sums of five images
    ("tv", 77, 32, 1300, 2),           # a side that is no multiple of four
    ("prox", 136, 0, 0, 2),            # slabs of one CTA per SM
    ("prox", 200, 0, 0, 1),
    ("prox", 200, 0, 0, 12),           # two slabs per CTA
    ("prox", 141, 0, 0, 3),
    ("prox", 280, 0, 0, 1),            # beyond the slabs: vectors in registers or in L2
]


def digest(what, n, D, T, W):
    import torch
    from msot_gb300 import (SB_ITV2, rec_nn_with_L1_eye_reg, rec_nn_with_L2_reg,
                            rec_nn_with_TV_reg)
    if what == "prox":
        out = SB_ITV2(torch.tensor(_images(n, W) + 0.1 * _images(n, W)[:, ::-1].copy()), 0.05)
    else:
        m = _model(n, D, T, W, fov=0.005 if n == 31 else 0.006)
        if what == "forward":
            out = m.forward(torch.tensor(_images(n, W)).cuda())
        else:
            y = _data(m, n, W)
            if what == "transpose":
                out = m.transpose(y)
            elif what == "l2":
                out = rec_nn_with_L2_reg(m, y, 12, 1e-2)[0]
            elif what == "l1":
                out = rec_nn_with_L1_eye_reg(m, y, 6, 1e-3)[0]
            else:
                out = rec_nn_with_TV_reg(m, y, 4, 5e-3, coupled=True)[0]
    out = np.ascontiguousarray(out.cpu().numpy())
    assert np.isfinite(out).all() and np.abs(out).max() > 0
    return hashlib.sha256((out + 0.0).tobytes()).hexdigest()  # + 0.0: one zero


def _check(case):
    with open(GOLDEN) as f:
        assert digest(*case) == json.load(f)["-".join(map(str, case))]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_operator_and_solves_keep_their_bits(cuda, case):
    _check(case)


@pytest.mark.parametrize("case", TV_CASES, ids=lambda c: "-".join(map(str, c)))
def test_tv_keeps_its_bits(cuda, case):
    _check(case)


if __name__ == "__main__":
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    sys.path[:0] = [root, os.path.join(root, "mb-rec-msot_gb300")]
    print(json.dumps({"-".join(map(str, c)): digest(*c) for c in CASES + TV_CASES}, indent=1))
