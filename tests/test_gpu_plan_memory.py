"""Device memory of a plan: nothing that its batches cannot use, and the kernels with
tables of their own are left out where those do not fit."""
import numpy as np
import pytest

from pairs import make_pair

pytestmark = pytest.mark.gpu

N, D, T = 96, 64, 1300


def _model(W, **kw):
    return make_pair(n=N, n_det=D, n_samples=T, radius=0.02, fov_half=0.006, max_batch=W, **kw)[0]


def _bytes(m):
    from msot_gb300 import _lib
    return _lib.load().msot_plan_device_bytes(m.plan)


def test_a_plan_holds_what_its_batches_use(cuda):
    b = {W: _bytes(_model(W)) for W in (1, 4, 5)}
    P = N * N

    def per_batch(W):  # two images, one padded to a tile, a recording, partial images, scales
        tile = 1 << (W - 1).bit_length()
        return 4 * (W * P + tile * P + W * D * T + min(32, 640 // W) * W * P + 2 * W)

    assert b[4] - b[1] == per_batch(4) - per_batch(1)
    # the batched adjoint serves five images and more: 4 bytes per (padded pixel, detector)
    assert b[5] - b[4] >= per_batch(5) - per_batch(4) + 4 * 128 * 128 * D
