"""Device memory of a plan: nothing that its batches cannot use, and the kernels with
tables of their own are left out where those do not fit."""
import gc

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


@pytest.mark.parametrize("sir", [False, True])
def test_tables_that_do_not_fit_are_left_out(cuda, sir):
    import torch
    n, D, W = (160, 256, 5) if sir else (320, 192, 5)
    rng = np.random.default_rng(3)
    tab = None
    if sir:
        idx = rng.integers(1, 5, (D, n * n)).astype(np.int32)
        tab = (rng.standard_normal((4, 31)), np.tile(np.int32([[1, 31]]), (4, 1)), idx)

    def model():
        return make_pair(n=n, n_det=D, n_samples=T, radius=0.02, fov_half=0.006, norm=2e-5,
                         max_batch=W, sir_tables=tab)[0]

    y = torch.tensor(rng.standard_normal((W, D, T)), dtype=torch.float32).cuda()
    m = model()
    want, full = m.transpose(y), _bytes(m)
    del m
    gc.collect()  # models refer to themselves: this one and other tests' now, not later
    tables = (24 if sir else 4) * D * n * n  # SIR: 32 bytes a pair for the 8 of k_sir_fwd
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - (full - tables // 2), dtype=torch.uint8, device="cuda")
    m = model()
    del hog
    torch.cuda.empty_cache()
    assert _bytes(m) < full - 0.9 * tables
    got = m.transpose(y)
    assert float((got - want).norm() / want.norm()) < 1e-5


def test_analytic_workspaces_are_given_back(cuda):
    import torch
    from msot_gb300 import dmas_cf
    from msot_gb300.analytic import release_workspaces
    sig = torch.randn(4, 64, 1200, device="cuda")
    x = np.linspace(-0.005, 0.005, 256)

    def call():  # the index table alone is 16 MiB
        out = dmas_cf(sig, x, x, 1500.0, 4e7, 0.0, 135.0, 0.015)
        torch.cuda.synchronize()
        return out

    gc.collect()
    kept = call()  # results and modules stay
    release_workspaces()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    again = call()
    assert torch.cuda.mem_get_info()[0] <= free - (16 << 20)
    release_workspaces()
    del kept, again
    torch.cuda.empty_cache()
    assert torch.cuda.mem_get_info()[0] >= free
