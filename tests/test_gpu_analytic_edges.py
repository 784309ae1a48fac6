"""Edges of the analytic path's kernels: odd frame counts and pixel tiles of the
gathers, the three column widths of the tensor-core GEMM, columns too long for
shared memory.  Bars: sums in pairs of floats with one FP32 rounding at the end
(1e-6 allows a few), the GEMM's 1e-5 of test_gpu_preprocess.py, 1e-4 of
test_gpu_analytic.py for backproject_waveeq."""
import numpy as np
import pytest

from oracle import backprojection as B
from oracle import preprocess as Q
from pairs import rel

pytestmark = pytest.mark.gpu

GEOM = dict(c=1500.0, fs=4e7, n_crop=3.0, coverage=135.0, R=0.015)


@pytest.mark.parametrize("W,nx,nz", [(1, 1, 33), (3, 9, 31), (5, 17, 40)])
def test_gathers_at_tile_edges(cuda, W, nx, nz):
    import torch
    from msot_gb300 import backproject_waveeq, dmas_cf
    rng = np.random.default_rng(W)
    D, T = 37, 901
    sig = rng.standard_normal((W, D, T)).astype(np.float32)
    x = np.linspace(-0.003, 0.003, nx) if nx > 1 else np.array([0.0011])
    z = np.linspace(-0.0028, 0.0028, nz)
    g = GEOM
    args = (g["c"], g["fs"], g["n_crop"], g["coverage"], g["R"])
    ref = B.dmas_cf(sig.astype(np.float64), x, z, *args)
    for a, b in zip(dmas_cf(torch.tensor(sig), x, z, *args), ref):
        assert rel(a.cpu().numpy(), b) < 1e-6
    if nx > 1:  # MATLAB's gradient needs two columns
        Nt = T + 3
        K = B.bp_kernel(np.arange(1, Nt + 1) / g["fs"])
        got = backproject_waveeq(torch.tensor(sig), x, z, *args, np.array([[2.0]]), K)
        want = B.backproject_waveeq(sig.astype(np.float64), x, z, *args, np.array([[2.0]]), K)
        assert rel(got.cpu().numpy(), want) < 1e-4


# M = 300 (three row tiles): 64-, 128- and 256-column tiles, one past a tile edge
@pytest.mark.parametrize("cols", [1, 63, 65, 6401, 12673, 13057])
def test_gemm_column_tiles(cuda, cols):
    import torch
    from msot_gb300.preprocess import Preprocessor
    rng = np.random.default_rng(cols)
    x = rng.standard_normal((cols, 303)).astype(np.float32)
    got = Preprocessor(303, 3, None, 4e7, 1e5, 12e6, max_cols=cols)(torch.tensor(x))
    got = got.cpu().numpy()
    at = np.unique(np.concatenate([np.arange(0, cols, max(1, cols // 97)), [cols - 1]]))
    ref = Q.preprocess(x[at], 3, None, 4e7, 1e5, 12e6)
    assert rel(got[at], ref) <= 1e-5
    assert np.isfinite(got).all()


def test_cumtrapz_of_long_columns(cuda):
    # T = 13001: the column is walked in global memory; with K = identity and a
    # signal that ends early the image equals the short recording's
    import torch
    from msot_gb300 import backproject_waveeq
    g = GEOM
    T, D = 901, 5
    rng = np.random.default_rng(0)
    sig = torch.tensor(rng.standard_normal((1, D, T)).astype(np.float32), device="cuda")
    long = torch.nn.functional.pad(sig, (0, 13001 - T))
    x = np.linspace(-0.003, 0.003, 20)
    args = (g["c"], g["fs"], 0.0, g["coverage"], g["R"], np.array([[1.0]]))
    a = backproject_waveeq(sig, x, x, *args, torch.eye(T, device="cuda"))
    b = backproject_waveeq(long, x, x, *args, torch.eye(13001, device="cuda"))
    assert rel(b.cpu().numpy(), a.cpu().numpy()) < 1e-6
