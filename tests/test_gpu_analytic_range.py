"""The analytic path's sums in pairs of floats where they leave FP32's range: recordings
scaled by a power of two give results scaled by it, as FP64 sums would.  1e-6: FP32 results
whose last bit may differ."""
import numpy as np
import pytest

from pairs import rel

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("window,band", [((2, 300.0, 700.0), (0.0, 0.0)), (None, (1e5, 12e6))])
def test_columns_of_large_samples(cuda, window, band):
    import torch
    from msot_gb300.preprocess import Preprocessor
    T = 1501
    big = 2.0 ** 123  # 1.1e37; a lane's sum over 47 samples passes 3.4e38
    x = (2 + np.random.default_rng(1).random((9, T))).astype(np.float32)
    p = Preprocessor(T, 0, window, 4e7, *band, max_cols=9)
    want = p(torch.tensor(x)).cpu().numpy().astype(np.float64)
    got = p(torch.tensor(x * np.float32(big))).cpu().numpy().astype(np.float64) / big
    assert np.isfinite(got).all()
    # the band-pass removes the offset: what it leaves is measured against the input
    assert np.abs(got - want).max() < 1e-6 * 3


@pytest.mark.parametrize("T", [901, 13001])  # columns in shared memory, in global memory
def test_backprojection_of_large_samples(cuda, T):
    import torch
    from msot_gb300 import backproject_waveeq
    D, big = 5, 2.0 ** 118  # 3.3e35; the sum over a column passes 3.4e38
    sig = torch.tensor(2 + np.random.default_rng(2).random((3, D, T)), dtype=torch.float32).cuda()
    x = np.linspace(-0.003, 0.003, 20)
    args = (1500.0, 4e7, 0.0, 135.0, 0.015, np.array([[1.0]]), torch.eye(T, device="cuda"))
    want = backproject_waveeq(sig, x, x, *args).cpu().numpy()
    got = backproject_waveeq(sig * big, x, x, *args).cpu().numpy()
    assert np.isfinite(got).all()
    assert rel(got / big, want) < 1e-6
