"""The DAS kernels whose lanes run over instances (batches above 8 forward, above
4 adjoint) at the edges of their tiles: part-filled instance tiles of 8, 16 and
32, odd detector counts, grids that are no multiple of the pixel blocks,
interpolation radii below one and up to nine samples, and knots that coincide
(r with fraction 0 and 1/2).  Bars of test_gpu_operator.py: 1e-5 relative to
the oracle's C operators in FP64."""
import numpy as np
import pytest

from oracle import native
from pairs import make_pair, rel

pytestmark = pytest.mark.gpu


# (n, fov_half in mm, W): r = 2 fov_half / (n - 1) / 0.0375 mm
@pytest.mark.parametrize("n,fov,W", [
    (70, 0.8, 5),             # r = 0.62
    (33, 1.2, 9),             # r = 2: p1 = 0
    (65, 3.0, 13),            # r = 2.5: p1 = p2
    (40, 3.9, 16),            # r = 5.33
    (31, 3.0, 17),            # r = 5.33
    (31, 4.95, 31),           # r = 8.8
    (37, 4.0, 33),
    (66, 5.0, 64),
])
def test_batched_interpolation_matches_oracle(cuda, n, fov, W):
    import torch
    D = 7
    pm, om = make_pair(n=n, n_det=D, n_samples=1300, radius=0.02, fov_half=fov * 1e-3,
                       norm=2e-5, max_batch=W)
    rng = np.random.default_rng(n + W)
    x = rng.random((W, n * n))
    y = pm.interp_forward(torch.tensor(x, dtype=torch.float32)).cpu().numpy()
    ref = native.port().forward_das(x.T, om.travel, om.n_t, om.radius)
    assert rel(y, np.transpose(ref, (2, 0, 1))) < 1e-5
    s = rng.standard_normal((W, D, 1300))
    xa = pm.interp_transpose(torch.tensor(s, dtype=torch.float32)).cpu().numpy()
    refa = native.port().transpose_das(np.ascontiguousarray(np.transpose(s, (1, 2, 0))),
                                       om.travel, om.radius)
    assert rel(xa, refa.T) < 1e-5
    # every instance is its own: the last one alone gives the same
    alone = pm.interp_forward(torch.tensor(x[-1:], dtype=torch.float32)).cpu().numpy()
    assert rel(alone, y[-1:]) < 1e-6
    alone = pm.interp_transpose(torch.tensor(s[-1:], dtype=torch.float32)).cpu().numpy()
    assert rel(alone, xa[-1:]) < 1e-6
    # through the convolution, which takes the support only
    yc = pm.forward(torch.tensor(x, dtype=torch.float32).reshape(W, n, n)).cpu().numpy()
    assert rel(yc[-2:], om.forward(x[-2:].reshape(2, n, n))) < 1e-5
    xc = pm.transpose(torch.tensor(s, dtype=torch.float32)).cpu().numpy()
    assert rel(xc[-2:], om.transpose(s[-2:])) < 1e-5
