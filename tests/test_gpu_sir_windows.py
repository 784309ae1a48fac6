"""The SIR interpolation on composite rows at its edges: windows cut by both ends
of the row, odd and even row lengths, columns longer than a warp's 64 samples,
part-filled instance tiles, radii with either order of the kinks, a NaN pixel.
Bars of test_gpu_operator.py: 1e-5 relative to the oracle's C operators."""
import numpy as np
import pytest

from oracle import native
from pairs import make_pair, rel

pytestmark = pytest.mark.gpu


# r = 2 fov / (n - 1) / 0.0375 mm
@pytest.mark.parametrize("n,fov,T,S,W", [
    (21, 2.0, 1301, 41, 1),    # r = 5.33, odd rows
    (21, 3.0, 830, 151, 3),    # r = 8: windows past the row's end, two chunks
    (33, 1.05, 1300, 91, 6),   # r = 1.75: first kink after the second
    (30, 0.4, 1300, 11, 17),   # r = 0.74
])
def test_sir_operator_at_window_edges(cuda, n, fov, T, S, W):
    import torch
    rng = np.random.default_rng(S)
    D, NS = 5, 13
    sir = rng.standard_normal((NS, S))
    se = np.stack([rng.integers(1, S // 2, NS), rng.integers(S // 2, S + 1, NS)], 1)
    se = se.astype(np.int32)
    idx = rng.integers(1, NS + 1, (D, n * n)).astype(np.int32)
    pm, om = make_pair(n=n, n_det=D, n_samples=T, radius=0.028, fov_half=fov * 1e-3, norm=2e-5,
                       max_batch=W, sir_tables=(sir, se, idx))
    x = rng.random((W, n * n))
    y = pm.interp_forward(torch.tensor(x, dtype=torch.float32)).cpu().numpy()
    ref = native.port().forward_sir(np.ascontiguousarray(x.T), idx, om.travel, sir, T, se,
                                    om.radius)
    assert rel(y, np.transpose(ref, (2, 0, 1))) < 1e-5
    s = rng.standard_normal((W, D, T))
    xa = pm.interp_transpose(torch.tensor(s, dtype=torch.float32)).cpu().numpy()
    refa = native.port().transpose_sir(np.ascontiguousarray(np.transpose(s, (1, 2, 0))), idx,
                                       om.travel, sir, se, om.radius)
    assert rel(xa, refa.T) < 1e-5
    yc = pm.forward(torch.tensor(x, dtype=torch.float32).reshape(W, n, n)).cpu().numpy()
    assert rel(yc[:1], om.forward(x[:1].reshape(1, n, n))) < 1e-5
    xc = pm.transpose(torch.tensor(s, dtype=torch.float32)).cpu().numpy()
    assert rel(xc[:1], om.transpose(s[:1])) < 1e-5
    # the adjoint of an unread sample's NaN is untouched
    lo = int(om.travel.min() - om.radius) - S
    if lo > 0:
        s[:, :, :lo] = np.nan
        again = pm.interp_transpose(torch.tensor(s, dtype=torch.float32)).cpu().numpy()
        assert np.array_equal(again, xa)
