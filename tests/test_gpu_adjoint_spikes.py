"""A NaN, an infinity or a spike in the recording reaches the pixels whose taps meet it
and no other, whatever kernel serves the batch: those others keep their bits."""
import numpy as np
import pytest

from pairs import make_pair

pytestmark = pytest.mark.gpu


# r = 2 fov / (n - 1) / 0.0375 mm; batches with 8, 16 and 32 instances per tile
@pytest.mark.parametrize("n,fov,W", [(70, 0.8, 5), (65, 3.0, 13), (40, 3.9, 17), (31, 4.95, 5),
                                     (66, 5.0, 48), (40, 3.9, 1)])
def test_samples_reach_their_own_pixels(cuda, n, fov, W):
    import torch
    D, T = 3, 1300
    pm, om = make_pair(n=n, n_det=D, n_samples=T, radius=0.02, fov_half=fov * 1e-3, eir_taps=0,
                       norm=2e-5, max_batch=W)
    rng = np.random.default_rng(n)
    s = rng.standard_normal((W, D, T)).astype(np.float32)
    clean = pm.interp_transpose(torch.tensor(s)).cpu().numpy().reshape(W, -1)
    tau = np.asarray(om.travel).reshape(D, -1)
    t0 = int(np.median(tau[1]))
    far = np.abs(tau[1] - t0) > om.radius + 1
    assert far.any() and not far.all()
    for bad in (1e6, np.inf, np.nan):
        s[W - 1, 1, t0] = bad
        got = pm.interp_transpose(torch.tensor(s)).cpu().numpy().reshape(W, -1)
        assert np.array_equal(got[:-1], clean[:-1])
        assert np.array_equal(got[-1][far], clean[-1][far])
        near = np.abs(tau[1] - t0) < om.radius - 1e-3
        if near.any() and bad != 1e6:
            assert not np.isfinite(got[-1][near]).any()
