"""A plan tuned at one batch size runs the built-in kernels at others."""
import numpy as np
import pytest

from pairs import make_pair

pytestmark = pytest.mark.gpu


def _kernels(fn):
    import torch
    from torch.profiler import ProfilerActivity, profile
    for _ in range(2):  # the first session of a process may miss the launches
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            fn()
            torch.cuda.synchronize()
    return {e.key for e in p.key_averages()}


@pytest.mark.parametrize("batch", [1, 3, 4, 8])
def test_a_tuned_batch_leaves_the_others_alone(cuda, batch):
    import torch
    W = 32
    pm, _ = make_pair(n=48, n_det=64, n_samples=1200, radius=0.02, fov_half=0.0063, max_batch=W)
    rng = np.random.default_rng(batch)
    x = torch.tensor(rng.random((W, 48, 48)), dtype=torch.float32).cuda()
    y = torch.tensor(rng.random((W, 64, 1200)), dtype=torch.float32).cuda()
    for _ in range(4):  # a choice by the scatter of two timings would not hold
        t = pm.autotune(batch)
        assert t["fwd_wt"] > 0 and batch % t["adj_wt"] == 0
        assert any("k_das_fwd6" in k for k in _kernels(lambda: pm.forward(x)))
        assert any("k_das_adj5" in k for k in _kernels(lambda: pm.transpose(y)))
    t = pm.autotune(W)
    names = _kernels(lambda: pm.forward(x))
    want = {0: "k_das_fwd6", 1: "k_das_fwd_st", 2: "k_das_fwd3", 4: "k_das_fwd3"}
    assert any(want[t["fwd_staged"]] in k for k in names)
