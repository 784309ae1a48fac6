"""SB_ITV2 by thread-block clusters, with part of its vectors in registers
(clusters of 4, 8 and 16 CTAs with two to four groups of pixels per thread) and
without: slabs that end ragged, threads that own fewer groups than the others,
columns that do not fill their last group of four pixels."""
import numpy as np
import pytest

from oracle import solvers as S
from pairs import rel
from test_gpu_tv import _noisy_blocks

pytestmark = pytest.mark.gpu


# C: CTAs per image (0: chosen by the number of images)
# 1e-3: the bar of the prox (its own stopping rule is a change of 1e-3); the
# images of one call do not influence each other
@pytest.mark.parametrize("n,W,C", [(132, 1, 4), (148, 2, 4), (160, 1, 4), (160, 1, 8),
                                   (172, 1, 8), (200, 1, 8), (200, 9, 0), (236, 1, 16),
                                   (256, 1, 16), (160, 20, 0),
                                   (3, 2, 0), (6, 1, 2), (97, 3, 0), (143, 1, 4), (161, 1, 8),
                                   (199, 2, 0), (201, 10, 0), (235, 1, 16), (302, 1, 0)])
def test_sb_itv2_with_vectors_in_registers(cuda, n, W, C):
    import torch
    from msot_gb300 import SB_ITV2, _lib
    L = _lib.load()
    g = _noisy_blocks(n, W, 500 + n)
    _lib.check(L.msot_tune_set(b"tv_prox_cluster", C))
    try:
        u = SB_ITV2(torch.tensor(g, dtype=torch.float32), 0.05).cpu().numpy()
    finally:
        _lib.check(L.msot_tune_set(b"tv_prox_cluster", 0))
    B, Bt, BtB = S.diff_oper(n)
    for w in {0, W - 1}:
        ref = S.sb_itv2(g[w].T, 0.05, B, Bt, BtB).reshape(n, n, order="F").T
        assert rel(u[w], ref) <= 1e-3
    assert np.isfinite(u).all()
