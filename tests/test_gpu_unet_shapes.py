"""The network's prediction at the edges of its tensor-core tiles: sides that
do not fill them, decoders that read their two inputs in place, pooled and
final layers in the convolution's epilogue, the narrow first layer."""
import numpy as np
import pytest

from test_gpu_unet import _ref_forward

pytestmark = pytest.mark.gpu


# sides whose coarsest level is odd or smaller than a tile; large batches and a
# batch of one; 64 and 96 channels at the top (the final layer inside and
# outside the epilogue); 16 (the top decoder on the CUDA cores); 3 input
# channels (the general first layer).
# TF32 activations, 2^-11 relative per layer and up to 15 layers: 3e-3, the
# bar of the network's other tests.  One image alone sums in the order of the
# batch: only the rounding of equal sums, 1e-5, may differ.
@pytest.mark.parametrize("L,c0,side,n,cin", [(4, 32, 72, 24, 1), (3, 32, 28, 70, 1),
                                             (2, 64, 24, 60, 2), (2, 96, 10, 90, 1),
                                             (3, 16, 36, 50, 1), (2, 32, 130, 2, 3),
                                             (2, 32, 8, 1, 1)])
def test_prediction_matches_the_reference_at_tile_edges(cuda, L, c0, side, n, cin):
    import torch
    from msot_gb300.warmstart import UNet
    net = UNet(levels=L, base_channels=c0, side=side, max_batch=n, seed=11, in_channels=cin)
    rng = np.random.default_rng(5)
    x = rng.standard_normal((n, cin, side, side)).astype(np.float32)
    t = np.zeros((n, 1, side, side), dtype=np.float32)
    out = net.forward(x).cpu()
    one = net.forward(x[-1:]).cpu()
    net.check()
    ref = _ref_forward(torch, torch.tensor(net.get_params()), torch.tensor(x), L, c0, [],
                       cin).detach()
    assert float((out - ref).norm() / ref.norm()) < 3e-3
    assert float((out[-1:] - one).norm() / one.norm()) < 1e-5
    # the training pass writes the concatenated inputs and the last decoder
    # layer; its loss against zero is the mean square of the prediction
    loss, _ = net.gradients(x, t)
    net.check()
    want = float((out.double() ** 2).mean())
    assert abs(loss - want) < 1e-5 * want
