"""The warm-start network's convolution kernels at the edges of their tiles and
of their dispatch, against the FP64 restatement (oracle/warmnet_ref.py).

Tolerance: a gradient entry is an FP32 sum of at most ~1000 terms in a row and
then a tree, a random-walk error of sqrt(1000) 2^-24 = 2e-6 of the terms' scale;
five layers in a chain and sums that cancel to a tenth of their terms' scale
give 1e-4 of a tensor's norm.  The forward pass (at most 32 x 8 terms a sum)
stays below 1e-5 of the amplitude's norm."""
import numpy as np
import pytest

from gpesolver_b200 import warmstart as W
from oracle.warmnet_ref import WarmNetRef

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,levels,channels,batch", [
    ((8, 8, 8), 3, (1, 2, 1, 1), 1),              # one coarse voxel, single channels
    ((16, 48, 16), 4, (32, 32, 16, 8, 8), 2),     # every channel group, odd coarse edges (1, 3, 1)
    ((40, 24, 8), 3, (16, 16, 8, 4), 9),          # ragged tiles, more than eight samples
    ((6, 10, 4), 1, (4, 32), 3),                  # 32 channels into the last convolution
    ((37, 5, 3), 0, (8,), 2),                     # no upsampling: the last convolution alone
    ((72, 64, 32), 2, (8, 8, 8), 2),              # large volume: two voxels a thread
    ((70, 96, 32), 1, (8, 8), 2),                 # its odd coarse edge along x
])
def test_edges_match_fp64(dims, levels, channels, batch):
    import torch

    nx, ny, nz = dims
    cfg = W.WarmConfig(nx=nx, ny=ny, nz=nz, levels=levels, channels=channels, hidden=20, max_batch=batch)
    net = W.WarmStartNet(cfg, seed=3)
    ref = WarmNetRef(nx, ny, nz, levels, channels, hidden=20)
    rng = np.random.default_rng(4)
    w = net.get_weights() + rng.uniform(-0.05, 0.05, net.n_weights).astype(np.float32)
    net.set_weights(w)
    x = rng.uniform(-1, 1, (batch, 4)).astype(np.float32)
    t = rng.uniform(0, 2, (batch, nx * ny * nz)).astype(np.float32)
    amp = torch.empty(batch, nx * ny * nz, device="cuda")
    net.forward(x, amp.data_ptr())
    loss, g = net.gradients(x, torch.tensor(t, device="cuda").data_ptr())
    net.close()
    rloss, rg = ref.loss_and_grad(w, x, t)
    got = amp.double().cpu().numpy()
    # the loss holds the whole amplitude: mean((a - t)^2)
    assert abs(((got - t) ** 2).mean() - rloss) <= 1e-5 * rloss
    assert abs(loss - rloss) <= 1e-5 * rloss
    for name, (o, n) in ref.off.items():
        d = np.linalg.norm(g[o:o + n] - rg[o:o + n])
        assert d <= 1e-4 * np.linalg.norm(rg[o:o + n]), (name, d)
