"""The warm-start network on volumes far from a cube, against the FP64 restatement
(oracle/warmnet_ref.py); the tolerances are those of test_warm_kernels.py."""
import numpy as np
import pytest

from gpesolver_b200 import warmstart as W

from . import test_warm_kernels as K

pytestmark = pytest.mark.gpu


# coarse volumes of 36 x 1 x 1, 64 x 2 x 1, 33 x 1 x 2, 40 x 2 x 1 and 34 x 1 x 1 voxels: the
# weight gradient's tiles are cut along x to fit into shared memory
@pytest.mark.parametrize("dims,levels,channels,batch", [
    ((72, 2, 2), 1, (8, 8), 2),
    ((128, 4, 2), 1, (8, 8), 1),
    ((66, 2, 4), 1, (16, 1), 2),
    ((80, 4, 2), 1, (4, 32), 1),
    ((272, 8, 8), 3, (8, 8, 8, 8), 1),
])
def test_thin_volumes_match_fp64(dims, levels, channels, batch):
    K.test_edges_match_fp64(dims, levels, channels, batch)


# more than 65535 chunks or blocks along x in the kernels that had them on a grid's second axis:
# a latent volume of 2.1 M values, the last convolution forward, its input gradient
@pytest.mark.parametrize("dims,levels,channels,batch", [
    ((64, 64, 16), 0, (32,), 1),
    ((262152, 1, 1), 0, (1,), 1),
    ((65544, 2, 2), 1, (8, 32), 1),
])
def test_long_volumes_match_fp64(dims, levels, channels, batch):
    K.test_edges_match_fp64(dims, levels, channels, batch)


def test_amplitudes_into_any_buffer():
    """Pinned host memory and an odd device address take the same bytes as a tensor on the device."""
    import torch

    net = W.WarmStartNet(W.WarmConfig(nx=16, ny=16, nz=8, levels=1, channels=(4, 4), hidden=8, max_batch=2), seed=1)
    x = np.random.default_rng(2).uniform(-1, 1, (2, 4)).astype(np.float32)
    n = 2 * net.n_voxels
    amp = torch.zeros(n, device="cuda")
    host = torch.zeros(n, pin_memory=True)
    odd = torch.zeros(4 * n + 8, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    net.forward(x, amp.data_ptr())
    net.forward(x, host.data_ptr())
    net.forward(x, odd.data_ptr() + 2)
    net.close()
    want = amp.cpu().numpy()
    assert np.abs(want).max() > 0
    assert np.array_equal(host.numpy(), want)
    assert odd[2:2 + 4 * n].cpu().numpy().tobytes() == want.tobytes()
