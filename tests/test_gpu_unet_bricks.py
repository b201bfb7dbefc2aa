"""U-Net weight gradients (k_wgrad, csrc/unet.cu) of grids with more bricks of 8 x 8
x 4 voxels than CTAs along the brick axis, where a CTA walks several bricks through
its two buffers: level 0 to 2 of these grids, in channel tiles of 32 and of 16, some
CTAs taking one brick more than others.  The activations are exact and the reference
has the GPU's bf16 storage (see test_gpu_unet.py), so what is left is FP32 sums and
the few gradients they push over a rounding boundary: one bf16 step of every value,
2^-8."""
import numpy as np
import pytest

from test_gpu_unet import U, _flat, _sparse_case, _unflat

pytestmark = pytest.mark.gpu

SMS = 148
LEVEL = {"W0": 0, "W1": 1, "W2": 2, "W3": 3, "W4": 2, "W5": 1, "W6": 0}
GRIDS = [(64, 64, 64), (72, 56, 64), (96, 40, 72)]


def _bricks_and_ctas(dims, k):
    """Bricks of weight k's level, and the CTAs along the brick axis (wgrad_launch)."""
    nx, ny, nz = (d >> LEVEL[k] for d in dims)
    cin, cout = U.CH[k]
    bricks = -(-nx // 8) * -(-ny // 8) * -(-nz // 4)
    ch = 32 if cin % 32 == 0 else 16
    tiles = (cout // 16) * (cin // ch)
    return bricks, -(-((1 if ch == 32 else 2) * SMS) // tiles)


def test_the_grids_reach_the_walk():
    walks = {(d, k): _bricks_and_ctas(d, k) for d in GRIDS for k in U.NAMES}
    reached = {k for (d, k), (b, c) in walks.items() if b > c and b % c}
    assert reached >= {"W0", "W1", "W4", "W5", "W6"}  # 16 input channels a tile: W0, W1; 32: the others


@pytest.mark.parametrize("nx,ny,nz", GRIDS)
def test_gradients_over_several_bricks(ctx, nx, ny, nz):
    import bsg
    import torch
    W, r, t, d, _, want = _sparse_case(nx, ny, nz)
    net = bsg.UNet(ctx, nx, ny, nz, train=True)
    net.set_weights(_flat(W))
    net.set_diag(torch.as_tensor(d, device="cuda"))
    net.train_sample(torch.as_tensor(r, device="cuda"), torch.as_tensor(t, device="cuda"))
    G = _unflat(net.grads())
    for k in want:
        err = np.linalg.norm(G[k] - want[k])
        assert err <= 2.0 ** -8 * np.linalg.norm(want[k]), (k, err)
    net.free()
