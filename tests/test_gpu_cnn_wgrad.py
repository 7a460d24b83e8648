"""The warm-start network's weight gradient at the edges of its 16 x 32 pixel
tiles: grids smaller than a tile, ragged in either axis, and more tiles than
blocks, against the FP64 oracle on the device's own activations' roundings.

Tolerance: activations, weights and the propagated gradients are BF16 operands
(2^-9 each); the relative L2 bound and the cosine are those of the network's
other gradient test."""
import numpy as np
import pytest
import torch

from gpu_util import need_gpu, rel_l2
from oracle import cnn_oracle as C
from test_gpu_cnn import _flat_to_dict


def _reference(params, x, target):
    q = {k: C.bf16_round(v) if k.startswith("W") else v for k, v in params.items()}
    return C.loss_and_grads(q, C.bf16_round(x), target.astype(np.float64))


@pytest.mark.gpu
@pytest.mark.parametrize("batch,grid", [(1, (8, 16)), (3, (24, 16)), (2, (16, 32)), (2, (40, 48)), (5, (128, 256)),
                                        (1, (8, 272))])
def test_weight_gradient_tiles(batch, grid):
    need_gpu()
    from fbme_b200.learned import WarmStartNet, init_params

    rng = np.random.default_rng(batch)
    n = grid[0] * grid[1]
    bp = (rng.normal(size=(batch, n)) + 1j * rng.normal(size=(batch, n))).astype(np.complex64)
    target = rng.normal(size=(batch, *grid)).astype(np.float32)
    p = init_params(11)
    p[-1] = 0.3
    net = WarmStartNet(torch.device("cuda", 0), p)  # no plan in this process has to come first
    net.features(torch.from_numpy(bp).cuda(), *grid)
    net.forward(batch, *grid)
    loss = float(net.backward(torch.from_numpy(target.reshape(batch, -1)).cuda(), batch, *grid))
    ref_loss, _, ref = _reference(_flat_to_dict(p), C.features(bp, grid), target)
    assert abs(loss - ref_loss) < 5e-3 * ref_loss
    got = _flat_to_dict(net.grad.cpu().numpy())
    for k in ("W1", "b1", "W2", "b2", "W3", "b3"):
        a, b = got[k].ravel(), ref[k].ravel()
        assert rel_l2(a, b) < 2e-2, k
        assert float(a @ b / (np.linalg.norm(a) * np.linalg.norm(b))) > 0.999, k
