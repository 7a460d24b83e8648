"""Dense mode's blocked in-place inverse at the edges of its panels (32) and
tiles (64): sample counts below, at and just above them, a ragged last panel,
several tiles, and a batch, against the FP64 oracle.

Tolerance: the prior and noise are FP32 between the EM iterations (6e-8 a
rounding), everything else FP64; three iterations on 20 dB scenes keep that
within two orders of magnitude, and the posterior variance gamma - gamma^2 dd
loses up to three more digits to cancellation."""
import numpy as np
import pytest
import torch

from fbme_b200 import scenes
from gpu_util import need_gpu
from oracle import fbme_oracle as O


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.gpu
@pytest.mark.parametrize("grid,sample,batch", [
    ((4, 4), (1, 1), 1), ((8, 8), (5, 6), 1), ((8, 8), (8, 4), 2), ((16, 8), (11, 3), 1), ((16, 16), (9, 7), 1),
    ((16, 16), (8, 8), 1), ((16, 16), (13, 5), 3), ((24, 16), (12, 8), 1), ((24, 20), (19, 17), 2)])
def test_dense_inverse_sizes(grid, sample, batch):
    need_gpu()
    from torch_sbl import SBLConfig, sbl_2d

    n = grid[0] * grid[1]
    ys = np.stack([scenes.point_scene(grid, sample, max(1, n // 20), 20.0, 40 + i).y for i in range(batch)])
    res = sbl_2d(torch.from_numpy(ys).cuda(), grid, config=SBLConfig(mode="dense", max_iter=3, tol=0.0))
    for i in range(batch):
        o = O.fast_sbl_dense(ys[i].astype(np.complex128), grid, O.OracleConfig(mode="dense", max_iter=3, tol=0.0))
        assert rel(res.x[i].cpu().numpy(), o["x"]) < 1e-5
        assert rel(res.precision[i].cpu().numpy(), o["precision"]) < 1e-5
        assert rel(res.posterior_variance[i].cpu().numpy(), o["posterior_variance"]) < 1e-3
        assert abs(float(res.noise_variance[i]) - o["noise_variance"]) < 1e-5 * o["noise_variance"]
    assert int(res.status.abs().sum()) == 0
