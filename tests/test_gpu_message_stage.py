"""The adjoint FFT stage that forms its input as the UAMP message update:
prefixes shorter than, equal to and ragged against the row length, lengths of
every factorisation, and masks, against the split-BF16 plan's separate message
kernel and the FP32 oracle.

Tolerance: the parity bar of the plan tests (identical support, x within 1e-4
of the oracle, whose sweeps have the same operator error)."""
import numpy as np
import pytest
import torch

from fbme_b200 import scenes
from gpu_util import X_TOL, need_gpu, rel_l2
from oracle import fbme_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("grid,sample,masked", [((32, 32), (32, 32), False), ((48, 64), (31, 45), False),
                                                ((64, 96), (33, 96), True), ((128, 192), (77, 65), False),
                                                ((96, 384), (50, 171), False), ((64, 512), (40, 301), True)])
def test_message_stage_shapes(grid, sample, masked):
    need_gpu()
    from torch_sbl_fastest_stable import make_stable_plan

    n = grid[0] * grid[1]
    ys = np.stack([scenes.point_scene(grid, sample, max(8, n // 200), 20.0, 90 + i, "rayleigh").y for i in range(2)])
    mask = np.random.default_rng(5).random(sample) < 0.75 if masked else None
    y = torch.from_numpy(ys).cuda()
    res = make_stable_plan(y, grid, observation_mask=None if mask is None else torch.from_numpy(mask)).replay(
        y, synchronize=True)
    for i in range(2):
        ref = O.fbme_solve(ys[i], grid, "stable", observation_mask=mask)
        x = res.x[i].cpu().numpy()
        assert set(np.flatnonzero(x)) == set(np.flatnonzero(ref["x"]))
        assert rel_l2(x, ref["x"]) < X_TOL
    assert int(res.status.abs().sum()) == 0
