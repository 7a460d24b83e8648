"""The UAMP message update formed in the load of the adjoint FFT stage against
the separate message kernel, which the split-BF16 stages of the same problem
run, at row lengths of the main workloads with ragged prefixes and a mask; and
the merged launches of an uneven plan against the single ones, bit for bit.

Tolerance: both forms meet the plan tests' bar (identical support, x within
1e-4 of the FP32 oracle), so they lie within twice that of each other."""
import numpy as np
import pytest
import torch

from fbme_b200 import scenes
from gpu_util import X_TOL, need_gpu, rel_l2
from oracle import fbme_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("grid,sample,masked", [((96, 48), (50, 31), False), ((64, 128), (40, 77), False),
                                                ((64, 128), (40, 77), True), ((128, 256), (70, 201), False)])
def test_message_forms_agree(grid, sample, masked):
    need_gpu()
    from fbme_b200.config import fbme_profile_config
    from fbme_b200.plans import CUDAGraphSBLPlan

    ys = np.stack([scenes.point_scene(grid, sample, 12, 20.0, 60 + i, "rayleigh").y for i in range(2)])
    mask = np.random.default_rng(5).random(sample) < 0.75 if masked else None
    y = torch.from_numpy(ys).cuda()
    got = {}
    for terms in (0, 3):
        cfg = fbme_profile_config("stable", polish_size=12)
        cfg.dft_terms = terms
        plan = CUDAGraphSBLPlan(y, grid, config=cfg, observation_mask=None if mask is None else torch.from_numpy(mask))
        got[terms] = plan.replay(y, synchronize=True).x.cpu().numpy()
    for i in range(2):
        ref = O.fbme_solve(ys[i], grid, "stable", polish_size=12, observation_mask=mask)["x"]
        for x in got.values():
            assert set(np.flatnonzero(x[i])) == set(np.flatnonzero(ref))
            assert rel_l2(x[i], ref) < X_TOL
        assert rel_l2(got[0][i], got[3][i]) < 2 * X_TOL


@pytest.mark.gpu
def test_merged_message_stage_equals_the_single_one():
    need_gpu()
    from fbme_b200.config import fbme_profile_config
    from fbme_b200.engine import FBMEEngine
    from fbme_b200.uneven import UnevenEngine

    dev = torch.device("cuda", 0)
    cfg = fbme_profile_config("stable")
    cfg.dft_terms = 0
    shapes = [((96, 48), (50, 31)), ((64, 128), (40, 77)), ((48, 128), (48, 128)), ((128, 256), (70, 201)), ((64, 384), (33, 160))]
    ys = [torch.from_numpy(scenes.point_scene(g, s, 40, 20.0, 8, "rayleigh").y).to(dev) for g, s in shapes]
    eng = UnevenEngine(shapes, cfg, dev)
    eng.run(eng.pack(ys))
    torch.cuda.synchronize()
    for i, (g, s) in enumerate(shapes):
        one = FBMEEngine(1, g, s, cfg, dev)
        one.run(ys[i].reshape(1, -1).contiguous())
        torch.cuda.synchronize()
        p0, n = eng.pix_off[i], g[0] * g[1]
        for f in ("x", "posterior_variance", "precision"):
            assert torch.equal(eng.out[f][p0:p0 + n], one.out[f][0]), (f, i)
        one.close()
    eng.close()
