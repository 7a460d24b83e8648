"""The adjoint FFT stage with the denoiser in its epilogue over a batch in
which every block takes three and more tiles in turn (both row buffers, the
last tile without a successor), against the batch of the same scenes in which
a block takes one, bit for bit: lengths with two buffers and with one, whole
and ragged row tiles."""
import numpy as np
import pytest
import torch

from fbme_b200 import scenes
from gpu_util import need_gpu


@pytest.mark.gpu
@pytest.mark.parametrize("grid,sample", [((64, 48), (31, 25)), ((96, 64), (96, 40)), ((128, 48), (61, 48)),
                                         ((256, 48), (129, 20)), ((256, 64), (255, 33))])
def test_tiles_of_a_block_in_turn(grid, sample):
    need_gpu()
    from fbme_b200.config import fbme_profile_config
    from fbme_b200.engine import FBMEEngine

    dev = torch.device("cuda", 0)
    cfg = fbme_profile_config("stable")
    cfg.dft_terms = 0
    few, many = 4, 4 * 128
    ys = np.stack([scenes.point_scene(grid, sample, 40, 20.0, 30 + i, "rayleigh").y.reshape(-1) for i in range(few)])
    y = torch.from_numpy(ys).to(dev)
    out = []
    for reps in (1, many // few):
        eng = FBMEEngine(few * reps, grid, sample, cfg, dev)
        eng.run(y.repeat(reps, 1).contiguous())
        torch.cuda.synchronize()
        out.append({f: eng.out[f].clone() for f in ("x", "posterior_variance", "precision", "noise_variance")})
        eng.close()
    for f, one in out[0].items():
        assert torch.equal(out[1][f], one.repeat(many // few, *(1,) * (one.dim() - 1))), f
