"""Tall grids, whose Dirichlet tables and polish state together take more than
48 KB of shared memory: single plans, an uneven plan and the certificate, up to
N1 + N2 of nearly 4032.

The prefix is the whole grid, so the atoms are orthogonal and the answer has a
closed form in FP64: the support is the 32 largest pixels of the inverse DFT z
of the data, x there is z gamma M / (gamma M + nu) of the result's own prior
variances and noise, and an inactive atom's evidence ratio is M |z|^2 / nu.  (The FP32 oracle's column
phases lose up to 1e-3 on axes this long.)

Tolerance: the plan tests' 1e-4 on x; the operator's error is 1e-5 of the
largest pixel at most, a few times the pixel of the ratio, so 1e-4 on it too."""
import numpy as np
import pytest
import torch

from fbme_b200 import scenes
from gpu_util import X_TOL, need_gpu, rel_l2

K = 32


def _scene(grid, seed):
    sc = scenes.point_scene(grid, grid, 60, 20.0, seed, "rayleigh")
    return sc.y, np.fft.ifft2(sc.y.astype(np.complex128)).reshape(-1)


def _check(res, z):
    x = res.x.cpu().numpy().reshape(-1)
    top = np.argsort(-np.abs(z))[:K]
    assert set(np.flatnonzero(x)) == set(top)
    gain = z.size / res.precision.cpu().numpy().reshape(-1)[top].astype(np.float64)
    assert rel_l2(x[top], z[top] * gain / (gain + float(res.noise_variance))) < X_TOL


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [(3600, 128), (3600, 90), (4000, 32), (3254, 2)])
def test_tall_plan(grid):
    need_gpu()
    from torch_sbl_fastest_stable import make_fastest_plan

    data, z = _scene(grid, 7)
    y = torch.from_numpy(data).cuda()
    res = make_fastest_plan(y, grid, polish_size=K).replay(y, synchronize=True)
    _check(res, z)
    assert int(res.status.abs().sum()) == 0


@pytest.mark.gpu
def test_tall_uneven_plan():
    need_gpu()
    from fbme_b200.uneven import make_uneven_plan

    grids = [(3600, 64), (40, 32)]
    data, zs = zip(*(_scene(g, 3) for g in grids))
    ys = [torch.from_numpy(d).cuda() for d in data]
    res = make_uneven_plan(ys, grids, profile="fast", polish_size=K).replay(ys, synchronize=True)
    for r, z in zip(res, zs):
        _check(r, z)


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [(3600, 128), (3880, 128)])
def test_tall_certificate(grid):
    need_gpu()
    from fbme_b200.config import SBLConfig
    from torch_sbl import sbl_2d

    data, z = _scene(grid, 11)
    cfg = SBLConfig.certified_hybrid_uamp(device="cuda", uamp_polish_size=K, uamp_polish_support_repairs=1)
    res = sbl_2d(torch.from_numpy(data).cuda(), grid, config=cfg)
    _check(res, z)
    best = np.argsort(-np.abs(z))[K]
    want = z.size * abs(z[best]) ** 2 / float(res.noise_variance)
    assert int(res.inactive_best_index) == best
    assert abs(float(res.inactive_max_evidence_ratio) - want) <= 1e-4 * want
    assert int(res.status) == 0
