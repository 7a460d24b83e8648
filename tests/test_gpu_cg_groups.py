"""PCG with right-hand-side counts around the vector kernels' groups (17) and
batches (4), ragged sample counts around their 256-sample slices, and grids
whose split intermediates are padded to tiles, against the FP64 oracle.

Tolerances: the operator's products carry 17-bit operands (about 1e-5 of the
result's norm); a solve stopped at a residual tolerance and a Hutchinson
average follow it within 1e-3, the bound of the other cg tests."""
import numpy as np
import pytest
import torch

from fbme_b200 import scenes
from gpu_util import need_gpu, rel_l2
from oracle import fbme_oracle as O

CASES = [((24, 20), (13, 11), 1, 1), ((24, 20), (16, 16), 15, 2), ((32, 40), (17, 16), 16, 1),
         ((40, 36), (21, 19), 17, 2), ((36, 132), (16, 33), 34, 1)]


def _engine(grid, sample, probes, batch, **over):
    from fbme_b200.cg import CGEngine
    from torch_sbl import SBLConfig

    cfg = SBLConfig(mode="cg", active_set=False, hutchinson_probes=probes, initial_hutchinson_probes=min(probes, 16),
                    max_hutchinson_probes=probes, auto_probe_scaling=False, **over)
    return CGEngine(batch, grid, sample, cfg, torch.device("cuda", 0))


@pytest.mark.gpu
@pytest.mark.parametrize("grid,sample,probes,batch", CASES)
def test_matvec_group_sizes(grid, sample, probes, batch):
    need_gpu()
    eng = _engine(grid, sample, probes, batch, max_iter=2)
    rng = np.random.default_rng(probes)
    n, m, r = grid[0] * grid[1], sample[0] * sample[1], 1 + probes
    prior = rng.uniform(0.1, 2.0, (batch, n)).astype(np.float32)
    noise = rng.uniform(0.5, 1.0, batch).astype(np.float32)
    v = (rng.standard_normal((batch, r, m)) + 1j * rng.standard_normal((batch, r, m))).astype(np.complex64)
    got = eng.matvec(torch.from_numpy(prior).cuda(), torch.from_numpy(noise).cuda(), torch.from_numpy(v).cuda())
    eng.close()
    coeff = np.fft.ifft2(v.astype(np.complex128).reshape(batch, r, *sample), s=grid) * n
    coeff *= prior.astype(np.float64).reshape(batch, 1, *grid)
    want = np.fft.fft2(coeff)[..., : sample[0], : sample[1]].reshape(batch, r, m)
    want += noise.astype(np.float64)[:, None, None] * v
    for b in range(batch):
        for j in range(r):
            assert rel_l2(got[b, j].cpu().numpy(), want[b, j]) < 3e-5


@pytest.mark.gpu
@pytest.mark.parametrize("grid,sample,probes,batch", CASES)
def test_solve_group_sizes(grid, sample, probes, batch):
    need_gpu()
    n, m = grid[0] * grid[1], sample[0] * sample[1]
    ys = np.stack([scenes.point_scene(grid, sample, max(2, n // 40), 20.0, 70 + i).y for i in range(batch)])
    eng = _engine(grid, sample, probes, batch, max_iter=3, tol=0.0)
    z = O.rademacher_probes(batch, m, probes, 0)
    res = eng.solve(torch.from_numpy(ys.reshape(batch, m)).cuda(),
                    torch.from_numpy(np.ascontiguousarray(np.swapaxes(z, 1, 2)).astype(np.float32)).cuda())
    eng.close()
    o = O.fast_sbl_cg(ys.astype(np.complex128), grid, O.OracleConfig(
        mode="cg", active_set=False, max_iter=3, tol=0.0, hutchinson_probes=probes,
        initial_hutchinson_probes=min(probes, 16), max_hutchinson_probes=probes, auto_probe_scaling=False),
        probes=z, chol_mode="cuda")
    for b in range(batch):
        assert rel_l2(res.x[b].cpu().numpy(), o["x"][b]) < 1e-3
        assert rel_l2(res.precision[b].cpu().numpy(), o["precision"][b]) < 1e-3
    assert int(res.status.abs().sum()) == 0
