"""The certificate scan's atom pairs at the edges: odd and tiny row lengths,
fewer pairs than threads, masked (2-D Gram table) and separable tables, small
active sets: the inactive certificate of the device's own final model against
|a_j^H C^-1 y|^2 / (a_j^H C^-1 a_j) evaluated in FP64 for every atom.

Tolerance: at most 32 substitution terms at 6e-8 each, and the atom precision
M / nu - |v|^2 / nu^2 loses at most another 50 to cancellation for atoms that
still lead: 1e-4 on the ratio; the reported atom's ratio must be the FP64
maximum to that accuracy."""
import numpy as np
import pytest
import torch

from fbme_b200 import scenes
from gpu_util import need_gpu


def _ratios(y, grid, mask, active, gamma, nu):
    """FP64 inactive ratios [N] of the model (active, gamma, nu)."""
    m1, m2 = y.shape
    i1, i2 = np.meshgrid(np.arange(m1), np.arange(m2), indexing="ij")
    keep = np.ones(y.shape, bool) if mask is None else mask
    i1, i2, d = i1[keep], i2[keep], y[keep].astype(np.complex128)
    n1, n2 = np.divmod(np.arange(grid[0] * grid[1]), grid[1])
    a = np.exp(-2j * np.pi * (np.outer(i1, n1) / grid[0] + np.outer(i2, n2) / grid[1]))
    s = a[:, active]
    c = nu * np.eye(d.size) + (s * gamma) @ s.conj().T
    num = np.abs(a.conj().T @ np.linalg.solve(c, d)) ** 2
    den = np.einsum("mn,mn->n", a.conj(), np.linalg.solve(c, a)).real
    r = num / den
    r[active] = 0.0
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("grid,sample,k,masked", [((8, 9), (6, 7), 5, False), ((16, 33), (12, 25), 8, False),
                                                  ((48, 32), (30, 20), 32, False), ((17, 64), (13, 40), 32, False),
                                                  ((24, 25), (20, 19), 9, True), ((32, 32), (24, 24), 31, True)])
def test_scan_pairs(grid, sample, k, masked):
    need_gpu()
    from torch_sbl import SBLConfig, sbl_2d

    sc = scenes.point_scene(grid, sample, max(2, k // 2), 25.0, 5, "rayleigh")
    mask = np.random.default_rng(3).random(sample) < 0.8 if masked else None
    cfg = SBLConfig.certified_hybrid_uamp(device="cuda", uamp_polish_size=k, uamp_polish_iterations=2,
                                          uamp_polish_support_repairs=1)
    res = sbl_2d(torch.from_numpy(sc.y).cuda(), grid, config=cfg, observation_mask=mask)
    active = np.flatnonzero(res.x.cpu().numpy().reshape(-1))
    gamma = 1.0 / res.precision.cpu().numpy().reshape(-1)[active].astype(np.float64)
    r = _ratios(sc.y, grid, mask, active, gamma, float(res.noise_variance))
    best, got = int(res.inactive_best_index), float(res.inactive_max_evidence_ratio)
    assert len(active) == k and best not in active
    assert abs(got - r[best]) <= 1e-4 * r[best]
    assert r[best] >= r.max() * (1.0 - 1e-4)
