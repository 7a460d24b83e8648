"""Workspace of a cg plan: the padding of the matvec's split intermediates is
not needed for a plan to run, so a solve that fits the device without it still
runs, with the same results."""
import ctypes

import numpy as np
import pytest

from fbme_b200 import _native as nat
from fbme_b200.cg import resolve_cg_config
from fbme_b200.config import SBLConfig

torch = pytest.importorskip("torch")


# bytes with FP32 intermediates alone
@pytest.mark.parametrize("grid,sample,batch,plain", [
    ((256, 256), (128, 128), 8, 783474688), ((64, 64), (32, 32), 64, 426484480),
    ((8000, 2), (4000, 2), 3, 2175752192), ((40, 32), (20, 16), 100, 249949184)])
def test_smallest_workspace_holds_no_padding(grid, sample, batch, plain):
    c = resolve_cg_config(SBLConfig(mode="cg", max_iter=6, active_set=False), grid[0] * grid[1], sample[0] * sample[1],
                          batch, False)
    shape = nat.FbmeShape(*grid, *sample)
    lib = nat.lib()
    least = lib.fbme_cg_workspace_bytes_min(ctypes.byref(shape), batch, ctypes.byref(c))
    assert least == plain <= lib.fbme_cg_workspace_bytes(ctypes.byref(shape), batch, ctypes.byref(c))
    bad = nat.FbmeShape(8, 8, 9, 8)
    assert lib.fbme_cg_workspace_bytes_min(ctypes.byref(bad), batch, ctypes.byref(c)) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("grid,sample,batch", [((64, 64), (32, 32), 2), ((40, 36), (20, 17), 3), ((130, 48), (61, 30), 1)])
def test_solve_in_the_smallest_workspace(grid, sample, batch, monkeypatch):
    from fbme_b200 import scenes
    from gpu_util import need_gpu
    from torch_sbl import sbl_2d

    need_gpu()
    ys = np.stack([scenes.point_scene(grid, sample, 12, 20.0, 5 + i, "rayleigh").y for i in range(batch)])
    y = torch.from_numpy(ys).cuda()
    cfg = SBLConfig(mode="cg", max_iter=4, active_set=False, hutchinson_probes=5, initial_hutchinson_probes=5,
                    max_hutchinson_probes=5, auto_probe_scaling=False)
    full = sbl_2d(y, grid, config=cfg)
    empty, refused = torch.empty, []

    def short_of_memory(*args, **kw):
        if kw.get("dtype") == torch.uint8 and not refused:
            refused.append(args)
            raise torch.OutOfMemoryError("no room for the padding")
        return empty(*args, **kw)

    monkeypatch.setattr(torch, "empty", short_of_memory)
    least = sbl_2d(y, grid, config=cfg)
    assert refused
    for f in ("x", "posterior_variance", "precision", "noise_variance"):
        assert torch.equal(getattr(full, f), getattr(least, f)), f
