"""The merge of the slices' candidate lists: one list, a ragged last list, the
most lists (2048 candidates), the whole answer in one list, answers spread
evenly over the lists, and equal scores everywhere.  Exact: the result is the
first k of a stable descending sort."""
import numpy as np
import pytest
import torch

from gpu_util import need_gpu
from test_gpu_topk import topk_native

SLICE = 8192


@pytest.mark.gpu
@pytest.mark.parametrize("slices,tail,k", [(1, 0, 32), (2, 5, 1), (3, 40, 32), (31, 1, 32), (33, 0, 31), (64, 0, 32)])
@pytest.mark.parametrize("kind", ["random", "one_list", "even", "equal"])
def test_topk_merge_lists(slices, tail, k, kind):
    need_gpu()
    n = slices * SLICE - (SLICE - tail if tail else 0)
    rng = np.random.default_rng(n + k)
    s = rng.random((2, n)).astype(np.float32)
    if kind == "one_list":
        s[:, (slices // 2) * SLICE:(slices // 2) * SLICE + k] += 2.0
    elif kind == "even":  # equal scores at the same place of every slice
        for p in range(k):
            s[:, 17 * p::SLICE] = 2.0 - 0.01 * (p // 3)
    elif kind == "equal":
        s[:] = 0.25
    idx, val = topk_native(torch.from_numpy(s).cuda(), k)
    for b in range(2):
        order = np.argsort(-s[b], kind="stable")[:k]
        assert idx[b].cpu().numpy().tolist() == order.tolist()
        assert (val[b].cpu().numpy() == s[b][order]).all()
