"""Rows that the sweep for even rows gives up on: what it has counted by then, and the launch that follows."""

import numpy as np
import pytest
import torch

from subsetix_b200 import _core, _lib
from tests.test_gpu_rowlane import _random_table, _table_eval
from tests.test_gpu_rowlane_groups import _skewed

pytestmark = pytest.mark.gpu


def _eval(leaves, rows, words, dev, monkeypatch):
    """``_core.bool_eval`` and the arguments and result of ``_uneven_tuning`` if it was called."""
    seen = []
    choose = _core._uneven_tuning

    def record(*args):
        seen.append((args[3:], choose(*args)))
        return seen[-1][1]

    monkeypatch.setattr(_core, "_uneven_tuning", record)
    monkeypatch.setattr(_core, "TUNED", {})
    ops = [tuple(torch.as_tensor(a, device=dev) for a in leaf) + (0,) for leaf in leaves]
    b, e, off, total, flags = _core.bool_eval(ops, rows, words, _lib.MODE_TABLE, dev)
    return (b[:total].cpu().numpy(), e[:total].cpu().numpy(), off.cpu().numpy(), flags), seen


def _most(leaves, rows, n):
    counts = sum(np.diff(leaf[2].astype(np.int64)) for leaf in leaves)
    counts = np.concatenate([counts, np.zeros(-rows % 32, np.int64)])
    return counts.reshape(-1, n).sum(1)


@pytest.mark.parametrize("k", [1, 2, 5, 8])
@pytest.mark.parametrize("rows", [5, 40, 3001])
@pytest.mark.parametrize("heavy,x_scale,kernel", [(60, 9000, 5), (4000, 1, 4), (4000, 900, 4)])
def test_second_launch(cuda_device, monkeypatch, k, rows, heavy, x_scale, kernel):
    rng = np.random.default_rng(k + rows + heavy)
    if kernel == 5:  # every row alike, and too wide for 16 bits
        leaves = []
        for _ in range(k):
            steps = rng.integers(1, 9, (rows, 2 * heavy)).cumsum(1) * x_scale
            leaves.append([steps[:, 0::2].ravel().astype(np.int32), steps[:, 1::2].ravel().astype(np.int32),
                           (heavy * np.arange(rows + 1)).astype(np.int32)])
    else:
        leaves = [_skewed(rng, rows, 0, x_scale) for _ in range(k)]
        row = rows // 2  # one row of every leaf that no slice holds
        for i, (b, e, off) in enumerate(leaves):
            x = (np.arange(2 * heavy) * 3 + i).astype(np.int64) * x_scale
            at, to = int(off[row]), int(off[row + 1])
            shift = np.where(np.arange(rows + 1) > row, heavy - (to - at), 0)
            leaves[i] = [np.concatenate([b[:at], x[0::2], b[to:]]).astype(np.int32),
                         np.concatenate([e[:at], x[1::2], e[to:]]).astype(np.int32), (off + shift).astype(np.int32)]
    words, _ = _random_table(rng, k)
    want = _table_eval(leaves, rows, words, {"kernel": 1}, cuda_device)
    got, seen = _eval(leaves, rows, words, cuda_device, monkeypatch)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
    for (even, most8, most32, wide), tuning in seen:
        assert most8 == _most(leaves, rows, 8).max()
        assert most32 in _most(leaves, rows, 32)
        assert tuning["kernel"] == kernel or (kernel == 4 and rows <= 40 and tuning["kernel"] in (5, 7))
        assert 2 * most32 <= tuning["staging_cap"] or tuning["kernel"] != 4 or tuning["staging_cap"] == 25000
        assert bool(wide) or kernel == 4
    if rows == 3001 and (kernel == 4 or k > 1):
        assert len(seen) == 1
