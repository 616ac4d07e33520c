"""Block means over runs of coarse cells and their transpose against the index-table kernels, bit for bit.

Runs of 1 to 64 cells, sub-rows that start at odd and even values, ratios 2 and
3, arrays aligned to a pair and not, and segments longer than one batch of loads.
"""

import numpy as np
import pytest
import torch

from subsetix_b200 import _lib
from subsetix_b200._runtime import ptr, stream_handle

pytestmark = pytest.mark.gpu


def _call(name, *args):
    _lib.check(getattr(_lib.load(), name)(*args, stream_handle(torch.device("cuda", 0))), name)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("ratio", [2, 3])
@pytest.mark.parametrize("shift", [0, 1])
def test_run_block_mean_equals_index_tables(cuda_device, dtype, ratio, shift):
    rng = np.random.default_rng(ratio)
    counts = [1, 2, 31, 32, 33, 63, 64, 64, 5]
    stride = (2 + ratio + 3) // 4 * 4
    plan = np.zeros((len(counts), stride), np.int32)
    cpos, child, c0, f0 = [], [], 3, 0
    for k, n in enumerate(counts):
        plan[k, :2] = c0, n
        rows = []
        for dy in range(ratio):
            f0 += int(rng.integers(0, 3))  # odd and even starts
            plan[k, 2 + dy] = f0
            rows.append(f0 + np.arange(n * ratio).reshape(n, ratio))
            f0 += n * ratio
        cpos.append(c0 + np.arange(n))
        child.append(np.concatenate(rows, axis=1))
        c0 += n + int(rng.integers(0, 2))
    code = _lib.SX_F64 if dtype == torch.float64 else _lib.SX_F32
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.int32), device=cuda_device)  # noqa: E731
    plan, cpos, child = dev(plan), dev(np.concatenate(cpos)), dev(np.concatenate(child).reshape(-1))
    fine = torch.as_tensor(rng.standard_normal(f0 + 5 + shift), device=cuda_device).to(dtype)[shift:]
    coarse = torch.as_tensor(rng.standard_normal(c0 + 5), device=cuda_device).to(dtype)
    norm, n = 1.0 / ratio ** 2, int(cpos.numel())
    got, ref = coarse.clone(), coarse.clone()
    _call("sx_run_block_mean", code, len(counts), ratio, stride, norm, ptr(plan), ptr(fine), ptr(got))
    _call("sx_index_block_mean", code, n, ratio ** 2, norm, ptr(cpos), ptr(child), ptr(fine), ptr(ref))
    assert torch.equal(got, ref)
    got_c, ref_c, ref_f = coarse.clone(), coarse.clone(), fine.clone()
    got_f = torch.cat([fine[:1], fine])[1:] if shift else fine.clone()  # the same alignment as `fine`
    _call("sx_run_block_mean_adj", code, len(counts), ratio, stride, norm, ptr(plan), ptr(got_c), ptr(got_f))
    _call("sx_index_block_mean_adj", code, n, ratio ** 2, norm, ptr(cpos), ptr(child), ptr(ref_c), ptr(ref_f))
    assert torch.equal(got_c, ref_c) and torch.equal(got_f, ref_f)


@pytest.mark.parametrize("zero", [0, 1])
def test_segment_add_in_order(cuda_device, zero):
    rng = np.random.default_rng(4)
    lens = [0, 1, 2, 3, 4, 5, 9]
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    src_idx = rng.permutation(50)[:off[-1]].astype(np.int32)
    dst_idx = rng.permutation(20)[:len(lens)].astype(np.int32)
    src, dst = rng.standard_normal(50).astype(np.float32), rng.standard_normal(20).astype(np.float32)
    t = [torch.as_tensor(a.copy(), device=cuda_device) for a in (off, src_idx, dst_idx, src, dst)]
    _call("sx_index_segment_add", _lib.SX_F32, len(lens), *(ptr(x) for x in t), zero)
    for s in range(len(lens)):
        for k in range(off[s], off[s + 1]):
            dst[dst_idx[s]] = np.float32(dst[dst_idx[s]] + src[src_idx[k]])
            if zero:
                src[src_idx[k]] = 0
    np.testing.assert_array_equal(t[4].cpu().numpy(), dst)
    np.testing.assert_array_equal(t[3].cpu().numpy(), src)
