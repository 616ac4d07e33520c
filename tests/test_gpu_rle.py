"""Mask-based threshold run-length encoding against the two-pass kernel and a dense mask.

Widths around a word, a strip (128), a chunk (1024) and not multiples of 4, one
row and one column, full and empty rows, NaN and infinity, unaligned fields.
"""

import ctypes

import numpy as np
import pytest
import torch

from subsetix_b200 import _core, _lib
from subsetix_b200._runtime import ptr, stream_handle

pytestmark = pytest.mark.gpu


def _two_pass(v, W, H, thr, grad, dev):
    lib, s = _lib.load(), stream_handle(dev)
    counts = torch.empty(H, dtype=torch.int32, device=dev)
    t = ctypes.c_float(thr)
    _lib.check(lib.sx_threshold_rle(ptr(v), W, H, t, grad, ptr(counts), None, None, None, s), "count")
    off, total = _core.scan(counts, dev)
    b, e = (torch.empty(total, dtype=torch.int32, device=dev) for _ in range(2))
    if total:
        _lib.check(lib.sx_threshold_rle(ptr(v), W, H, t, grad, None, ptr(off), ptr(b), ptr(e), s), "write")
    return b, e, off


@pytest.mark.parametrize("width", [1, 2, 31, 32, 33, 100, 127, 128, 129, 1023, 1024, 1028, 2050])
@pytest.mark.parametrize("height", [1, 2, 9, 65])
@pytest.mark.parametrize("grad", [0, 1])
@pytest.mark.parametrize("shift", [0, 1])
def test_mask_runs_equal_two_pass(cuda_device, width, height, grad, shift):
    rng = np.random.default_rng(width * 7 + height)
    v = rng.standard_normal((height, width)).astype(np.float32)
    v[height // 2] = 2.0  # a row set (or, by gradient, clear) from end to end
    v[0, :: 5] = np.nan
    v[-1, width // 2] = np.inf
    base = torch.empty(width * height + shift, dtype=torch.float32, device=cuda_device)
    f = base[shift:]
    f.copy_(torch.as_tensor(v.reshape(-1)))
    for thr in (-10.0, 0.0, 0.7, 50.0):
        got = _core.threshold_rle(f, width, height, thr, bool(grad), cuda_device)
        ref = _two_pass(f, width, height, thr, grad, cuda_device)
        for a, b in zip(got, ref):
            assert torch.equal(a, b)


@pytest.mark.parametrize("height", [3551, 3552, 3553, 4096])
def test_rows_per_block_both_sides(cuda_device, height):
    """Two rows per block below 3552 rows, eight from there on; the last block is partial."""
    g = torch.Generator(device=cuda_device).manual_seed(height)
    v = torch.rand(height * 140, device=cuda_device, generator=g)
    for a, b in zip(_core.threshold_rle(v, 140, height, 0.5, True, cuda_device),
                    _two_pass(v, 140, height, 0.5, 1, cuda_device)):
        assert torch.equal(a, b)
