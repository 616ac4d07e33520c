"""Prolongation and restriction of fields where a block of a coarse row can go wrong, against the oracle, exactly.

Rows around a block's share (1024 cells) and around a batch of intervals (512),
few long rows (shared by several blocks), odd and even starts, unaligned values.
"""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from subsetix_b200 import _core
from subsetix_b200.subsetix_cupy import IntervalField, prolong_field, restrict_field
from tests.gpu_util import assert_same, dev_set, iset, rand_set

pytestmark = pytest.mark.gpu


def _rows(lists, rows=None):
    off = np.zeros(len(lists) + 1, np.int64)
    np.cumsum([len(b) for b, _ in lists], out=off[1:])
    cat = lambda k: np.concatenate([np.asarray(x[k]) for x in lists]).astype(np.int32)  # noqa: E731
    return cat(0), cat(1), off.astype(np.int32), np.arange(len(lists), dtype=np.int32)


def _geometries():
    for w in (1, 2, 255, 257, 1023, 1024, 1025, 5000):
        yield _rows([([3], [3 + w])])
    for k in (511, 512, 513, 1100):  # intervals per row around a batch
        b = np.arange(k) * 7 + 1
        yield _rows([(b, b + 1 + b % 5), ([0], [40])])
    yield rand_set(400, 12.0, seed=5, row_stride=3, min_per_row=1)
    yield _rows([([0], [300000]), ([5], [9])])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ratio", [2, 3, 4, 5])
@pytest.mark.parametrize("shift", [0, 1])
def test_field_transfer_equals_oracle(cuda_device, dtype, ratio, shift):
    rng = np.random.default_rng(2)
    tdt = torch.float32 if dtype == np.float32 else torch.float64

    def dev(values):
        base = torch.empty(values.size + shift, dtype=tdt, device=cuda_device)
        base[shift:].copy_(torch.as_tensor(values))
        return base[shift:]

    for h in _geometries():
        cf = O.create_field(iset(h), 0.0, dtype)
        cf.values[...] = rng.standard_normal(cf.values.size).astype(dtype)
        s = dev_set(h)
        off, _ = _core.cell_offsets(s.begin, s.end, cuda_device)
        fine = prolong_field(IntervalField(s, dev(cf.values), off), ratio, dtype=dtype)
        ef = O.prolong_field(cf, ratio, dtype=dtype)
        assert_same(fine.interval_set, ef.iset)
        np.testing.assert_array_equal(fine.values.cpu().numpy(), ef.values)
        ef.values[...] = rng.standard_normal(ef.values.size).astype(dtype)
        noisy = IntervalField(fine.interval_set, dev(ef.values), fine.interval_cell_offsets)
        for red in ("mean", "sum", "min", "max"):
            got, exp = restrict_field(noisy, ratio, reducer=red, dtype=dtype), O.restrict_field(ef, ratio, red, dtype)
            assert_same(got.interval_set, exp.iset)
            np.testing.assert_array_equal(got.values.cpu().numpy(), exp.values)
