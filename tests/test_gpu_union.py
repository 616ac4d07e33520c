"""The union sweep (dilation, restriction) where its tiles and pieces can go wrong.

Row counts around the tile heights, rows from empty to longer than a staged
slice, every number of lanes per row, leaves with their own arrays, and input
outside the contract; outputs are integers and compared exactly with the
oracle.
"""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from subsetix_b200 import _core, _lib
from tests.gpu_util import assert_same, dev_set, iset, rand_set

pytestmark = pytest.mark.gpu

sc = pytest.importorskip("subsetix_b200.subsetix_cupy")


@pytest.mark.parametrize("rows", [1, 2, 7, 31, 33, 257])
@pytest.mark.parametrize("mean", [0.3, 3.0, 90.0])
@pytest.mark.parametrize("hx,hy", [(0, 1), (3, 4), (40, 2)])
def test_dilate_tile_edges(cuda_device, rows, mean, hx, hy):
    h = rand_set(rows, mean, seed=rows + hy, row_stride=2 if hx else 1, touching=True, min_per_row=1 if rows == 1 else 0)
    assert_same(sc.dilate_interval_set(dev_set(h), halo_x=hx, halo_y=hy), O.dilate(iset(h), hx, hy))


@pytest.mark.parametrize("rows,long_row", [(3, 30000), (200, 20000), (5000, 9000)])
def test_dilate_rows_longer_than_a_slice(cuda_device, rows, long_row):
    """One row holds most intervals: its tiles exceed the staged slice and run on global memory."""
    counts = np.full(rows, 2)
    counts[rows // 2] = long_row
    off = np.zeros(rows + 1, np.int64)
    np.cumsum(counts, out=off[1:])
    b = np.concatenate([np.arange(c) * 5 for c in counts])
    h = (b.astype(np.int32), (b + 1 + b % 3).astype(np.int32), off.astype(np.int32), np.arange(rows, dtype=np.int32))
    assert_same(sc.dilate_interval_set(dev_set(h), halo_x=1, halo_y=1), O.dilate(iset(h), 1, 1))
    assert_same(sc.restrict_set(dev_set(h), 3), O.restrict_set(iset(h), 3))


@pytest.mark.parametrize("k", [2, 5, 9])
def test_leaves_with_their_own_arrays(cuda_device, k):
    hs = [rand_set(150, 2.0 + l, seed=l, row_stride=1, touching=True) for l in range(k)]
    specs = []
    for l, h in enumerate(hs):
        b, e, off, _ = (torch.as_tensor(a, device=cuda_device) for a in h)
        specs.append((b, e, off, l % 3))
    ob, oe, off, total, flags = _core.bool_eval(specs, 150, [0] * 8, _lib.MODE_UNION, cuda_device)
    assert flags == 0
    rows = np.concatenate([np.repeat(np.arange(150), np.diff(h[2])) for h in hs])
    begin = np.concatenate([h[0] - l % 3 for l, h in enumerate(hs)])
    end = np.concatenate([h[1] + l % 3 for l, h in enumerate(hs)])
    exp = O.build_from_rows(rows.astype(np.int32), begin.astype(np.int32), end.astype(np.int32))
    np.testing.assert_array_equal(ob[:total].cpu().numpy(), exp.begin)
    np.testing.assert_array_equal(oe[:total].cpu().numpy(), exp.end)
    got = np.diff(off.cpu().numpy())
    np.testing.assert_array_equal(got[got > 0], np.diff(exp.row_offsets))


@pytest.mark.parametrize("begin,end", [([0, 5, 3], [2, 6, 9]), ([0, 2, 4], [9, 3, 5]), ([0, 4, 8], [1, 4, 9])])
def test_rows_outside_the_contract_are_reported(cuda_device, begin, end):
    """Begins that fall, ends that fall, an empty interval: reported, and the reference's order runs instead."""
    n = 64
    b = np.concatenate([np.arange(n) * 10 - 1000, begin]).astype(np.int32)
    e = np.concatenate([np.arange(n) * 10 - 995, end]).astype(np.int32)
    t = [torch.as_tensor(x, device=cuda_device) for x in (b, e, np.array([0, n + 3], np.int32))]
    *_, flags = _core.bool_eval([(t[0], t[1], t[2], 0)], 1, [0] * 8, _lib.MODE_UNION, cuda_device)
    assert flags & _lib.FLAG_CONTRACT
    h = (b, e, np.array([0, n + 3], np.int32), np.array([4], np.int32))
    assert_same(sc.dilate_interval_set(dev_set(h), halo_x=0, halo_y=1), O.dilate(iset(h), 0, 1))
