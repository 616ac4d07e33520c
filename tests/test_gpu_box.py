"""Box sweeps (dilate, clip, ghost zones, erode, grading in one launch) against the oracle's chains, exactly.

Row counts around the tile heights, dense and sparse row lists, rows outside the
domain, columns on both sides of it, touching intervals, whole and empty rows,
every halo, rows longer than a staged slice, and input outside the contract
(which takes the general path).
"""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from subsetix_b200.subsetix_amr2.regrid import enforce_two_level_grading_set
from subsetix_b200.subsetix_cupy import morphology as M
from tests.gpu_util import assert_same, dev_set, iset, rand_set

pytestmark = pytest.mark.gpu


def _dense(h):
    """The same set with the marker of consecutive rows, as build_interval_set(rows=None) sets it."""
    s = dev_set(h)
    if np.array_equal(h[3], np.arange(h[3].size)):
        object.__setattr__(s, "_dense_rows", int(h[3].size))
    return s


def _check(h, hx, hy, W, H):
    s, o = _dense(h), iset(h)
    assert_same(M.dilate_interval_set(s, hx, hy), O.dilate(o, hx, hy), "dilate")
    assert_same(M.clip_interval_set(s, width=W, height=H), O.clip(o, W, H), "clip")
    assert_same(M.ghost_zones(s, hx, hy, width=W, height=H), O.ghost_zones(o, hx, hy, width=W, height=H), "ghost")
    assert_same(M.erode_interval_set(s, hx, hy, width=W, height=H), O.erode(o, hx, hy, width=W, height=H), "erode")
    if hy:
        for mode in ("von_neumann", "moore"):
            assert_same(enforce_two_level_grading_set(s, padding=hy, mode=mode, width=W, height=H),
                        O.grading(o, hy, mode, width=W, height=H), mode)


@pytest.mark.parametrize("rows", [1, 2, 31, 33, 129])
@pytest.mark.parametrize("mean", [0.4, 5.0, 60.0])
@pytest.mark.parametrize("hx,hy", [(0, 0), (1, 1), (0, 2), (3, 3), (7, 4), (2, 0), (1, 6)])
def test_box_operations(cuda_device, rows, mean, hx, hy):
    for stride, row0 in ((1, 0), (3, -4)):
        h = rand_set(rows, mean, seed=rows + 10 * hy, row_stride=stride, row0=row0, touching=True,
                     min_per_row=1 if mean < 1 and rows < 3 else 0)
        top = int(h[1].max()) if h[1].size else 4
        for W, H in ((max(1, top // 2), rows + 2), (top + 9, max(1, rows - 1))):
            _check(h, hx, hy, W, H)


def _rows(lists):
    counts = [len(b) for b, _ in lists]
    off = np.zeros(len(lists) + 1, np.int64)
    np.cumsum(counts, out=off[1:])
    cat = lambda k: np.concatenate([np.asarray(r[k], np.int32) for r in lists]).astype(np.int32)  # noqa: E731
    return cat(0), cat(1), off.astype(np.int32), np.arange(len(lists), dtype=np.int32)


def test_whole_touching_and_outside_rows(cuda_device):
    W = 20
    lists = [([0], [W]), ([-5], [30]), ([0, 4, 9], [4, 9, W]), ([-9, -6], [-7, -6 + 1]), ([25, 28], [26, 30]),
             ([], []), ([0, 19], [1, 20]), ([-3, 2, 19], [1, 19, 25]), ([5], [6]), ([0, 1], [1, 2])]
    for hx, hy in [(0, 0), (1, 0), (0, 1), (1, 1), (2, 2), (5, 1), (30, 4)]:
        _check(_rows(lists), hx, hy, W, len(lists))
        _check(_rows(lists[:3] * 12), hx, hy, W, 36)


@pytest.mark.parametrize("rows,long_row", [(3, 20000), (400, 9000)])
def test_rows_longer_than_a_slice(cuda_device, rows, long_row):
    lists = [(np.arange(long_row if r == rows // 2 else 3) * 6,) for r in range(rows)]
    _check(_rows([(b, b + 2 + b % 4) for (b,) in lists]), 1, 2, 6 * long_row, rows)


def test_sparse_rows_take_the_alignment(cuda_device):
    h = rand_set(40, 6.0, seed=3, row_stride=1000, row0=-7)
    s = dev_set(h)
    assert M._box_dilate(s, 1, 2) is None
    assert_same(M.dilate_interval_set(s, 1, 2), O.dilate(iset(h), 1, 2))


@pytest.mark.parametrize("lists", [
    [([0, 5, 3], [2, 6, 9])], [([0, 2, 4], [9, 3, 5])], [([3, 6], [3, 9])],
    [([1], [4]), ([2, 1], [3, 9]), ([5], [6])],
])
def test_outside_the_contract(cuda_device, lists):
    h = _rows(lists)
    s = _dense(h)
    assert M._box_sweep(s, 1, 1, 1, y_base=0, out_rows=4, x_lo=0, x_hi=12) is None
    assert_same(M.dilate_interval_set(s, 1, 1), O.dilate(iset(h), 1, 1))
    assert_same(M.clip_interval_set(s, width=12, height=4), O.clip(iset(h), 12, 4))
    assert_same(M.erode_interval_set(s, 1, 1, width=12, height=4), O.erode(iset(h), 1, 1, width=12, height=4))


def test_coordinates_next_to_the_int32_limits(cuda_device):
    """Widening past int32 is reported; clipping there is exact."""
    lo, hi = -(1 << 31), (1 << 31) - 1
    h = (np.array([lo, hi - 9], np.int32), np.array([lo + 4, hi], np.int32), np.array([0, 2], np.int32),
         np.array([0], np.int32))
    s = dev_set(h)
    assert M._box_dilate(s, 1, 1) is None
    assert_same(M.dilate_interval_set(s, 0, 1), O.dilate(iset(h), 0, 1))
    got = M.clip_interval_set(s, width=hi, height=1)
    assert got.begin.tolist() == [hi - 9] and got.end.tolist() == [hi]
