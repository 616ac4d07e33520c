"""Field transfers over sets whose rows are many and short, few and long, or out of order, against a plain restatement.

Groups of several rows (from 5921 rows on), rows of more intervals than a
batch shared by several blocks, shares that end inside intervals, and rows
whose begins fall, so that a fine interval is wider or narrower than its
coarse one and the values past a coarse interval are read.
"""

import numpy as np
import pytest
import torch

from subsetix_b200 import _core
from subsetix_b200.subsetix_cupy.multilevel import prolong_set
from tests.gpu_util import dev_set, host

pytestmark = pytest.mark.gpu


def _set(rng, counts, most, falling=False):
    """``counts[y]`` intervals of 1 to ``most`` cells in row y; ``falling``: some rows backwards."""
    off = np.concatenate([[0], np.cumsum(counts)])
    length = rng.integers(1, most + 1, off[-1])
    x = np.cumsum(length + rng.integers(1, 4, off[-1])) - length
    x -= np.repeat(x[np.minimum(off[:-1], max(off[-1] - 1, 0))], counts)
    b, e = x, x + length
    if falling:
        for y in range(0, len(counts), 3):
            b[off[y]:off[y + 1]], e[off[y]:off[y + 1]] = b[off[y]:off[y + 1]][::-1].copy(), e[off[y]:off[y + 1]][::-1].copy()
    return b.astype(np.int32), e.astype(np.int32), off.astype(np.int32), np.arange(len(counts), dtype=np.int32)


GEOMETRIES = {
    "short rows": lambda rng: _set(rng, rng.integers(1, 4, 7000), 3),
    "one cell per row": lambda rng: _set(rng, np.ones(6000, np.int64), 1),
    "one long row": lambda rng: _set(rng, [7000], 3),
    "long rows": lambda rng: _set(rng, [1, 1500, 2, 900], 40),
    "one interval": lambda rng: (np.array([4], np.int32), np.array([9004], np.int32),
                                 np.array([0, 1], np.int32), np.array([2], np.int32)),
    "falling": lambda rng: _set(rng, rng.integers(1, 30, 200), 9, falling=True),
}


@pytest.mark.parametrize("name", list(GEOMETRIES))
@pytest.mark.parametrize("ratio", [2, 3, 5, 9])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_transfers(cuda_device, name, ratio, dtype):
    _transfers(cuda_device, GEOMETRIES[name], ratio, dtype, name == "falling")


def test_large_ratio(cuda_device):
    _transfers(cuda_device, lambda rng: _set(rng, [40, 1, 700], 5), 37, torch.float32, False)


def _transfers(cuda_device, geometry, ratio, dtype, falling):
    rng = np.random.default_rng(8)
    h = geometry(rng)
    s = dev_set(h)
    fine = prolong_set(s, ratio)
    f_off, f_rows = host(fine)[2], host(fine)[3]
    assert len(f_rows) == ratio * len(h[3])
    c_off, cells = _core.cell_offsets(s.begin, s.end, cuda_device)
    ff_off, f_cells = _core.cell_offsets(fine.begin, fine.end, cuda_device)
    co, fo = c_off.cpu().numpy().astype(np.int64), ff_off.cpu().numpy().astype(np.int64)
    cv = torch.rand(cells, device=cuda_device, dtype=dtype)
    got = torch.full((f_cells,), -1.0, device=cuda_device, dtype=dtype)
    _core.prolong_field(s.row_offsets, c_off, len(h[0]), fine.row_offsets, ff_off, ratio, cv, got, cuda_device)
    # interval i (number o in row p) goes to interval o of each sub-row, fine cell t from its cell t / ratio
    rows = np.repeat(np.arange(len(h[3])), np.diff(h[2]))
    nth = np.arange(len(h[0])) - h[2][rows]
    f = (f_off[(rows[:, None] * ratio + np.arange(ratio)[None, :])] + nth[:, None]).reshape(-1)
    width = fo[f + 1] - fo[f]
    t = np.arange(width.sum()) - np.repeat(np.cumsum(width) - width, width)
    src = np.repeat(np.repeat(co[:-1], ratio), width) + t // ratio
    at = np.repeat(fo[f], width) + t
    want = np.full(f_cells, -1.0)
    want[at] = np.where(src < cells, cv.cpu().numpy()[np.minimum(src, cells - 1)], 0.0)
    np.testing.assert_array_equal(got.cpu().numpy().astype(np.float64), want)
    if falling:
        return
    # restriction by the largest value (exact in any order), and the sum of whole numbers
    fv = torch.randint(0, 8, (f_cells,), device=cuda_device).to(dtype)
    cell = np.repeat(np.repeat(co[:-1], ratio), width) + t // ratio
    for reducer, reduce in ((3, np.maximum), (1, np.add)):
        out = torch.full((cells,), -1.0, device=cuda_device, dtype=dtype)
        _core.restrict_field(s.row_offsets, c_off, len(h[0]), fine.row_offsets, ff_off, ratio, reducer, fv, out,
                             cuda_device)
        want = np.zeros(cells)
        reduce.at(want, cell, fv.cpu().numpy()[at])
        np.testing.assert_array_equal(out.cpu().numpy().astype(np.float64), want)
