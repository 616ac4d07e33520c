"""Row-lane tiles that exceed their slice or span more than 65534 columns, and skewed rows, against dense or oracle results.

Such tiles are swept in groups of rows, twice (count, then write); rows that
do not fit a slice alone and groups too wide for 16 bits over 32-bit
coordinates; and once a row holds twice its share of a group's intervals the
lanes go to the rows in proportion.  Results are whole numbers and must be
equal, whatever the split.
"""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from subsetix_b200 import _core, _lib
from tests.test_gpu_rowlane import _random_table, _rows, _table_eval

pytestmark = pytest.mark.gpu


def _skewed(rng, rows, heavy, x_scale=1):
    """Rows of 0 to 6 intervals; every seventh of ``heavy`` (0 = none)."""
    begins, ends, off = [], [], [0]
    for r in range(rows):
        n = heavy if heavy and r % 7 == 3 else int(rng.integers(0, 7))
        x = int(rng.integers(-50, 50)) * x_scale
        for _ in range(n):
            x += int(rng.integers(1, 6)) * x_scale
            begins.append(x)
            x += int(rng.integers(1, 9)) * x_scale
            ends.append(x)
        off.append(len(begins))
    return [np.asarray(a, np.int32) for a in (begins, ends, off)]


@pytest.mark.parametrize("k", [1, 2, 5, 6, 8])
@pytest.mark.parametrize("heavy,x_scale", [(0, 1), (40, 1), (400, 1), (3000, 1), (40, 9000), (400, 9000)])
def test_groups_equal_the_segmented_sweep(cuda_device, k, heavy, x_scale):
    rng = np.random.default_rng(1000 * k + heavy + x_scale)
    rows = 77  # partial last tiles
    leaves = [_skewed(rng, rows, heavy, x_scale) for _ in range(k)]
    words, _ = _random_table(rng, k)
    want = _table_eval(leaves, rows, words, {"kernel": 1}, cuda_device)
    assert want[3] == 0
    even = _core.even_tuning([tuple(torch.as_tensor(a) for a in leaf) + (0,) for leaf in leaves], rows)
    for tuning in ({}, even, {"kernel": 7, "tile_rows": 8, "staging_cap": 2, "warps": 1},
                   {"kernel": 7, "tile_rows": 16, "staging_cap": 100, "warps": 4},
                   {"kernel": 7, "tile_rows": 32, "staging_cap": 900, "warps": 2},
                   {"kernel": 7, "tile_rows": 32, "staging_cap": 25000, "warps": 2}):
        got = _table_eval(leaves, rows, words, tuning, cuda_device)
        assert got[3] == 0, tuning
        for g, w in zip(got[:3], want[:3]):
            np.testing.assert_array_equal(g, w, str(tuning))


@pytest.mark.parametrize("x_scale", [1, 9000])
def test_skewed_rows_against_the_oracle(cuda_device, x_scale):
    rng = np.random.default_rng(11)
    rows = 77
    a, b = _skewed(rng, rows, 900, x_scale), _skewed(rng, rows, 500, x_scale)
    ids = np.arange(rows, dtype=np.int32)
    want = O.symmetric_difference(O.ISet(a[0], a[1], a[2], ids), O.ISet(b[0], b[1], b[2], ids))
    for cap in (2, 300, 4000):
        got = _table_eval([a, b], rows, [0b0110] + [0] * 7,
                          {"kernel": 7, "tile_rows": 16, "staging_cap": cap, "warps": 2}, cuda_device)
        assert got[3] == 0
        np.testing.assert_array_equal(got[0], want.begin)
        np.testing.assert_array_equal(got[1], want.end)
        np.testing.assert_array_equal(got[2], want.row_offsets)


@pytest.mark.parametrize("heavy,x_scale,cap,long_tile", [
    (0, 1, 600, False), (40, 1, 600, False), (3000, 1, 600, True),  # rows that no slice holds
    (0, 9000, 600, False),  # wide, at most 192 intervals per tile: swept in place
    (40, 9000, 600, True), (150, 9000, 2400, True)])  # wide, about 270 and 770
def test_the_even_sweep_gives_up_on_long_rows_and_wide_tiles(cuda_device, heavy, x_scale, cap, long_tile):
    rng = np.random.default_rng(13)
    rows = 3000
    leaves = [tuple(torch.as_tensor(a, device=cuda_device) for a in _skewed(rng, rows, heavy, x_scale)) + (0,)
              for _ in range(2)]
    tuning = dict(_core.even_tuning(leaves, rows), staging_cap=cap, tile_rows=16)
    _, _, _, result = _core.bool_eval_async(leaves, rows, [0b0110] + [0] * 7, _lib.MODE_TABLE, cuda_device,
                                            tuning=tuning, even=True)
    assert int(result[1]) == (_lib.FLAG_LONG_TILE if long_tile else 0)


def test_the_even_sweep_wants_a_row_lane_tuning(cuda_device):
    leaf = tuple(torch.as_tensor(a, device=cuda_device) for a in _rows(np.random.default_rng(1), 40, 2.0)) + (0,)
    with pytest.raises(ValueError, match="kernel 7"):
        _core.bool_eval_async([leaf], 40, [0b10] + [0] * 7, _lib.MODE_TABLE, cuda_device, tuning={"kernel": 5},
                              even=True)


def test_broken_rows_in_groups_are_flagged(cuda_device):
    rng = np.random.default_rng(12)
    rows = 40
    for x_scale in (1, 9000):
        b, e, off = (a.copy() for a in _skewed(rng, rows, 200, x_scale))
        j = int(off[3]) + 100  # inside the heavy row of the first tile
        b[j] = e[j - 1]  # touches its neighbour
        for cap in (2, 100, 4000):
            got = _table_eval([(b, e, off), tuple(_rows(rng, rows, 3.0))], rows, [0b1110] + [0] * 7,
                              {"kernel": 7, "tile_rows": 16, "staging_cap": cap, "warps": 2}, cuda_device)
            assert got[3] != 0
