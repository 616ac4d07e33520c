"""Row-lane sweep with a fixed number of lanes per row: a tuning whose largest tile is close to the mean one."""

import numpy as np
import pytest

from tests.test_gpu_rowlane import _random_table, _table_eval

pytestmark = pytest.mark.gpu


def _even(rng, rows, n):
    steps = rng.integers(1, 9, (rows, 2 * n)).cumsum(1) + rng.integers(-40, 40, (rows, 1))
    return [steps[:, 0::2].ravel().astype(np.int32), steps[:, 1::2].ravel().astype(np.int32),
            (n * np.arange(rows + 1)).astype(np.int32)]


@pytest.mark.parametrize("k", [1, 2, 5, 8])
@pytest.mark.parametrize("tile_rows", [8, 16, 32])
@pytest.mark.parametrize("rows,n", [(1, 9), (7, 1), (33, 20), (64, 5), (1000, 23)])
def test_even_rows(cuda_device, k, tile_rows, rows, n):
    rng = np.random.default_rng(100 * k + tile_rows + rows)
    leaves = [_even(rng, rows, n) for _ in range(k)]
    words, _ = _random_table(rng, k)
    want = _table_eval(leaves, rows, words, {"kernel": 1}, cuda_device)
    tuning = {"kernel": 7, "tile_rows": tile_rows, "staging_cap": 2 * k * n * min(tile_rows, rows), "warps": 2}
    got = _table_eval(leaves, rows, words, tuning, cuda_device)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
    b, e, off = (a.copy() for a in leaves[-1])  # an empty interval in the last row
    e[-1] = b[-1]
    assert _table_eval([*leaves[:-1], [b, e, off]], rows, words, tuning, cuda_device)[3] != 0
