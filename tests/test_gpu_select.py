"""sx_select_top against a sort: the value that a fraction of the values above epsilon reaches, exactly."""

import numpy as np
import pytest
import torch

from subsetix_b200 import _core

pytestmark = pytest.mark.gpu


def _expected(v, eps, frac):
    above = np.sort(v[v > np.float32(eps)])
    if above.size == 0:
        return None, 0
    count = max(1, min(above.size, int(np.ceil(above.size * frac))))
    return above[above.size - count], above.size


def _fields():
    rng = np.random.default_rng(5)
    yield np.zeros(1, np.float32)
    yield np.array([0.5], np.float32)
    yield np.full(5000, 0.25, np.float32)
    for n in (15, 16, 17, 4095, 4097, 300_001):
        yield rng.standard_normal(n).astype(np.float32)
        yield np.exp(30 * rng.standard_normal(n)).astype(np.float32)  # every leading bit pattern, subnormals too
    yield np.round(rng.standard_normal(100_000) * 4).astype(np.float32)  # few values, many ties
    x = rng.random(50_000).astype(np.float32)
    x[::7], x[::11], x[::13] = np.nan, np.inf, -np.inf
    yield x
    base = np.float32(1.0).view(np.int32)
    yield (base + rng.integers(0, 3000, 70_000).astype(np.int32)).view(np.float32)  # differ in the last bits only


@pytest.mark.parametrize("shift", [0, 1])  # 1: not 16-byte aligned
@pytest.mark.parametrize("eps", [1e-8, 0.0, -0.5, 10.0])
def test_select_equals_a_sort(cuda_device, shift, eps):
    for v in _fields():
        d = torch.as_tensor(np.concatenate([np.zeros(shift, np.float32), v]), device=cuda_device)[shift:]
        for frac in (1e-9, 0.1, 1.0 / 3.0, 0.5, 1.0):
            want, m = _expected(v, eps, frac)
            got, above = _core.select_top(d, float(np.float32(eps)), frac, cuda_device)
            assert above == m
            if m:
                assert got == want, (v.size, frac)
