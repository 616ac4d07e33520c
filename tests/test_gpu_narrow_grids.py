"""Threshold runs and gradients of narrow grids: both sides of the lines where the kernels change, against dense masks."""

import numpy as np
import pytest
import torch

from subsetix_b200 import _core, _lib
from subsetix_b200._runtime import ptr, stream_handle
from tests.test_gpu_rle import _two_pass

pytestmark = pytest.mark.gpu


def _grid(width, height, device):
    g = torch.Generator(device=device).manual_seed(width)
    return torch.rand(height * width, device=device, generator=g)


def _dense(b, e, off, width, height):
    mask = np.zeros((height, width + 1), np.int64)
    rows = np.repeat(np.arange(height), np.diff(off.cpu().numpy()))
    np.add.at(mask, (rows, b.cpu().numpy()), 1)
    np.add.at(mask, (rows, e.cpu().numpy()), -1)
    return np.cumsum(mask, 1)[:, :width]


@pytest.mark.parametrize("width", [1, 3, 32, 128, 129])
@pytest.mark.parametrize("height", [10000, 10001])
@pytest.mark.parametrize("gradient", [False, True])
def test_threshold_runs(cuda_device, width, height, gradient):
    v = _grid(width, height, cuda_device)
    got = _core.threshold_rle(v, width, height, 0.4, gradient, cuda_device)
    for x, y in zip(got, _two_pass(v, width, height, 0.4, int(gradient), cuda_device)):
        assert torch.equal(x, y)
    if not gradient:
        want = (v >= 0.4).cpu().numpy().reshape(height, width)
        np.testing.assert_array_equal(_dense(*got, width, height), want)


@pytest.mark.parametrize("width", [1, 2, 3, 47, 48, 49])
@pytest.mark.parametrize("height", [1, 2, 500])
def test_gradient_magnitude(cuda_device, width, height):
    v = _grid(width, height, cuda_device)
    out = torch.full((width * height + 3,), -1.0, device=cuda_device)
    _lib.check(_lib.load().sx_gradient_magnitude(ptr(v), width, height, ptr(out), stream_handle(cuda_device)), "gradient")
    assert bool((out[-3:] == -1.0).all())
    for thr in (0.05, 0.2, 0.5):
        want = _dense(*_two_pass(v, width, height, thr, 1, cuda_device), width, height)
        np.testing.assert_array_equal((out[:-3] >= thr).cpu().numpy().reshape(height, width), want)
