"""Composite levels whose covered cells lie in short runs, or not in runs at all: block means by runs and by cells agree."""

import numpy as np
import pytest
import torch

from subsetix_b200 import adjoint
from subsetix_b200.subsetix_cupy import full_interval_set
from subsetix_b200.subsetix_cupy.expressions import IntervalSet
from tests.gpu_util import dev_set

pytestmark = pytest.mark.gpu


def _patches(n, size, apart):
    """Squares of ``size`` cells, ``apart`` cells from one to the next, inside an n x n grid, refined by 2."""
    at = np.arange(2, n - size - 2, apart)
    rows = np.concatenate([2 * y + np.arange(2 * size) for y in at])
    b = np.tile(2 * at, rows.size)
    return (b.astype(np.int32), (b + 2 * size).astype(np.int32),
            (at.size * np.arange(rows.size + 1)).astype(np.int32), rows.astype(np.int32))


def _run(H):
    gen = torch.Generator(device="cuda").manual_seed(2)
    vel = torch.tensor([0.5, -0.7], dtype=torch.float64, device="cuda", requires_grad=True)
    u = [torch.rand(n, dtype=torch.float64, device="cuda", generator=gen).requires_grad_() for n in H.inner_cells]
    out = adjoint.advect_composite(vel, H, u, dt=1e-3, steps=6, checkpoint_every=3)
    return [*out, *torch.autograd.grad(sum(x.square().sum() for x in out), [vel, *u])]


@pytest.mark.parametrize("size,apart", [(1, 5), (3, 8), (11, 16), (13, 20)])
def test_both_forms_agree(cuda_device, monkeypatch, size, apart):
    n = 96
    sets = [full_interval_set(n, n), dev_set(_patches(n, size, apart))]
    by_runs = adjoint.Hierarchy(sets, n, n)
    assert by_runs.cover[1][1] is None  # few runs
    monkeypatch.setattr(adjoint, "_FEW_RUNS", 0)
    H = adjoint.Hierarchy(sets, n, n)
    assert (H.cover[1][0] is None) == (size < 12)
    for x, y in zip(_run(by_runs), _run(H)):
        assert torch.equal(x, y)


def test_overlapping_rows_of_the_coarse_level(cuda_device):
    """A coarse row as [0, 14) and [10, 24): cells side by side whose values lie apart."""
    n = 24
    b = np.tile(np.array([0, 10], np.int32), n)
    coarse = IntervalSet(*(torch.as_tensor(np.asarray(a, np.int32), device="cuda") for a in
                           (b, b + 14, 2 * np.arange(n + 1), np.arange(n))))
    H = adjoint.Hierarchy([coarse, dev_set(_patches(n, 15, 40))], n, n)  # one patch, cells 2 to 16
    u = H.extend([torch.rand(28 * n, dtype=torch.float64, device="cuda"),
                  torch.rand(30 * 30, dtype=torch.float64, device="cuda")])
    want, inner = u[0].clone(), H.interior(u)[1]
    y, x = (t.reshape(-1).to(torch.int32) for t in torch.meshgrid(*2 * [torch.arange(2, 17, device="cuda")], indexing="ij"))
    at = adjoint._positions(coarse, H.levels[0].cell_off, y, x).long()
    block = inner.view(15, 2, 15, 2)
    want[at] = ((block[:, 0, :, 0] + block[:, 0, :, 1] + block[:, 1, :, 0] + block[:, 1, :, 1]) * 0.25).reshape(-1)
    H._restrict(u)
    assert torch.equal(u[0], want)
