"""The flat stencil and its adjoint against the generic kernels, bit for bit.

Cell counts around a group of four, intervals that start and end inside groups,
touching intervals, empty rows, every upwind side, both precisions, arrays that
are not 16-byte aligned, bands that start inside a group, and cells outside the
domain (which keep the chunked kernel).  The velocity gradient is a sum of the
same products in another order: relative 1e-12 in float64, far above the
2^-53 * log2(cells) of a pairwise sum.
"""

import numpy as np
import pytest
import torch

from subsetix_b200 import _core, _lib
from subsetix_b200._runtime import ptr, stream_handle
from tests.gpu_util import dev_set, rand_set

pytestmark = pytest.mark.gpu

adj = pytest.importorskip("subsetix_b200.adjoint")
SIDES = [(0.6, 0.3), (-0.4, -0.9), (0.6, -0.3), (-0.4, 0.9), (0.0, -0.0)]


def _geometries():
    yield (np.array([3], np.int32), np.array([4], np.int32), np.array([0, 1], np.int32), np.array([2], np.int32))
    for cells in (3, 4, 5, 127, 128, 129, 1023, 1025):  # one row of one interval
        yield (np.array([1], np.int32), np.array([1 + cells], np.int32), np.array([0, 1], np.int32),
               np.array([0], np.int32))
    yield rand_set(300, 40.0, seed=3, row_stride=1, max_col=2000, touching=True, row0=0)   # short intervals
    yield rand_set(200, 0.7, seed=4, row_stride=2, max_col=300, row0=1)                    # empty and missing rows
    b = np.zeros(70, np.int32)
    yield (b, b + 777, np.arange(71, dtype=np.int32), np.arange(70, dtype=np.int32))       # a rectangle
    # all cells single and apart, next to a full row: every group jumps
    x = np.arange(0, 1200, 3, dtype=np.int32)
    yield (np.concatenate([x, [0], x]).astype(np.int32), np.concatenate([x + 1, [1200], x + 1]).astype(np.int32),
           np.array([0, 400, 401, 801], np.int32), np.array([0, 1, 2], np.int32))


def _plan(h, dev):
    b, e, off, rows = (torch.as_tensor(np.asarray(a, np.int32), device=dev) for a in h)
    H = int(np.max(h[3])) + 2
    coff, cells = _core.cell_offsets(b, e, dev)
    lookup, bad = _core.row_lookup(rows, H, dev)
    assert not bad
    return (b, e, off, rows), H, coff, cells, lookup, _core.FlatPlan(rows, off, b, e, coff, cells, lookup, H, dev)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shift", [0, 1])  # 1: the arrays are not 16-byte aligned
def test_flat_step_equals_generic(cuda_device, dtype, shift):
    rng = np.random.default_rng(7)
    for h in _geometries():
        (b, e, off, rows), H, coff, cells, lookup, plan = _plan(h, cuda_device)
        W = plan.hi
        assert plan.covers(W) and not plan.covers(W - 1)
        v = torch.as_tensor(rng.standard_normal(cells + shift), device=cuda_device).to(dtype)[shift:]
        for a_, b_ in SIDES:
            for dx in (1e-2, 2.0 ** -7):
                ref = torch.empty_like(v)
                _core.upwind(rows, off, b, e, coff, cells, lookup, v.contiguous(), ref, W, H, a_, b_, 1e-3, dx, 1e-2,
                             False, cuda_device)
                got = torch.full((cells + shift + 4,), float("nan"), dtype=dtype, device=cuda_device)
                plan.step(v, got[shift:], a_, b_, 1e-3, dx, 1e-2, cuda_device)
                assert torch.equal(got[shift:shift + cells], ref)
                assert bool(torch.isnan(got[shift + cells:]).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_flat_adjoint_equals_generic(cuda_device, dtype):
    rng = np.random.default_rng(8)
    lib = _lib.load()
    for h in _geometries():
        W, H = int(np.max(h[1])), int(np.max(h[3])) + 2
        lvl = adj.Level(dev_set(h), W, H, 1.0 / W, 1e-2)
        assert lvl.flat is not None
        w = torch.as_tensor(rng.standard_normal(lvl.cells), device=cuda_device).to(dtype)
        u = torch.as_tensor(rng.standard_normal(lvl.cells), device=cuda_device).to(dtype)
        for a_, b_ in SIDES:
            g = torch.full((2,), 0.25, dtype=torch.float64, device=cuda_device)
            got = lvl.adjoint(w, u, a_, b_, 1e-3, g)
            ref, g_ref = torch.empty_like(w), torch.empty(2, dtype=torch.float64, device=cuda_device)
            code = _lib.SX_F64 if dtype == torch.float64 else _lib.SX_F32
            _lib.check(lib.sx_upwind_adjoint(code, ptr(lvl.rows), ptr(lvl.off), int(lvl.rows.numel()), ptr(lvl.begin),
                                             ptr(lvl.end), ptr(lvl.cell_off), int(lvl.begin.numel()), lvl.cells,
                                             ptr(lvl.lookup), ptr(w), ptr(u), ptr(ref), W, H, a_, b_, 1e-3, lvl.dx,
                                             lvl.dy, 0, ptr(g_ref), ptr(lvl.scratch), int(lvl.scratch.numel()),
                                             stream_handle(cuda_device)), "sx_upwind_adjoint")
            assert torch.equal(got, ref)
            scale = 1e-3 * float((w.double().abs().max() * u.double().abs().max())) * lvl.cells / min(lvl.dx, lvl.dy)
            assert torch.allclose(g - 0.25, g_ref, rtol=1e-12, atol=1e-12 * scale + 1e-15)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_bands_that_start_inside_groups(cuda_device, dtype):
    """Sets of 1 to 9 cells each, so bands start at every position of a group; each equals its own call."""
    from subsetix_b200.batch import SetBatch, batched_upwind
    from subsetix_b200.subsetix_cupy import build_interval_set, create_interval_field, step_upwind_interval

    sets, sides = [], []
    for k in list(range(1, 10)) * 5 + [1500, 3]:
        sets.append(build_interval_set([0, 1, 1, 2], [0, k // 2], [k, k + 1]))
        sides.append(k + 1)
    batch = SetBatch.from_sets(sets, [3] * len(sets))
    n = batch.stencil_plan().cells
    v = torch.as_tensor(np.random.default_rng(9).standard_normal(n), device=cuda_device).to(dtype)
    for a_, b_ in SIDES:
        dx = [1.0 / s for s in sides]
        dt = [0.3 * d for d in dx]
        got = batched_upwind(batch, v, width=sides, a=a_, b=b_, dt=dt, dx=dx, dy=dx)
        at = 0
        for s, d, t, side in zip(sets, dx, dt, sides):
            f = create_interval_field(s, 0.0, dtype=dtype)
            m = f.values.numel()
            f.values.copy_(v[at:at + m])
            assert torch.equal(got[at:at + m], step_upwind_interval(f, width=side, height=3, a=a_, b=b_, dt=t, dx=d,
                                                                     dy=d))
            at += m


def test_cells_outside_the_domain_keep_the_chunked_kernel(cuda_device):
    from subsetix_b200.subsetix_cupy import create_interval_field, step_upwind_interval

    h = rand_set(60, 8.0, seed=5, row_stride=1, touching=True, row0=0)  # begins at -5 and up
    f = create_interval_field(dev_set(h), 0.0, dtype=np.float32)
    f.values.copy_(torch.as_tensor(np.random.default_rng(1).standard_normal(f.values.numel()), device=cuda_device))
    kw = dict(height=61, a=0.5, b=-0.5, dt=1e-3, dx=1e-2, dy=1e-2)
    rid = torch.repeat_interleave(torch.as_tensor(h[3]), torch.as_tensor(np.diff(h[2])).long())
    for width in (70, 10 ** 6):
        got = step_upwind_interval(f, width=width, **kw)
        assert torch.equal(got, step_upwind_interval(f, width=width, row_ids=rid.to(cuda_device), **kw))
