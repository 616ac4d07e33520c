"""Index arithmetic at the top of the int32 range: the largest flat plan, the most rows of a mask, the longest tiles."""

import ctypes

import pytest
import torch

from subsetix_b200 import _core, _lib
from subsetix_b200._runtime import ptr, stream_handle

pytestmark = pytest.mark.gpu


def test_flat_plan_of_the_most_cells(cuda_device):
    n = 2 ** 31 - 1  # 2^29 groups, the last with three cells
    b, e, off, rows = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0], [n], [0, 1], [0]))
    coff, lookup = torch.tensor([0, n], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    plan = _core.FlatPlan(rows, off, b, e, coff, n, lookup, 1, cuda_device)
    assert (plan.lo, plan.hi) == (0, n) and plan.covers(n)
    flags = plan._keep[2]
    left, right = 0xF00, 1 << 14  # every cell has a left neighbour, every group's last cell a right one
    assert flags[0] == (left & ~0x100) | right and flags[-1] == (left & ~0x800)
    assert bool((flags[1:-1] == left | right).all())


def test_mask_of_the_most_rows(cuda_device):
    h = 2 ** 27 + 37  # 2^32 threads and more, one warp per row
    values = (torch.arange(h, device="cuda", dtype=torch.int32) % 3 == 1).to(torch.float32)
    lib, st = _lib.load(), stream_handle(cuda_device)
    mask, off = (torch.empty(h + i, dtype=torch.int32, device="cuda") for i in (0, 1))
    result = torch.empty(2, dtype=torch.int32, device="cuda")
    ws = torch.empty(int(lib.sx_threshold_mask_workspace_bytes(h)), dtype=torch.uint8, device="cuda")
    _lib.check(lib.sx_threshold_mask(ptr(values), 1, h, 0.5, 0, ptr(mask), ptr(off), ptr(result), ptr(ws),
                                     int(ws.numel()), st), "sx_threshold_mask")
    counts = values.to(torch.int32)
    assert torch.equal(off[1:] - off[:-1], counts)
    b, e = (torch.full((int(off[-1]),), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    _lib.check(lib.sx_mask_runs(ptr(mask), 1, h, ptr(off), ptr(b), ptr(e), st), "sx_mask_runs")
    assert result.tolist() == [int(off[-1]), 0] and bool((b == 0).all()) and bool((e == 1).all())


def test_even_sweep_gives_up_on_tiles_of_2_31_intervals(cuda_device):
    n, rows = 2 ** 28, 8
    j = torch.arange(n // rows, dtype=torch.int32, device="cuda").repeat(rows)
    b, e = 2 * j, 2 * j + 1
    del j
    off = torch.arange(rows + 1, dtype=torch.int32, device="cuda") * (n // rows)
    table, lib = (ctypes.c_uint32 * 8)(*[0] * 7, 1 << 31), _lib.load()
    leaves = (_lib.SxLeaf * 8)(*[_lib.SxLeaf(ptr(b), ptr(e), ptr(off), None, 0, 0)] * 8)
    tuning = _lib.SxTuning(*(_core.even_tuning([(b,)] * 8, rows).get(key, 0) for key, _ in _lib.SxTuning._fields_))
    out, result = (torch.empty(32, dtype=torch.int32, device="cuda") for _ in range(2))
    out_off = torch.empty(rows + 1, dtype=torch.int32, device="cuda")
    ws = torch.empty(int(lib.sx_bool_workspace_bytes(rows)), dtype=torch.uint8, device="cuda")
    _lib.check(lib.sx_bool_eval_even(leaves, 8, rows, table, ptr(out), ptr(out[16:]), ptr(out_off), 16, ptr(result),
                                     ptr(ws), int(ws.numel()), ctypes.byref(tuning), stream_handle(cuda_device)),
               "sx_bool_eval_even")
    assert result.tolist()[1] == _lib.FLAG_LONG_TILE
