"""Device-level building blocks over torch tensors, each one C-ABI call.

Everything here takes and returns int32 CUDA tensors and enqueues work on
the current torch stream.  Functions whose output size depends on the data
read one small ``result`` pair back from the device.  The reference API
returns sized arrays, so it synchronises at the same points
(``subsetix_cupy/expressions.py:503``).
"""

from __future__ import annotations

import ctypes
import struct
from typing import List, Optional, Sequence, Tuple

import torch

from . import _lib
from ._runtime import ptr, read_pair, stream_handle, workspace, workspace_words

I32 = torch.int32

OP_UNION, OP_INTERSECTION, OP_DIFFERENCE = 0, 1, 2

# Launch tuning for the row sweep (sx_tuning).  TUNING, when not empty,
# applies to every evaluation.  TUNED maps a workload key (workload_key) to
# the launch shape the autotuner (subsetix_b200/autotune.py) found fastest for
# that kind of workload; buffer sizes are still taken from each evaluation's
# own largest tile.  Neither ever changes results.
TUNING: dict = {}
TUNED: dict = {}

_SM_SHARED = 228 * 1024  # shared memory of an SM; a block takes 1 KB beside its own
_TILE_INTERVALS = 1600  # a mean tile of the automatic row-lane sweep (13 KB of shared memory)


def workload_key(sizes: Sequence[int], rows: int) -> str:
    """Bucket of a set-algebra workload: leaf count, log2 rows, log2 mean boundaries per 32-row tile."""
    import math

    tiles = max(1, (int(rows) + 31) // 32)
    per_tile = 2 * sum(int(s) for s in sizes) / tiles
    return f"k{len(sizes)}-r{int(math.log2(max(rows, 1)))}-t{int(math.log2(max(per_tile, 1.0)))}"


def empty_i32(n: int, device) -> torch.Tensor:
    return torch.empty(max(int(n), 0), dtype=I32, device=device)


def tile_stats(leaves, rows: int, device, tile_rows_a: int = 8, tile_rows_b: int = 32):
    """``(largest a-row tile, largest b-row tile, largest a-row tile span)`` in boundaries and coordinates.

    One launch of ``sx_tile_boundaries_max`` and one read-back.
    """
    if rows <= 0 or any(len(leaf) > 5 and leaf[5] is not None for leaf in leaves):
        return 0, 0, 0  # no rows, or explicit row ranges (the union sweep has no tiles)
    lib = _lib.load()
    arr = (_lib.SxLeaf * len(leaves))()
    for i, leaf in enumerate(leaves):
        arr[i].begin = ptr(leaf[0])
        arr[i].end = ptr(leaf[1])
        arr[i].row_offsets = ptr(leaf[2])
    out = empty_i32(3, device)
    _lib.check(lib.sx_tile_boundaries_max(arr, len(leaves), int(rows), int(tile_rows_a), int(tile_rows_b), ptr(out),
                                          stream_handle(device)), "sx_tile_boundaries_max")
    a, b, span = (int(x) for x in out.tolist())
    return a, b, span


def max_tile_boundaries(leaves, rows: int, device, tile_rows=32):
    """Largest number of leaf boundaries in one tile of ``tile_rows`` aligned rows (one synchronisation).

    ``tile_rows`` may be a pair of tile heights; the result is then a list
    with one maximum per height, from the same launch and read-back.
    """
    heights = list(tile_rows) if isinstance(tile_rows, (tuple, list)) else [tile_rows, tile_rows]
    a, b, _ = tile_stats(leaves, rows, device, heights[0], heights[1])
    return [a, b] if isinstance(tile_rows, (tuple, list)) else a


def _default_keys(leaves, rows: int, tile_rows: int = 32) -> int:
    tiles = max(1, (rows + tile_rows - 1) // tile_rows)
    avg = 2 * sum(int(leaf[0].numel()) for leaf in leaves) // tiles
    return avg + avg // 4 + 64


def auto_tuning(leaves, rows: int, device) -> dict:
    """The launch shape of a truth-table sweep measured on its operands (one launch and one read-back, two when rows are skewed).

    Even rows (the largest 8-row tile within 3x the mean plus 256
    boundaries): the row-lane sweep on 16-row tiles when every such tile
    spans at most 65534 columns (16-bit coordinates), else 8-row warp tiles
    with 32-bit keys; buffers are sized for the largest tile, so no tile
    leaves the staged sweep (tiles that no buffer holds: 8 rows, for twice
    the warps).  Skewed rows: 32-row block tiles sized for their
    largest tile, which evens out the load.
    """
    need16, need8, span16 = tile_stats(leaves, rows, device, 16, 8)
    mean8 = 2 * sum(int(leaf[0].numel()) for leaf in leaves) / max(1, (rows + 7) // 8)
    if need8 <= 3 * mean8 + 256:
        if span16 <= 65534:
            return {"kernel": 7, "staging_cap": min(need16, 25000), "tile_rows": 16 if need16 <= 25000 else 8,
                    "warps": 2}
        return {"kernel": 5, "staging_cap": min(need8, 25000), "tile_rows": 8, "warps": 2}
    need32 = max_tile_boundaries(leaves, rows, device, tile_rows=32)
    return {"kernel": 4, "staging_cap": min(need32, 25000), "tile_rows": 32, "warps": 4}


def even_tuning(leaves, rows: int, total: Optional[int] = None) -> dict:
    """The launch shape of ``sx_bool_eval_even``, from the operands' sizes alone.

    The row-lane sweep on tiles of 16 rows, or 8 when rows are so long that a
    mean tile would exceed ``_TILE_INTERVALS``.  The sweep waits for latencies,
    so its speed goes with the resident blocks: as many as slices for the
    mean tile and a twentieth more allow (at most what the registers leave
    room for), each with all the shared memory that this count gives it.  The
    tiles above that are swept in groups of rows by the same launch.
    Measured: five shape leaves over 128 copies of 4096 rows (mean 16-row tile
    1155 intervals, largest 1253) 421 us with 16 rows, 433 us with 8, 474 us
    with 32, 615 us when the slices fall short of the largest tiles; the sweep
    alone 274 us at 10 blocks per SM, 289 us at 9.
    """
    k = len(leaves)
    total = sum(int(leaf[0].numel()) for leaf in leaves) if total is None else total
    tr = 16 if 16 * total <= _TILE_INTERVALS * rows else 8
    mean = tr * total // max(1, rows)
    gap = max((k - 1) * (tr - 7) + tr, k * (tr + 1) + tr - 16 * k) + 4
    fixed = 22 * k + 16 + gap  # words of a warp's slice beside two per interval
    per_block = 2 * 4 * (2 * (mean + mean // 20 + 32) + fixed) + 1024
    blocks = max(1, min(_SM_SHARED // per_block, 16 if k <= 4 else 12))
    room = ((min(_SM_SHARED // blocks, 200 * 1024) - 1024) // 8 - fixed) // 2
    return {"kernel": 7, "staging_cap": min(2 * room, 25000), "tile_rows": tr, "warps": 2}


def bool_eval(leaves: Sequence[Tuple[torch.Tensor, torch.Tensor, torch.Tensor, int]], rows: int, table: Sequence[int],
              mode: int, device, out: Optional[Tuple[torch.Tensor, torch.Tensor]] = None):
    """Run the row sweep (sx_bool_eval) and read back its result pair.

    ``leaves`` are ``(begin, end, aligned_offsets, widen[, scale[, row_ends]])``
    tuples; ``mode``
    is ``_lib.MODE_TABLE`` (truth table over canonical leaves) or
    ``_lib.MODE_UNION`` (merged union of widened leaves).  Returns
    ``(begin, end, offsets, total, flags)``; begin and end are capacity
    buffers to be sliced to ``total``.
    """
    tuning = None
    tuned = TUNED.get(workload_key([int(leaf[0].numel()) for leaf in leaves], rows)) if TUNED else None
    if mode == _lib.MODE_TABLE and not TUNING and rows > 0 and tuned is not None:
        tuning = dict(tuned)
        if tuning.get("kernel") in (3, 4, 5, 6, 7):
            tr = int(tuning.get("tile_rows", 0)) or {5: 8, 6: 8, 7: 16}.get(tuning["kernel"], 32)
            tuning["staging_cap"] = min(max_tile_boundaries(leaves, rows, device, tile_rows=tr), 25000)
    elif mode == _lib.MODE_TABLE and not TUNING and rows > 0:
        # Most operands have rows alike, and the sweep that assumes it needs no pass that
        # measures them first (59 us and a read-back beside a 270 us sweep of 5 x 128 x 4096
        # rows; 35 us of 160 at 256 rows).  It gives up early on others (rows too long, or
        # too wide for 16-bit coordinates), and what it has counted by then shapes the launch
        # for those.
        return _eval_even(leaves, rows, table, device, out)
    ob, oe, ooff, result = bool_eval_async(leaves, rows, table, mode, device, out, tuning=tuning)
    if result is None:
        return ob, oe, ooff, 0, 0
    total, flags = read_pair(result)
    return ob, oe, ooff, total, flags


def _eval_even(leaves, rows: int, table, device, out):
    """:func:`bool_eval` of a truth table without a launch shape: the sweep for even rows, then another if it gives up."""
    lib = _lib.load()
    args, cap, (ob, oe, ooff) = _sweep_args(leaves, rows, table, device, out, None)
    wsp, wsn, words = workspace_words(device, int(lib.sx_bool_workspace_bytes(int(rows))))
    stream = stream_handle(device)
    tuning = even_tuning(leaves, rows, cap)
    outs = (ob.data_ptr(), oe.data_ptr(), ooff.data_ptr(), cap, wsp + 160, wsp, wsn)
    _lib.check(lib.sx_bool_eval_even(*args, *outs, ctypes.byref(_tuning_struct(tuning)), stream), "sx_bool_eval_even")
    most8, most32, why, *_, total, flags = words.tolist()
    if flags == _lib.FLAG_LONG_TILE:
        tuning = _uneven_tuning(leaves, rows, device, tuning, most8, most32, why == 3)
        _lib.check(lib.sx_bool_eval(*args, _lib.MODE_TABLE, *outs, ctypes.byref(_tuning_struct(tuning)), stream),
                   "sx_bool_eval")
        total, flags = words.tolist()[8:]
    return ob, oe, ooff, total, flags


def _uneven_tuning(leaves, rows: int, device, even: dict, most8: int, most32: int, wide: bool) -> dict:
    """The launch shape after ``sx_bool_eval_even`` (tuned ``even``) has given up, by what it has counted.

    The choice is that of :func:`auto_tuning`: kernel 5 for even rows too
    wide for 16 bits, its buffers for the largest 8 rows; kernel 4 for
    skewed ones, its buffers for the largest 32 rows, those around a tile
    that gave up or tiles that fitted.  Even, narrow rows that no slice
    holds are long; measuring them costs little beside their sweep.
    """
    mean8 = 2 * sum(int(leaf[0].numel()) for leaf in leaves) / max(1, (rows + 7) // 8)
    if 2 * most8 > 3 * mean8 + 256:
        fitted = 32 // even["tile_rows"] * even["staging_cap"]
        return {"kernel": 4, "staging_cap": min(max(2 * most32, fitted), 25000), "tile_rows": 32, "warps": 4}
    if wide:
        return {"kernel": 5, "staging_cap": min(2 * most8, 25000), "tile_rows": 8, "warps": 2}
    return auto_tuning(leaves, rows, device)


_TUNING_FIELDS = [name for name, _ in _lib.SxTuning._fields_]
_TABLE_WORDS = ctypes.c_uint32 * 8


def _tuning_struct(t: dict) -> "_lib.SxTuning":
    return _lib.SxTuning(*[int(t.get(name, 0)) for name in _TUNING_FIELDS])


def _sweep_args(leaves, rows: int, table, device, out, offsets):
    """``((leaves, k, rows, table), capacity, (begin, end, offsets))`` of a sweep, for the C calls."""
    k = len(leaves)
    cap = max(1, sum([int(leaf[0].numel()) for leaf in leaves]))
    if out is None:
        ob = empty_i32(cap, device)
        oe = empty_i32(cap, device)
    else:
        ob, oe = out
        if ob.numel() < cap or oe.numel() < cap:
            raise ValueError("output buffers below the required capacity")
    ooff = empty_i32(rows + 1, device) if offsets is None else offsets
    arr = (_lib.SxLeaf * k)(*[_lib.SxLeaf(ptr(leaf[0]), ptr(leaf[1]), ptr(leaf[2]),
                                          ptr(leaf[5]) if len(leaf) > 5 else None, int(leaf[3]),
                                          int(leaf[4]) if len(leaf) > 4 else 0) for leaf in leaves])
    tab = _TABLE_WORDS(*[int(x) & 0xFFFFFFFF for x in (list(table) + [0] * 8)[:8]])
    return (arr, k, int(rows), tab), cap, (ob, oe, ooff)


def bool_eval_async(leaves: Sequence[Tuple[torch.Tensor, torch.Tensor, torch.Tensor, int]], rows: int,
                    table: Sequence[int], mode: int, device, out: Optional[Tuple[torch.Tensor, torch.Tensor]] = None,
                    result: Optional[torch.Tensor] = None, offsets: Optional[torch.Tensor] = None,
                    tuning: Optional[dict] = None, scratch: Optional[torch.Tensor] = None, even: bool = False):
    """Enqueue the row sweep without waiting (``even``: ``sx_bool_eval_even``, a truth table with a kernel 7 tuning).

    Returns ``(begin, end, offsets, result)``; ``result`` is the device pair
    ``(total, flags)``, or None when there are no rows.  ``scratch`` (bytes,
    at least ``sx_bool_workspace_bytes(rows)``) replaces the per-stream
    workspace, for launches captured in a graph.
    """
    lib = _lib.load()
    args, cap, (ob, oe, ooff) = _sweep_args(leaves, rows, table, device, out, offsets)
    if rows == 0:
        ooff.zero_()
        return ob, oe, ooff, None
    if result is None:
        result = empty_i32(2, device)
    need = int(lib.sx_bool_workspace_bytes(int(rows)))
    if scratch is None:
        wsp, wsn = workspace(device, need)
    else:
        if int(scratch.numel()) < need:
            raise ValueError("scratch below sx_bool_workspace_bytes(rows)")
        wsp, wsn = scratch.data_ptr(), int(scratch.numel())
    tun = _tuning_struct(TUNING if tuning is None else tuning)
    if even:
        rc = lib.sx_bool_eval_even(*args, ptr(ob), ptr(oe), ptr(ooff), cap, ptr(result), wsp, wsn, ctypes.byref(tun),
                                   stream_handle(device))
    else:
        rc = lib.sx_bool_eval(*args, int(mode), ptr(ob), ptr(oe), ptr(ooff), cap, ptr(result), wsp, wsn,
                              ctypes.byref(tun), stream_handle(device))
    _lib.check(rc, "sx_bool_eval")
    return ob, oe, ooff, result


def scan(counts: torch.Tensor, device) -> Tuple[torch.Tensor, int]:
    """Exclusive prefix sum: ``(offsets[n + 1], total)`` (synchronising)."""
    lib = _lib.load()
    n = int(counts.numel())
    out = empty_i32(n + 1, device)
    result = empty_i32(2, device)
    wsp, wsn = workspace(device, lib.sx_scan_workspace_bytes(n))
    rc = lib.sx_scan_i32(ptr(counts), n, ptr(out), ptr(result), wsp, wsn, stream_handle(device))
    _lib.check(rc, "sx_scan_i32")
    total, flags = read_pair(result)
    if flags & _lib.FLAG_TIMEOUT:
        raise _lib.SubsetixError("sx_scan_i32: look-back wait timed out")
    return out, total


def exact_setop(op: int, lhs, rhs, rows: int, device):
    """Reference-order binary op on aligned operands.  Returns ``(begin, end, offsets)``."""
    lib = _lib.load()
    lb, le, loff = lhs
    rb, re, roff = rhs
    if rows == 0:
        return empty_i32(0, device), empty_i32(0, device), torch.zeros(1, dtype=I32, device=device)
    counts = empty_i32(rows, device)
    s = stream_handle(device)
    rc = lib.sx_exact_setop(op, rows, ptr(lb), ptr(le), ptr(loff), ptr(rb), ptr(re), ptr(roff), ptr(counts), None,
                            None, None, s)
    _lib.check(rc, "sx_exact_setop(count)")
    off, total = scan(counts, device)
    ob = empty_i32(total, device)
    oe = empty_i32(total, device)
    if total:
        rc = lib.sx_exact_setop(op, rows, ptr(lb), ptr(le), ptr(loff), ptr(rb), ptr(re), ptr(roff), None, ptr(off),
                                ptr(ob), ptr(oe), s)
        _lib.check(rc, "sx_exact_setop(write)")
    return ob, oe, off


def merge_rows(begin: torch.Tensor, end: torch.Tensor, offsets: torch.Tensor, device):
    """Run merge of begin-sorted rows (kernels.py:292-381).  Returns ``(begin, end, offsets)``."""
    lib = _lib.load()
    rows = int(offsets.numel()) - 1
    if rows <= 0:
        return empty_i32(0, device), empty_i32(0, device), torch.zeros(max(rows, 0) + 1, dtype=I32, device=device)
    counts = empty_i32(rows, device)
    s = stream_handle(device)
    _lib.check(lib.sx_merge_rows(rows, ptr(begin), ptr(end), ptr(offsets), ptr(counts), None, None, None, s),
               "sx_merge_rows(count)")
    off, total = scan(counts, device)
    ob = empty_i32(total, device)
    oe = empty_i32(total, device)
    if total:
        _lib.check(lib.sx_merge_rows(rows, ptr(begin), ptr(end), ptr(offsets), None, ptr(off), ptr(ob), ptr(oe), s),
                   "sx_merge_rows(write)")
    return ob, oe, off


def box_sweep(begin, end, offsets, rows, device, *, dense: bool, y_base: int, out_rows: int, x_lo: int, x_hi: int,
              halo_y: int = 0, w_center: int = 0, w_other: int = 0, mode: int = _lib.BOX_DILATE, ratio: int = 0,
              compact: bool = False):
    """sx_box_sweep and its read-back: ``(intervals, offsets, row ids or None, total, flags)``.

    ``intervals`` holds the begins and the ends, two rows of the output's
    capacity; with ``compact`` offsets and row ids are cut to the kept rows.
    """
    lib = _lib.load()
    n, out_rows = int(begin.numel()), int(out_rows)
    views = 1 if mode == _lib.BOX_RESTRICT else 2 * int(halo_y) + 1  # output rows that one source row reaches
    cap = views * n + (views + 1) * out_rows if mode == _lib.BOX_ERODE else max(1, views * n)
    box = _lib.SxBox(ptr(begin), ptr(end), ptr(offsets), None if dense else ptr(rows), n, int(offsets.numel()) - 1,
                     1 if dense else 0, 0, int(y_base), out_rows, int(x_lo), int(x_hi), int(halo_y), int(w_center),
                     int(w_other), int(mode), int(ratio))
    out = torch.empty((2, (cap + 3) & ~3), dtype=I32, device=device)  # both rows 16-byte aligned
    off = empty_i32(out_rows + 1, device)
    ids = empty_i32(out_rows, device) if compact else None
    result = empty_i32(3, device)
    wsp, wsn = workspace(device, lib.sx_bool_workspace_bytes(out_rows))
    _lib.check(lib.sx_box_sweep(ctypes.byref(box), ptr(out[0]), ptr(out[1]), ptr(off), ptr(ids), cap, ptr(result),
                                wsp, wsn, stream_handle(device)), "sx_box_sweep")
    total, flags, kept = result.tolist()
    if compact:
        off, ids = off[:kept + 1], ids[:kept]
    return out, off, ids, total, flags


def align_rows(lists: Sequence[tuple], row_min: int, row_max: int, device, want_offsets: Sequence[bool],
               want_ends: Optional[Sequence[bool]] = None):
    """Sorted union of ``floor((rows + shift) / div)`` over the lists, plus aligned offsets.

    ``lists`` holds ``(rows, offsets, shift, skip_empty[, div, phase])``
    tuples.  Returns ``(rows_out, [aligned offsets or None])``, or with
    ``want_ends`` ``(rows_out, [starts or None], [stops or None])``.  This
    call synchronises.
    """
    lib = _lib.load()
    k = len(lists)
    cap = 0
    for item in lists:
        cap += int(item[0].numel())
    span = int(row_max) - int(row_min) + 1
    cap = max(1, min(cap, max(span, 1)))
    rows_out = empty_i32(cap, device)
    aligned = [empty_i32(cap + 1, device) if w else None for w in want_offsets]
    ends = [empty_i32(cap, device) if w else None for w in (want_ends or [False] * k)]
    arr = (_lib.SxRowList * k)()
    for i, item in enumerate(lists):
        rows, off, shift, skip = item[:4]
        arr[i].rows = ptr(rows)
        arr[i].row_offsets = ptr(off)
        arr[i].count = int(rows.numel())
        arr[i].shift = int(shift)
        arr[i].skip_empty = 1 if skip else 0
        arr[i].div = int(item[4]) if len(item) > 4 else 1
        arr[i].phase = int(item[5]) if len(item) > 5 else 0
    aptrs = (ctypes.c_void_p * k)(*[ptr(a) if a is not None else None for a in aligned])
    eptrs = (ctypes.c_void_p * k)(*[ptr(a) if a is not None else None for a in ends])
    result = empty_i32(2, device)
    wsp, wsn = workspace(device, lib.sx_align_workspace_bytes(int(row_min), int(row_max)))
    rc = lib.sx_align_rows(arr, k, int(row_min), int(row_max), ptr(rows_out), cap, aptrs,
                           eptrs if want_ends else None, ptr(result), wsp, wsn, stream_handle(device))
    _lib.check(rc, "sx_align_rows")
    n, flags = read_pair(result)
    if flags & _lib.FLAG_TIMEOUT:
        raise _lib.SubsetixError("sx_align_rows: look-back wait timed out")
    starts = [a[: n + 1] if a is not None else None for a in aligned]
    if want_ends:
        return rows_out[:n], starts, [a[:n] if a is not None else None for a in ends]
    return rows_out[:n], starts


# ---------------------------------------------------------------------------
# Interval fields and multilevel kernels
# ---------------------------------------------------------------------------

def _flag_word(device) -> torch.Tensor:
    return empty_i32(1, device)


def check_rows(begin: torch.Tensor, end: torch.Tensor, offsets: torch.Tensor, device, sync: bool = True):
    """OR of ``_lib.ROWS_*`` bits over adjacent interval pairs (sx_check_rows)."""
    lib = _lib.load()
    flags = _flag_word(device)
    rows = int(offsets.numel()) - 1
    _lib.check(lib.sx_check_rows(ptr(begin), ptr(end), ptr(offsets), max(rows, 0), int(begin.numel()), ptr(flags),
                                 stream_handle(device)), "sx_check_rows")
    return int(flags.item()) if sync else flags


def cell_offsets(begin: torch.Tensor, end: torch.Tensor, device, sync: bool = True,
                 result: Optional[torch.Tensor] = None):
    """int32 exclusive scan of interval lengths.  Returns ``(offsets, total)``, without ``sync`` ``(offsets, result)``."""
    lib = _lib.load()
    n = int(begin.numel())
    out = empty_i32(n + 1, device)
    if result is None:
        result = empty_i32(2, device)
    wsp, wsn = workspace(device, lib.sx_scan_workspace_bytes(n))
    _lib.check(lib.sx_cell_offsets(ptr(begin), ptr(end), n, ptr(out), ptr(result), wsp, wsn, stream_handle(device)),
               "sx_cell_offsets")
    if not sync:
        return out, result
    total, flags = read_pair(result)
    check_scan(flags, "sx_cell_offsets")
    return out, total


def check_scan(flags: int, what: str) -> None:
    if flags & _lib.FLAG_TIMEOUT:
        raise _lib.SubsetixError(f"{what}: look-back wait timed out")


def prolong_set(rows: torch.Tensor, offsets: torch.Tensor, begin: torch.Tensor, end: torch.Tensor, ratio: int,
                device, cells: bool = False):
    """sx_prolong_set.  Returns ``(rows_out, offsets_out, begin, end, unsorted)`` sized to the output.

    With ``cells`` also ``(cell offsets, cell total)`` of the intervals as
    they come, from the same read-back.
    """
    lib = _lib.load()
    R = int(rows.numel())
    n = int(begin.numel())
    rows_out = empty_i32(R * ratio, device)
    off_out = empty_i32(R * ratio + 1, device)
    ob = empty_i32(n * ratio, device)
    oe = empty_i32(n * ratio, device)
    result = empty_i32(4, device)
    wsp, wsn = workspace(device, lib.sx_prolong_set_workspace_bytes(R))
    _lib.check(lib.sx_prolong_set(ptr(rows), ptr(offsets), ptr(begin), ptr(end), R, n, int(ratio), ptr(rows_out),
                                  ptr(off_out), ptr(ob), ptr(oe), ptr(result), wsp, wsn, stream_handle(device)),
               "sx_prolong_set")
    if cells:
        cell_off, _ = cell_offsets(ob, oe, device, sync=False, result=result[2:])
        occupied, flags, total, scan_flags = result.tolist()
        check_scan(scan_flags, "sx_cell_offsets")
    else:
        occupied, flags = read_pair(result[:2])
    check_scan(flags, "sx_prolong_set")
    m = occupied * ratio
    out = (rows_out[:m], off_out[: m + 1], ob, oe, bool(flags & 1))
    return (*out, cell_off, total) if cells else out


def _dtype_code(t: torch.Tensor) -> int:
    if t.dtype == torch.float32:
        return _lib.SX_F32
    if t.dtype == torch.float64:
        return _lib.SX_F64
    raise TypeError(f"field values must be float32 or float64, got {t.dtype}")


def prolong_field(coarse_offsets, coarse_cell_offsets, n: int, fine_offsets, fine_cell_offsets, ratio: int,
                  coarse_values, fine_values, device):
    lib = _lib.load()
    rows = int(coarse_offsets.numel()) - 1
    _lib.check(lib.sx_prolong_field(_dtype_code(coarse_values), ptr(coarse_offsets), rows, ptr(coarse_cell_offsets),
                                    int(n), ptr(fine_offsets), ptr(fine_cell_offsets), int(ratio), ptr(coarse_values),
                                    ptr(fine_values), stream_handle(device)), "sx_prolong_field")


def coarse_fine_check(coarse, fine, ratio: int, device, flags: Optional[torch.Tensor] = None):
    """Flags of sx_coarse_fine_check.  ``coarse``/``fine`` are ``(rows, offsets, begin, end)``.

    Given ``flags`` (one int on the device) they are left there unread.
    """
    lib = _lib.load()
    cr, coff, cb, ce = coarse
    fr, foff, fb, fe = fine
    own = flags is None
    flags = _flag_word(device) if own else flags
    _lib.check(lib.sx_coarse_fine_check(ptr(cr), int(cr.numel()), ptr(coff), ptr(cb), ptr(ce), int(cb.numel()),
                                        ptr(fr), int(fr.numel()), ptr(foff), ptr(fb), ptr(fe), int(fb.numel()),
                                        int(ratio), ptr(flags), stream_handle(device)), "sx_coarse_fine_check")
    return int(flags.item()) if own else flags


def restrict_field(coarse_offsets, coarse_cell_offsets, coarse_n: int, fine_offsets, fine_cell_offsets, ratio: int,
                   reducer: int, fine_values, coarse_values, device):
    lib = _lib.load()
    rows = int(coarse_offsets.numel()) - 1
    _lib.check(lib.sx_restrict_field(_dtype_code(fine_values), ptr(coarse_offsets), rows, ptr(coarse_cell_offsets),
                                     int(coarse_n), ptr(fine_offsets), ptr(fine_cell_offsets), int(ratio),
                                     int(reducer), ptr(fine_values), ptr(coarse_values), stream_handle(device)),
               "sx_restrict_field")


def subset_rows(sub_offsets, sub_rows, sub_n: int, sup_rows, device, sync: bool = True):
    """Superset row ordinal per subset interval.  Returns ``(pos, missing)``."""
    lib = _lib.load()
    pos = empty_i32(sub_n, device)
    flags = _flag_word(device)
    _lib.check(lib.sx_subset_rows(ptr(sub_offsets), ptr(sub_rows), int(sub_rows.numel()), int(sub_n), ptr(sup_rows),
                                  int(sup_rows.numel()), ptr(pos), ptr(flags), stream_handle(device)),
               "sx_subset_rows")
    return pos, (bool(flags.item()) if sync else flags)


def subset_copy(scatter: bool, pos, sub, sup, sub_values, sup_values, device):
    """sx_subset_copy.  ``sub`` = ``(begin, end, cell_offsets)``; ``sup`` = ``(offsets, begin, end, cell_offsets)``."""
    lib = _lib.load()
    sb, se, scoff = sub
    uoff, ub, ue, ucoff = sup
    _lib.check(lib.sx_subset_copy(1 if scatter else 0, int(sb.numel()), ptr(pos), ptr(sb), ptr(se), ptr(scoff),
                                  ptr(uoff), ptr(ub), ptr(ue), ptr(ucoff), int(uoff.numel()) - 1, ptr(sub_values),
                                  ptr(sup_values), int(sub_values.element_size()), stream_handle(device)),
               "sx_subset_copy")


def row_lookup(rows, height: int, device, sync: bool = True):
    """Row ordinal per row id in [0, height) (-1 when absent).  Returns ``(lookup, out_of_range)``."""
    lib = _lib.load()
    lookup = empty_i32(height, device)
    flags = _flag_word(device)
    _lib.check(lib.sx_row_lookup(ptr(rows), int(rows.numel()), int(height), ptr(lookup), ptr(flags),
                                 stream_handle(device)), "sx_row_lookup")
    return lookup, (bool(flags.item()) if sync else flags)


def stencil_geometry(rows, offsets, begin, end, height: int, device):
    """What a stencil needs to know about a new set, with one read-back.

    Returns ``(lookup, out_of_range, row flags, cell offsets, cells, (first
    column, last column + 1))``; the last three hold for sorted, disjoint rows.
    """
    lib, s = _lib.load(), stream_handle(device)
    n, rows_n = int(begin.numel()), int(rows.numel())
    facts = empty_i32(6, device)
    at = facts.data_ptr()
    lookup, cell_off = empty_i32(height, device), empty_i32(n + 1, device)
    _lib.check(lib.sx_row_lookup(ptr(rows), rows_n, int(height), ptr(lookup), at, s), "sx_row_lookup")
    _lib.check(lib.sx_check_rows(ptr(begin), ptr(end), ptr(offsets), max(int(offsets.numel()) - 1, 0), n, at + 4, s),
               "sx_check_rows")
    wsp, wsn = workspace(device, lib.sx_scan_workspace_bytes(n))
    _lib.check(lib.sx_cell_offsets(ptr(begin), ptr(end), n, ptr(cell_off), at + 8, wsp, wsn, s), "sx_cell_offsets")
    # no cells: the plan's launch finds the columns only
    _lib.check(lib.sx_upwind_flat_plan(None, None, 0, ptr(begin), ptr(end), None, n, 0, None, int(height), None, None,
                                       None, None, at + 16, s), "sx_upwind_flat_plan")
    bad, flags, cells, scan_flags, lo, hi = facts.tolist()
    check_scan(scan_flags, "sx_cell_offsets")
    return lookup, bool(bad), flags, cell_off, cells, (lo, hi)


def upwind(rows, offsets, begin, end, cell_offs, cells: int, lookup, values, out, width: int, height: int, a, b, dt,
           dx, dy, direct: bool, device, row_ids=None):
    lib = _lib.load()
    _lib.check(lib.sx_upwind(_dtype_code(values), ptr(rows), ptr(row_ids), ptr(offsets), int(rows.numel()), ptr(begin),
                             ptr(end), ptr(cell_offs), int(begin.numel()), int(cells), ptr(lookup), ptr(values),
                             ptr(out), int(width), int(height), float(a), float(b), float(dt), float(dx), float(dy),
                             1 if direct else 0, stream_handle(device)), "sx_upwind")


def upwind_plan(rows, offsets, begin, end, cell_offs, lookup, height: int, device):
    """Plan of sx_upwind_chunked for a fixed geometry: ``(chunk_info, chunks)`` (one synchronisation)."""
    lib = _lib.load()
    n = int(begin.numel())
    chunk_off = empty_i32(n + 1, device)
    result = empty_i32(2, device)
    wsp, wsn = workspace(device, lib.sx_scan_workspace_bytes(n))
    s = stream_handle(device)
    _lib.check(lib.sx_upwind_plan(ptr(begin), ptr(end), n, ptr(chunk_off), ptr(result), wsp, wsn, s),
               "sx_upwind_plan")
    chunks, flags = read_pair(result)
    if flags & _lib.FLAG_TIMEOUT:
        raise _lib.SubsetixError("sx_upwind_plan: look-back wait timed out")
    info = empty_i32(16 * max(chunks, 1), device)
    _lib.check(lib.sx_upwind_plan_fill(ptr(rows), ptr(offsets), int(rows.numel()), ptr(begin), ptr(end),
                                       ptr(cell_offs), n, ptr(chunk_off), chunks, ptr(lookup), int(height), ptr(info),
                                       s), "sx_upwind_plan_fill")
    return info, chunks


def upwind_table(begin, end, cell_offs, chunk_info, chunks: int, cells: int, device):
    """Neighbour table of a chunk plan (uint16 per cell; one synchronisation)."""
    lib = _lib.load()
    table = torch.empty(max(int(cells), 1), dtype=torch.int16, device=device)
    status = empty_i32(1, device)
    _lib.check(lib.sx_upwind_plan_table(ptr(begin), ptr(end), ptr(cell_offs), ptr(chunk_info), int(chunks), ptr(table),
                                        ptr(status), stream_handle(device)), "sx_upwind_plan_table")
    if int(status.item()):
        raise _lib.SubsetixError("sx_upwind_plan_table: cell offsets are not the packed prefix sum")
    return table


def upwind_chunked(offsets, begin, end, cell_offs, chunk_info, chunks: int, lookup, values, out, width: int,
                   height: int, a, b, dt, dx, dy, device, table=None):
    lib = _lib.load()
    _lib.check(lib.sx_upwind_chunked(_dtype_code(values), ptr(offsets), ptr(begin), ptr(end), ptr(cell_offs),
                                     ptr(chunk_info), int(chunks), ptr(lookup), ptr(table), ptr(values), ptr(out),
                                     int(width), int(height), float(a), float(b), float(dt), float(dx), float(dy),
                                     stream_handle(device)), "sx_upwind_chunked")


class FlatPlan:
    """Plan of sx_upwind_flat for sorted, disjoint rows and packed values, with the columns it spans.

    ``columns`` is that span, where known; else it is read back.
    """

    __slots__ = ("cells", "lo", "hi", "_keep", "_struct", "_ref")

    def __init__(self, rows, offsets, begin, end, cell_offs, cells: int, lookup, height: int, device,
                 columns: Optional[Tuple[int, int]] = None):
        lib = _lib.load()
        n, cells = int(begin.numel()), int(cells)
        groups = (cells + 3) // 4
        below, above = empty_i32(groups, device), empty_i32(groups, device)
        flags = torch.empty(groups, dtype=torch.int16, device=device)
        side = empty_i32(8 * n, device)
        span = empty_i32(2, device)
        _lib.check(lib.sx_upwind_flat_plan(ptr(rows), ptr(offsets), int(rows.numel()), ptr(begin), ptr(end),
                                           ptr(cell_offs), n, cells, ptr(lookup), int(height), ptr(below), ptr(above),
                                           ptr(flags), ptr(side), ptr(span), stream_handle(device)),
                   "sx_upwind_flat_plan")
        self.cells = cells
        self.lo, self.hi = span.tolist() if columns is None else columns
        self._keep = (below, above, flags, side)
        self._struct = _lib.SxFlatPlan(ptr(below), ptr(above), ptr(flags), ptr(side), n, cells)
        self._ref = ctypes.byref(self._struct)

    def covers(self, width: int) -> bool:
        """Whether every cell lies in columns [0, width)."""
        return self.cells > 0 and self.lo >= 0 and self.hi <= int(width)

    def step(self, values, out, a, b, dt, dx, dy, device) -> None:
        _lib.check(_lib.load().sx_upwind_flat(_dtype_code(values), self._ref, ptr(values), ptr(out), float(a), float(b),
                                              float(dt), float(dx), float(dy), stream_handle(device)), "sx_upwind_flat")

    def step_bands(self, values, out, a, b, band_cell, band_table, bands: int, device) -> None:
        _lib.check(_lib.load().sx_upwind_flat_bands(_dtype_code(values), self._ref, ptr(values), ptr(out), float(a),
                                                    float(b), ptr(band_cell), ptr(band_table), int(bands),
                                                    stream_handle(device)), "sx_upwind_flat_bands")

    def adjoint(self, w, u, out, a, b, dt, dx, dy, grad, scratch, device) -> None:
        """``out`` = the transposed step of ``w``; the velocity gradient is added to ``grad``."""
        _lib.check(_lib.load().sx_upwind_flat_adjoint(_dtype_code(w), self._ref, ptr(w), ptr(u), ptr(out), float(a),
                                                      float(b), float(dt), float(dx), float(dy), ptr(grad), 1,
                                                      ptr(scratch), int(scratch.numel()), stream_handle(device)),
                   "sx_upwind_flat_adjoint")


def threshold_rle(values, width: int, height: int, threshold: float, gradient: bool, device):
    """Runs of value >= threshold per row of a full grid.  Returns ``(begin, end, offsets)`` (synchronising).

    Tall, narrow grids are read twice, a warp per row: the mask's strips of
    128 columns are mostly empty there, and its rows many (200,000 rows, device
    time of both ways with the threshold of the values and of the gradient:
    3 columns 55 against 145 and 82 against 188 us, 128 columns 121 against
    177 and 203 against 227, 256 columns 211 against 203 and 370 against 308;
    20,000 rows of 3 columns 19 against 29; 2000 rows 16 against 17, and two
    launches more).
    """
    lib = _lib.load()
    width, height = int(width), int(height)
    if width <= 128 and height > 10000:
        counts = empty_i32(height, device)
        s = stream_handle(device)
        args = (ptr(values), width, height, float(threshold), 1 if gradient else 0)
        _lib.check(lib.sx_threshold_rle(*args, ptr(counts), None, None, None, s), "sx_threshold_rle(count)")
        off, total = scan(counts, device)
        ob, oe = empty_i32(total, device), empty_i32(total, device)
        if total:
            _lib.check(lib.sx_threshold_rle(*args, None, ptr(off), ptr(ob), ptr(oe), s), "sx_threshold_rle(write)")
        return ob, oe, off
    mask = empty_i32(height * ((width + 31) // 32), device)
    off = empty_i32(height + 1, device)
    result = empty_i32(2, device)
    s = stream_handle(device)
    wsp, wsn = workspace(device, lib.sx_threshold_mask_workspace_bytes(height))
    _lib.check(lib.sx_threshold_mask(ptr(values), width, height, float(threshold), 1 if gradient else 0, ptr(mask),
                                     ptr(off), ptr(result), wsp, wsn, s), "sx_threshold_mask")
    total, flags = read_pair(result)
    if flags & _lib.FLAG_TIMEOUT:
        raise _lib.SubsetixError("sx_threshold_mask: look-back wait timed out")
    ob = empty_i32(total, device)
    oe = empty_i32(total, device)
    if total:
        _lib.check(lib.sx_mask_runs(ptr(mask), width, height, ptr(off), ptr(ob), ptr(oe), s), "sx_mask_runs")
    return ob, oe, off


def select_top(values: torch.Tensor, epsilon: float, fraction: float, device) -> Tuple[float, int]:
    """``(value, m)``: the value that ``ceil(fraction * m)`` of the ``m`` float32 values above ``epsilon`` reach."""
    lib = _lib.load()
    result = empty_i32(2, device)
    scratch = torch.empty(int(lib.sx_select_top_workspace_bytes()), dtype=torch.uint8, device=device)
    _lib.check(lib.sx_select_top(ptr(values), int(values.numel()), float(epsilon), float(fraction), ptr(result),
                                 ptr(scratch), int(scratch.numel()), stream_handle(device)), "sx_select_top")
    bits, above = result.tolist()
    return struct.unpack("<f", struct.pack("<i", bits))[0], above


def mass_integral(values, scale: float, device, out: Optional[torch.Tensor] = None, parts: int = 592):
    """Compensated FP64 sum times ``scale`` into a device scalar (no synchronisation)."""
    lib = _lib.load()
    if out is None:
        out = torch.empty(1, dtype=torch.float64, device=device)
    part = torch.empty(2 * parts, dtype=torch.float64, device=device)
    _lib.check(lib.sx_mass_integral(_dtype_code(values), ptr(values), int(values.numel()), float(scale), ptr(part),
                                    int(parts), ptr(out), stream_handle(device)), "sx_mass_integral")
    return out
