"""Differentiable multi-step upwind advection on fixed interval geometry.

``advect`` runs ``steps`` first-order upwind steps on one or more interval
fields (levels) that share a velocity ``(a, b)`` and a time step, and is a
``torch.autograd.Function``: the backward pass applies the hand-written
adjoint kernel ``sx_upwind_adjoint`` step by step, which returns the
gradient with respect to the step's input and the gradient with respect to
the velocity (time step held fixed).  Forward states are kept only every
``checkpoint_every`` steps; the backward pass recomputes each segment from
its checkpoint, so memory holds ``steps / checkpoint_every + checkpoint_every``
states per level instead of ``steps``.

``advect_composite`` couples nested levels the way a composite AMR step does
(:class:`Hierarchy`): before each step the ghost ring of every finer level
takes its coarse parents' values (injection), every level is advanced on its
cells plus that ring, and after the step the coarse cells under a finer level
take the mean of their children (restriction, finest level first).  Each
coupling is a gather over an index table or a block mean over runs of cells
(over a table of cells where runs are short), built once for the fixed geometry
(``sx_index_copy``, ``sx_run_block_mean``, ``sx_index_block_mean``); the backward
pass applies their transposes (``sx_index_segment_add``, ``sx_run_block_mean_adj``,
``sx_index_block_mean_adj``) around the adjoint upwind kernel, in reverse order.

There is no counterpart in the reference, which has no derivatives.
"""

from __future__ import annotations

import gc
from dataclasses import dataclass
from typing import List, Optional, Sequence, Tuple

import torch

from . import _core, _lib
from ._runtime import ptr, stream_handle
from .subsetix_cupy.expressions import IntervalSet, _t

# Block means go by runs of cells from this mean length on, else cell by cell: 1.18 M coarse
# cells in runs of 8, float32, 12.4 us by runs and 8.3 by cells (transposes 18.8 and 14.5), in
# runs of 16 7.1 and 8.3 (10.2 and 12.4), in runs of 2 44 and 8.3 (75 and 16.5).  Few runs are
# quick at any length (20,000 of one cell 3.1 us, by cells 4.2).
_RUN_CELLS = 12
_FEW_RUNS = 30000

_ROWS_UNSAFE = _lib.ROWS_UNSORTED_BEGIN | _lib.ROWS_OVERLAP | _lib.ROWS_EMPTY


@dataclass
class Level:
    """One level's geometry: an interval set in ``[0, width) x [0, height)`` and its cell spacing."""

    interval_set: IntervalSet
    width: int
    height: int
    dx: float
    dy: float

    def __post_init__(self):
        s = self.interval_set
        device = _t(s.row_offsets).device
        self.rows = _t(s.rows)
        self.off = _t(s.row_offsets)
        self.begin = _t(s.begin)
        self.end = _t(s.end)
        self.lookup, bad, flags, self.cell_off, self.cells, columns = _core.stencil_geometry(
            self.rows, self.off, self.begin, self.end, self.height, device)
        if bad:
            raise ValueError("interval_set rows exceed provided height")
        self.direct = not flags & _ROWS_UNSAFE
        self.device = device
        self._chunk_off, self._chunks, self._table = None, 0, None
        self._chunked = False
        self.flat = None
        if self.direct and self.cells > 0 and columns[0] >= 0 and columns[1] <= self.width:
            self.flat = _core.FlatPlan(self.rows, self.off, self.begin, self.end, self.cell_off, self.cells, self.lookup,
                                       self.height, device, columns)
        elif self.direct:  # cells outside the domain: the chunk plan's kernels test every column
            self._chunk_plan()  # built here, so that steps can be captured
        lib = _lib.load()
        nbytes = max(int(lib.sx_upwind_adjoint_scratch_bytes(self.cells)),
                     int(lib.sx_upwind_adjoint_chunked_scratch_bytes((1 << 31) - 1)))
        self.scratch = torch.empty(nbytes, dtype=torch.uint8, device=device)

    def _chunk_plan(self) -> None:
        if not self._chunked and self.direct:
            self._chunk_off, self._chunks = _core.upwind_plan(self.rows, self.off, self.begin, self.end, self.cell_off,
                                                              self.lookup, self.height, self.device)
            self._table = _core.upwind_table(self.begin, self.end, self.cell_off, self._chunk_off, self._chunks,
                                             self.cells, self.device)
        self._chunked = True

    @property
    def chunk_off(self) -> Optional[torch.Tensor]:
        """Chunk plan (built on first use; None when the rows are not sorted and disjoint)."""
        self._chunk_plan()
        return self._chunk_off

    @property
    def chunks(self) -> int:
        self._chunk_plan()
        return self._chunks

    @property
    def table(self) -> Optional[torch.Tensor]:
        """Neighbour table of the chunk plan; None makes the chunked kernels search the neighbour rows."""
        self._chunk_plan()
        return self._table

    @table.setter
    def table(self, value: Optional[torch.Tensor]) -> None:
        self._chunk_plan()
        self._table = value

    def step(self, u: torch.Tensor, out: torch.Tensor, a: float, b: float, dt: float) -> torch.Tensor:
        if self.flat is not None:
            self.flat.step(u, out, a, b, dt, self.dx, self.dy, self.device)
        elif self.chunk_off is not None:
            _core.upwind_chunked(self.off, self.begin, self.end, self.cell_off, self.chunk_off, self.chunks,
                                 self.lookup, u, out, self.width, self.height, a, b, dt, self.dx, self.dy, self.device,
                                 table=self.table)
        else:
            _core.upwind(self.rows, self.off, self.begin, self.end, self.cell_off, self.cells, self.lookup, u, out,
                         self.width, self.height, a, b, dt, self.dx, self.dy, self.direct, self.device)
        return out

    def adjoint_scratch(self) -> Optional[torch.Tensor]:
        """Scratch of :meth:`adjoint` for calls that follow one another on one stream (None: it needs none).

        Its block counter starts at zero and every launch leaves it so, but
        launches that overlap would mix their counts: each pass and each
        captured segment has its own.
        """
        if self.flat is None:
            return None
        return torch.zeros(int(_lib.load().sx_upwind_flat_adjoint_scratch_bytes(self.cells)), dtype=torch.uint8,
                           device=self.device)

    def adjoint(self, w: torch.Tensor, u: torch.Tensor, a: float, b: float, dt: float, grad_ab: torch.Tensor,
                out: Optional[torch.Tensor] = None, scratch: Optional[torch.Tensor] = None) -> torch.Tensor:
        """dL/du for one step (into ``out``), and dL/d(a, b) added into ``grad_ab`` (float64 device pair).

        ``scratch`` is this stream's (:meth:`adjoint_scratch`), made for the call if not given.
        """
        lib = _lib.load()
        ubar = torch.empty_like(w) if out is None else out
        if self.flat is not None:
            scratch = self.adjoint_scratch() if scratch is None else scratch
            self.flat.adjoint(w, u, ubar, a, b, dt, self.dx, self.dy, grad_ab, scratch, self.device)
            return ubar
        g = torch.empty(2, dtype=torch.float64, device=self.device)
        code = _lib.SX_F64 if w.dtype == torch.float64 else _lib.SX_F32
        if self.chunk_off is not None:
            _lib.check(lib.sx_upwind_adjoint_chunked(code, ptr(self.off), ptr(self.begin), ptr(self.end),
                                                     ptr(self.cell_off), ptr(self.chunk_off), self.chunks,
                                                     ptr(self.lookup), ptr(self.table), ptr(w), ptr(u), ptr(ubar),
                                                     self.width,
                                                     self.height, a, b, dt, self.dx, self.dy, ptr(g),
                                                     ptr(self.scratch), int(self.scratch.numel()),
                                                     stream_handle(self.device)), "sx_upwind_adjoint_chunked")
            grad_ab += g
            return ubar
        _lib.check(lib.sx_upwind_adjoint(code, ptr(self.rows), ptr(self.off), int(self.rows.numel()), ptr(self.begin),
                                         ptr(self.end), ptr(self.cell_off), int(self.begin.numel()), self.cells,
                                         ptr(self.lookup), ptr(w), ptr(u), ptr(ubar), self.width, self.height, a, b,
                                         dt, self.dx, self.dy, 1 if self.direct else 0, ptr(g), ptr(self.scratch),
                                         int(self.scratch.numel()), stream_handle(self.device)), "sx_upwind_adjoint")
        grad_ab += g
        return ubar


def _run(levels: Sequence[Level], states: List[torch.Tensor], a: float, b: float, dt: float, n: int,
         keep: bool) -> List[List[torch.Tensor]]:
    """Advance every level ``n`` steps; with ``keep`` return all intermediate inputs per level."""
    trail: List[List[torch.Tensor]] = [[] for _ in levels]
    cur = list(states)
    for _ in range(n):
        for k, lvl in enumerate(levels):
            if keep:
                trail[k].append(cur[k])
            cur[k] = lvl.step(cur[k], torch.empty_like(cur[k]), a, b, dt)
    for k in range(len(levels)):
        trail[k].append(cur[k])
    return trail


class _Advect(torch.autograd.Function):
    @staticmethod
    def forward(ctx, velocity: torch.Tensor, levels, dt: float, steps: int, every: int, *u0):
        a, b = (float(v) for v in velocity.detach().cpu().tolist())
        checkpoints = [list(u.detach() for u in u0)]
        cur = [u.detach().contiguous() for u in u0]
        done = 0
        while done < steps:
            n = min(every, steps - done)
            trail = _run(levels, cur, a, b, dt, n, keep=False)
            cur = [t[-1] for t in trail]
            done += n
            if done < steps:
                checkpoints.append(list(cur))
        ctx.levels, ctx.dt, ctx.steps, ctx.every, ctx.ab = levels, dt, steps, every, (a, b)
        ctx.checkpoints = checkpoints
        ctx.vel_dtype = velocity.dtype
        ctx.vel_device = velocity.device
        return tuple(cur)

    @staticmethod
    def backward(ctx, *grad_out):
        levels, dt, steps, every = ctx.levels, ctx.dt, ctx.steps, ctx.every
        a, b = ctx.ab
        w = [g.contiguous() if g is not None else torch.zeros_like(c) for g, c in zip(grad_out, ctx.checkpoints[0])]
        grad_ab = torch.zeros(2, dtype=torch.float64, device=levels[0].device)
        scratch = [lvl.adjoint_scratch() for lvl in levels]
        seg_starts = list(range(0, steps, every))
        for si in reversed(range(len(seg_starts))):
            n = min(every, steps - seg_starts[si])
            trail = _run(levels, ctx.checkpoints[si], a, b, dt, n, keep=True)  # recompute the segment
            for j in reversed(range(n)):
                for k, lvl in enumerate(levels):
                    w[k] = lvl.adjoint(w[k], trail[k][j], a, b, dt, grad_ab, scratch=scratch[k])
        ctx.checkpoints = None
        grad_v = grad_ab.to(device=ctx.vel_device, dtype=ctx.vel_dtype)
        return (grad_v, None, None, None, None, *w)


def advect(velocity: torch.Tensor, levels: Sequence[Level], u0: Sequence[torch.Tensor], *, dt: float, steps: int,
           checkpoint_every: int = 10) -> Tuple[torch.Tensor, ...]:
    """``steps`` upwind steps of every level; differentiable in ``velocity`` (2 values) and ``u0``."""
    if len(levels) != len(u0):
        raise ValueError("one initial field per level")
    if steps < 0 or checkpoint_every < 1:
        raise ValueError("steps must be >= 0 and checkpoint_every >= 1")
    return _Advect.apply(velocity, tuple(levels), float(dt), int(steps), int(checkpoint_every), *u0)


# ---------------------------------------------------------------------------------------------------------------
# Nested levels coupled by ghost filling and restriction
# ---------------------------------------------------------------------------------------------------------------

def _cells(s: IntervalSet, cell_off: torch.Tensor):
    """(rows, cols) of every cell of ``s`` in value order, as int32 device tensors."""
    b, e, off, rows = _t(s.begin), _t(s.end), _t(s.row_offsets), _t(s.rows)
    n = int(b.numel())
    total = int(cell_off[-1].item()) if n else 0
    dev = off.device
    if total == 0:
        z = torch.zeros(0, dtype=torch.int32, device=dev)
        return z, z.clone()
    iv = torch.repeat_interleave(torch.arange(n, device=dev), (e - b).to(torch.int64))
    x = b[iv] + (torch.arange(total, device=dev, dtype=torch.int32) - cell_off[:-1][iv])
    irow = torch.repeat_interleave(rows, (off[1:] - off[:-1]).to(torch.int64))
    return irow[iv].to(torch.int32), x.to(torch.int32)


def _positions(s: IntervalSet, cell_off: torch.Tensor, rows: torch.Tensor, cols: torch.Tensor) -> torch.Tensor:
    """Value index of each cell (rows, cols) in a field on ``s``; -1 where the cell is not in ``s``."""
    from .subsetix_cupy.interval_field import IntervalField, locate_interval_cells

    if rows.numel() == 0:
        return rows.clone()
    f = IntervalField(interval_set=s, values=torch.empty(0, device=rows.device), interval_cell_offsets=cell_off)
    iv = torch.as_tensor(locate_interval_cells(f, rows, cols)).to(torch.int64)
    found = iv >= 0
    ivc = iv.clamp_min(0)
    pos = cell_off[ivc].to(torch.int64) + (cols.to(torch.int64) - _t(s.begin)[ivc].to(torch.int64))
    return torch.where(found, pos, torch.full_like(pos, -1)).to(torch.int32)


class Hierarchy:
    """Nested interval sets on grids refined by ``ratio`` per level, coupled as a composite AMR step.

    ``sets[k]`` lies in the ``(width * ratio**k) x (height * ratio**k)`` grid
    of level ``k``.  Every finer level needs its ghost ring (the cells next
    to it, left/right/below/above, inside the grid) to have parents in the
    coarser level's set, and every coarse cell under it to have all its
    ``ratio x ratio`` children in it; building a level from the prolongation
    of a coarse set that keeps a one-cell margin satisfies both.  Fields
    given to and returned by :func:`advect_composite` hold the cells of
    ``sets[k]`` in their usual order.
    """

    def __init__(self, sets: Sequence[IntervalSet], width: int, height: int, *, ratio: int = 2,
                 extent: Tuple[float, float] = (1.0, 1.0)):
        from .subsetix_cupy import (clip_interval_set, dilate_interval_set, evaluate, make_input, make_union,
                                    restrict_set)

        if not sets:
            raise ValueError("a hierarchy needs at least one level")
        self.ratio = r = int(ratio)
        if r < 2:
            raise ValueError("levels must be refined by a ratio of at least 2")
        self.levels: List[Level] = []
        self.inner: List[torch.Tensor] = []
        self.inner_cells: List[int] = []
        self.ghost: List[Optional[tuple]] = []
        self.cover: List[Optional[tuple]] = []
        self._segments: dict = {}
        for k, s in enumerate(sets):
            W, H = int(width) * r ** k, int(height) * r ** k
            if k == 0:
                ext = s
            else:
                cross = evaluate(make_union(make_input(dilate_interval_set(s, 1, 0)),
                                            make_input(dilate_interval_set(s, 0, 1))))
                ext = clip_interval_set(cross, width=W, height=H)
            lvl = Level(ext, W, H, extent[0] / W, extent[1] / H)
            self.levels.append(lvl)
            s_off, _ = _core.cell_offsets(_t(s.begin), _t(s.end), lvl.device)
            ys, xs = _cells(s, s_off)
            inner = _positions(ext, lvl.cell_off, ys, xs)
            if bool((inner < 0).any()):
                raise ValueError(f"level {k}: the set is not inside its grid")
            self.inner.append(inner)
            self.inner_cells.append(int(inner.numel()))
            if k == 0:
                self.ghost.append(None)
                self.cover.append(None)
                continue
            prev, prev_set = self.levels[k - 1], sets[k - 1]
            # ghost ring: cells of the extended set outside the set, with their parents on level k-1
            is_inner = torch.zeros(lvl.cells, dtype=torch.bool, device=lvl.device)
            is_inner[inner.to(torch.int64)] = True
            ey, ex = _cells(ext, lvl.cell_off)
            gpos = torch.nonzero(~is_inner).reshape(-1).to(torch.int32)
            py, px = torch.div(ey[gpos.to(torch.int64)], r, rounding_mode="floor"), \
                torch.div(ex[gpos.to(torch.int64)], r, rounding_mode="floor")
            ppos = _positions(prev.interval_set, prev.cell_off, py.to(torch.int32), px.to(torch.int32))
            p_set_off, _ = _core.cell_offsets(_t(prev_set.begin), _t(prev_set.end), lvl.device)
            if bool((ppos < 0).any()) or bool((_positions(prev_set, p_set_off, py.to(torch.int32),
                                                          px.to(torch.int32)) < 0).any()):
                raise ValueError(f"level {k}: its ghost ring is not covered by level {k - 1}")
            order = torch.argsort(ppos.to(torch.int64), stable=True)
            sp = ppos[order]
            uniq, counts = torch.unique_consecutive(sp, return_counts=True)
            seg_off = torch.zeros(uniq.numel() + 1, dtype=torch.int32, device=lvl.device)
            seg_off[1:] = torch.cumsum(counts, 0).to(torch.int32)
            self.ghost.append((gpos.contiguous(), ppos.contiguous(), seg_off, gpos[order].contiguous(),
                               uniq.to(torch.int32).contiguous()))
            # restriction: coarse cells under level k and their r x r children (sub-row outer, column inner)
            covered = restrict_set(s, r)
            c_off, _ = _core.cell_offsets(_t(covered.begin), _t(covered.end), lvl.device)
            cy, cx = _cells(covered, c_off)
            cpos = _positions(prev.interval_set, prev.cell_off, cy, cx)
            dy = torch.arange(r, device=lvl.device).repeat_interleave(r)
            dx = torch.arange(r, device=lvl.device).repeat(r)
            chy = (cy.to(torch.int64)[:, None] * r + dy[None, :]).reshape(-1).to(torch.int32)
            chx = (cx.to(torch.int64)[:, None] * r + dx[None, :]).reshape(-1).to(torch.int32)
            child = _positions(s, s_off, chy, chx)
            if bool((cpos < 0).any()) or bool((child < 0).any()):
                raise ValueError(f"level {k}: a coarse cell under it does not have all its children in it")
            runs = None
            if prev.direct:  # else neighbouring cells need not be neighbouring values
                runs = self._cover_runs(covered, c_off, cpos, child, inner, r)
                if runs[0] > _FEW_RUNS and int(cpos.numel()) < _RUN_CELLS * runs[0]:
                    runs = None
            cells = (cpos.contiguous(), inner[child.to(torch.int64)].contiguous()) if runs is None else None
            self.cover.append((runs, cells))

    @staticmethod
    def _cover_runs(covered: IntervalSet, c_off, cpos, child, inner, r: int) -> tuple:
        """Plan of sx_run_block_mean: ``(runs, ints per run, plan)``, runs of up to 64 cells of one covered interval.

        ``cpos`` and ``child`` are the covered cells' values and their
        children's in the finer set (``inner``: in the finer level).
        """
        size = (c_off[1:] - c_off[:-1]).to(torch.int64)
        per = (size + 63) // 64
        which = torch.repeat_interleave(torch.arange(size.numel(), device=size.device), per)
        nth = torch.arange(which.numel(), device=size.device) - (torch.cumsum(per, 0) - per)[which]
        cell = c_off[:-1].to(torch.int64)[which] + 64 * nth
        plan = torch.zeros((which.numel(), (2 + r + 3) // 4 * 4), dtype=torch.int32, device=size.device)
        plan[:, 0] = cpos[cell]
        plan[:, 1] = torch.clamp(size[which] - 64 * nth, max=64)
        rows = torch.arange(r, device=size.device) * r  # a sub-row's first child among a cell's
        plan[:, 2:2 + r] = inner[child[cell[:, None] * (r * r) + rows].to(torch.int64)]
        return int(plan.shape[0]), int(plan.shape[1]), plan

    # -- the coupled step and its transpose ------------------------------------------------------------------------
    def _fill_ghosts(self, u: List[torch.Tensor]) -> None:
        lib = _lib.load()
        for k in range(1, len(self.levels)):
            gpos, ppos = self.ghost[k][0], self.ghost[k][1]
            _lib.check(lib.sx_index_copy(_code(u[k]), int(gpos.numel()), ptr(gpos), ptr(ppos), ptr(u[k - 1]),
                                         ptr(u[k]), stream_handle(u[k].device)), "sx_index_copy")

    def _restrict(self, u: List[torch.Tensor]) -> None:
        lib = _lib.load()
        r = self.ratio
        for k in range(len(self.levels) - 1, 0, -1):
            runs, cells = self.cover[k]
            code, st = _code(u[k]), stream_handle(u[k].device)
            if runs is not None:
                _lib.check(lib.sx_run_block_mean(code, runs[0], r, runs[1], 1.0 / (r * r), ptr(runs[2]), ptr(u[k]),
                                                 ptr(u[k - 1]), st), "sx_run_block_mean")
            else:
                _lib.check(lib.sx_index_block_mean(code, int(cells[0].numel()), r * r, 1.0 / (r * r), ptr(cells[0]),
                                                   ptr(cells[1]), ptr(u[k]), ptr(u[k - 1]), st), "sx_index_block_mean")

    def step(self, u: List[torch.Tensor], a: float, b: float, dt: float, out: Optional[List[torch.Tensor]] = None
             ) -> Tuple[List[torch.Tensor], List[torch.Tensor]]:
        """One coupled step of the extended-level fields ``u``; returns (new fields, in ``out`` if given, upwind inputs)."""
        self._fill_ghosts(u)
        out = [torch.empty_like(x) for x in u] if out is None else out
        new = [lvl.step(x, y, a, b, dt) for lvl, x, y in zip(self.levels, u, out)]
        self._restrict(new)
        return new, u

    def adjoint_scratch(self) -> List[Optional[torch.Tensor]]:
        """Every level's :meth:`Level.adjoint_scratch`."""
        return [lvl.adjoint_scratch() for lvl in self.levels]

    def step_adjoint(self, w: List[torch.Tensor], inputs: List[torch.Tensor], a: float, b: float, dt: float,
                     grad_ab: torch.Tensor, out: Optional[List[torch.Tensor]] = None,
                     scratch: Optional[List[Optional[torch.Tensor]]] = None) -> List[torch.Tensor]:
        """Transpose of :meth:`step` applied to ``w`` (modified); ``inputs`` are that step's upwind inputs.

        The result is in ``out`` if given (tensors other than ``w``);
        ``scratch`` is this stream's (:meth:`adjoint_scratch`).
        """
        lib = _lib.load()
        r = self.ratio
        for k in range(1, len(self.levels)):
            runs, cells = self.cover[k]
            code, st = _code(w[k]), stream_handle(w[k].device)
            if runs is not None:
                _lib.check(lib.sx_run_block_mean_adj(code, runs[0], r, runs[1], 1.0 / (r * r), ptr(runs[2]),
                                                     ptr(w[k - 1]), ptr(w[k]), st), "sx_run_block_mean_adj")
            else:
                _lib.check(lib.sx_index_block_mean_adj(code, int(cells[0].numel()), r * r, 1.0 / (r * r),
                                                       ptr(cells[0]), ptr(cells[1]), ptr(w[k - 1]), ptr(w[k]), st),
                           "sx_index_block_mean_adj")
        outs = [None] * len(w) if out is None else out
        scratch = [None] * len(w) if scratch is None else scratch
        w = [lvl.adjoint(x, u, a, b, dt, grad_ab, y, z) for lvl, x, u, y, z in zip(self.levels, w, inputs, outs, scratch)]
        for k in range(len(self.levels) - 1, 0, -1):
            _, _, seg_off, src, dst = self.ghost[k]
            _lib.check(lib.sx_index_segment_add(_code(w[k]), int(dst.numel()), ptr(seg_off), ptr(src), ptr(dst),
                                                ptr(w[k]), ptr(w[k - 1]), 1, stream_handle(w[k].device)),
                       "sx_index_segment_add")
        return w

    # -- fields on the sets <-> fields on the extended sets ----------------------------------------------------------
    def extend(self, fields: Sequence[torch.Tensor]) -> List[torch.Tensor]:
        out = []
        lib = _lib.load()
        for lvl, inner, f in zip(self.levels, self.inner, fields):
            x = torch.zeros(lvl.cells, dtype=f.dtype, device=lvl.device)
            f = f.contiguous()
            _lib.check(lib.sx_index_copy(_code(x), int(inner.numel()), ptr(inner), None, ptr(f), ptr(x),
                                         stream_handle(lvl.device)), "sx_index_copy")
            out.append(x)
        return out

    def interior(self, fields: Sequence[torch.Tensor]) -> List[torch.Tensor]:
        out = []
        lib = _lib.load()
        for inner, x in zip(self.inner, fields):
            y = torch.empty(int(inner.numel()), dtype=x.dtype, device=x.device)
            _lib.check(lib.sx_index_copy(_code(x), int(inner.numel()), None, ptr(inner), ptr(x), ptr(y),
                                         stream_handle(x.device)), "sx_index_copy")
            out.append(y)
        return out


def _code(t: torch.Tensor) -> int:
    return _lib.SX_F64 if t.dtype == torch.float64 else _lib.SX_F32


def _run_composite(h: Hierarchy, states: List[torch.Tensor], a: float, b: float, dt: float, n: int, keep: bool):
    """``n`` coupled steps; with ``keep`` also the upwind inputs of every step."""
    inputs = []
    cur = list(states)
    for _ in range(n):
        cur, used = h.step(cur, a, b, dt)
        if keep:
            inputs.append(used)
    return cur, inputs


class _Segment:
    """``n`` coupled steps and their transposes as CUDA graphs on fixed buffers.

    ``forward`` advances ``state`` by ``n`` steps; the backward pass needs
    every step's upwind inputs, which a second graph recomputes from
    ``state`` (all but the last step, whose result nothing reads); the third
    applies the steps' transposes, last step first, to ``w`` and adds each
    step's velocity gradient onto ``grad``.  All work in place, so segment
    follows segment with no copies in between (of 757 us of copies per pass
    over 50 steps on 13.7 M cells, 460 were those).
    Velocity and time step are baked into the graphs.  Every launch of a
    segment becomes one graph replay instead of about seven launches per step
    issued from Python.
    """

    def __init__(self, h: "Hierarchy", n: int, a: float, b: float, dt: float, dtype: torch.dtype):
        dev = h.levels[0].device
        self.state = [torch.zeros(lvl.cells, dtype=dtype, device=dev) for lvl in h.levels]
        self.w = [torch.zeros(lvl.cells, dtype=dtype, device=dev) for lvl in h.levels]
        self.grad = torch.zeros(2, dtype=torch.float64, device=dev)
        self.scratch = h.adjoint_scratch()
        for last in (False, True):
            try:
                self._capture(h, n, a, b, dt)
                break
            except torch.OutOfMemoryError:
                if last:
                    raise
            # A capture allocates from a pool of its own, and memory that the allocator keeps
            # cached elsewhere is not released for it meanwhile: release it and capture again.
            self.fwd = self.keep = self.bwd = self.inputs = None
            torch.cuda.synchronize(dev)
            gc.collect()
            torch.cuda.empty_cache()

    def _capture(self, h: "Hierarchy", n: int, a: float, b: float, dt: float) -> None:
        dev = h.levels[0].device
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        self.fwd, self.keep, self.bwd = (torch.cuda.CUDAGraph() for _ in range(3))

        def settle(result, into):  # a lone step cannot work in place
            if n == 1:
                for dst, src in zip(into, result):
                    dst.copy_(src)

        def forward():
            cur, _ = _run_composite(h, list(self.state), a, b, dt, n - 1, keep=False)
            settle(h.step(cur, a, b, dt, out=self.state if n > 1 else None)[0], self.state)

        def inputs():
            cur, self.inputs = _run_composite(h, list(self.state), a, b, dt, n - 1, keep=True)
            h._fill_ghosts(cur)
            self.inputs.append(cur)

        def backward():
            w = list(self.w)
            for j in reversed(range(n)):
                w = h.step_adjoint(w, self.inputs[j], a, b, dt, self.grad, out=self.w if j == 0 and n > 1 else None,
                                   scratch=self.scratch)
            settle(w, self.w)

        # Captured one after another without torch.cuda.graph's emptying of the allocator's
        # cache before each, which a new hierarchy would pay for.  They share their memory:
        # one replays at a time, and the inputs that outlive their graph are held here.
        with torch.cuda.stream(side):
            for graph, work in ((self.fwd, forward), (self.keep, inputs), (self.bwd, backward)):
                graph.capture_begin(**({} if graph is self.fwd else {"pool": self.fwd.pool()}))
                try:
                    work()
                except BaseException:
                    try:
                        graph.capture_end()
                    except RuntimeError:
                        pass  # the capture is over either way, and the first error is the one to report
                    raise
                graph.capture_end()
        torch.cuda.current_stream(dev).wait_stream(side)

    def forward(self, states: Sequence[torch.Tensor]) -> List[torch.Tensor]:
        """``n`` steps from ``states`` (this segment's own result goes on without a copy)."""
        _load(self.state, states)
        self.fwd.replay()
        return self.state

    def backward(self, states: Sequence[torch.Tensor], w: Sequence[torch.Tensor], grad: torch.Tensor):
        """Transposes of the ``n`` steps from ``states`` applied to ``w``; ``grad`` plus their velocity gradients."""
        _load(self.state, states)
        self.keep.replay()
        _load(self.w, w)
        _load([self.grad], [grad])
        self.bwd.replay()
        return self.w, self.grad


def _load(into: Sequence[torch.Tensor], values: Sequence[torch.Tensor]) -> None:
    for dst, src in zip(into, values):
        if src is not dst:
            dst.copy_(src)


def _segment(h: "Hierarchy", n: int, a: float, b: float, dt: float, dtype: torch.dtype) -> _Segment:
    """Cached segment graphs of ``h`` (the two most recent parameter sets are kept)."""
    key = (n, a, b, dt, dtype)
    cache = h._segments
    seg = cache.pop(key, None)
    if seg is None:
        while len(cache) >= 2:
            cache.pop(next(iter(cache)))
        seg = _Segment(h, n, a, b, dt, dtype)
    cache[key] = seg
    return seg


class _AdvectComposite(torch.autograd.Function):
    @staticmethod
    def forward(ctx, velocity: torch.Tensor, h: Hierarchy, dt: float, steps: int, every: int, graphs: bool, *u0):
        a, b = (float(v) for v in velocity.detach().cpu().tolist())
        cur = h.extend([u.detach() for u in u0])
        # the graphs copy their input; the eager steps fill its ghosts
        checkpoints = [list(cur) if graphs else [x.clone() for x in cur]]
        done = 0
        while done < steps:
            n = min(every, steps - done)
            if graphs:
                cur = _segment(h, n, a, b, dt, cur[0].dtype).forward(cur)
            else:
                cur, _ = _run_composite(h, cur, a, b, dt, n, keep=False)
            done += n
            if done < steps:
                checkpoints.append([x.clone() for x in cur])
        ctx.h, ctx.dt, ctx.steps, ctx.every, ctx.ab, ctx.graphs = h, dt, steps, every, (a, b), graphs
        ctx.checkpoints = checkpoints
        ctx.vel = (velocity.dtype, velocity.device)
        return tuple(h.interior(cur))

    @staticmethod
    def backward(ctx, *grad_out):
        h, dt, steps, every = ctx.h, ctx.dt, ctx.steps, ctx.every
        a, b = ctx.ab
        zeros = [torch.zeros(n, dtype=c.dtype, device=c.device) for n, c in zip(h.inner_cells, ctx.checkpoints[0])]
        w = h.extend([g if g is not None else z for g, z in zip(grad_out, zeros)])
        grad_ab = torch.zeros(2, dtype=torch.float64, device=h.levels[0].device)
        scratch = None if ctx.graphs else h.adjoint_scratch()
        starts = list(range(0, steps, every))
        for si in reversed(range(len(starts))):
            n = min(every, steps - starts[si])
            if ctx.graphs:
                # the graph adds every step's velocity gradient onto the running sum, in the eager order
                w, grad_ab = _segment(h, n, a, b, dt, w[0].dtype).backward(ctx.checkpoints[si], w, grad_ab)
            else:
                _, inputs = _run_composite(h, [x.clone() for x in ctx.checkpoints[si]], a, b, dt, n, keep=True)
                for j in reversed(range(n)):
                    w = h.step_adjoint(w, inputs[j], a, b, dt, grad_ab, scratch=scratch)
        ctx.checkpoints = None
        grads = h.interior(w)
        # a copy: the sum may be a segment's own buffer
        return (grad_ab.to(device=ctx.vel[1], dtype=ctx.vel[0], copy=True), None, None, None, None, None, *grads)


def advect_composite(velocity: torch.Tensor, hierarchy: Hierarchy, u0: Sequence[torch.Tensor], *, dt: float,
                     steps: int, checkpoint_every: int = 10, graphs: bool = True) -> Tuple[torch.Tensor, ...]:
    """``steps`` coupled steps of a :class:`Hierarchy`; differentiable in ``velocity`` (2 values) and ``u0``.

    ``u0[k]`` holds the cells of level ``k``'s set; so does each returned field.
    With ``graphs`` every checkpoint segment runs as a CUDA-graph replay (the
    graphs for a velocity and time step are captured on first use and kept for
    the two most recent ones); without, the same launches are issued one by
    one.  Results are the same either way.
    """
    if len(u0) != len(hierarchy.levels):
        raise ValueError("one initial field per level")
    for k, (u, n) in enumerate(zip(u0, hierarchy.inner_cells)):
        if int(u.numel()) != n:
            raise ValueError(f"level {k}: expected {n} values, got {int(u.numel())}")
    if steps < 0 or checkpoint_every < 1:
        raise ValueError("steps must be >= 0 and checkpoint_every >= 1")
    return _AdvectComposite.apply(velocity, hierarchy, float(dt), int(steps), int(checkpoint_every), bool(graphs),
                                  *u0)


__all__ = ["Level", "advect", "Hierarchy", "advect_composite"]
