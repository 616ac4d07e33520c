"""Fused, batched, graph-replayed two-level AMR advection on full grids.

``AMR2Simulation`` (``subsetix_amr2/simulation.py`` of the reference) keeps
both levels as full rectangles and runs, per step,

    synchronize; regrid every k steps; upwind on both levels; synchronize.

On full rectangles every interval kernel of that loop is a dense one, so
``FusedTwoLevelAMR`` runs the same loop on ``[batch, rows, cols]`` arrays
with ``sx_upwind_full`` (both levels), ``sx_amr_sync_full`` (restriction
into refined coarse cells and prolongation into the rest, in one pass) and
``sx_amr_regrid_full`` (gradient tag and grading into action bytes).  For
ratio 2 the upwind of both levels and the synchronisation run as one kernel
per step (``sx_amr_step_full``, ``fused=True``), and steps with no regrid
between them as one kernel for up to five (``sx_amr_steps_full``).  The results are bit-identical to ``AMR2Simulation`` on the same
initial field, in float32 and in float64.  The first synchronisation of a
step always follows the previous step's last one with nothing in between,
so it recomputes identical values and is skipped.

A regrid period is a fixed sequence of launches on fixed buffers, so it is
captured once per buffer parity into a CUDA graph and replayed with no host
synchronisation; so is a single step, with a regrid or without.  The interval sets of the geometry
(refine, fine, coarse-only) are rebuilt on request from the action bytes,
which give the same sets as the reference's interval pipeline.

Compensated float64 mass integrals (``sx_mass_integral``) and the
conservation defect of the restriction report the accuracy of float32
storage against float64.
"""

from __future__ import annotations

from typing import Optional, Sequence

import numpy as np
import torch

from .. import _core, _lib
from .._runtime import ptr, stream_handle

_MODES = {"von_neumann": 0, "moore": 1}


def _check(rc: int, what: str) -> None:
    _lib.check(rc, what)


class FusedTwoLevelAMR:
    """Batched two-level advection with the reference's step order (``simulation.py:232-354``).

    ``coarse0`` is ``[rows, cols]`` or ``[batch, rows, cols]`` (square
    grids, as in AMR2Simulation).  ``dtype`` is torch.float32 or
    torch.float64.
    """

    def __init__(self, coarse0: torch.Tensor, *, velocity: Sequence[float], cfl: float = 0.9,
                 refine_threshold: float = 0.05, grading: int = 1, grading_mode: str = "von_neumann", ratio: int = 2,
                 dtype: torch.dtype = torch.float32, epsilon: float = 1e-8, fused: bool = True):
        if dtype not in (torch.float32, torch.float64):
            raise TypeError("dtype must be torch.float32 or torch.float64")
        if grading_mode not in _MODES:
            raise ValueError("grading_mode must be 'von_neumann' or 'moore'")
        if refine_threshold <= 0.0:
            raise ValueError("refine_threshold must be > 0")
        if ratio < 1:
            raise ValueError("ratio must be >= 1")
        c0 = coarse0 if coarse0.dim() == 3 else coarse0.unsqueeze(0)
        if not c0.is_cuda:
            raise ValueError("coarse0 must be a CUDA tensor")
        self.batch, self.height, self.width = (int(s) for s in c0.shape)
        if self.height != self.width:
            raise ValueError("AMR2Simulation grids are square")
        self.device = c0.device
        self.dtype = dtype
        self.fused = bool(fused) and int(ratio) == 2
        self.code = _lib.SX_F64 if dtype == torch.float64 else _lib.SX_F32
        self.ratio = int(ratio)
        self.velocity = (float(velocity[0]), float(velocity[1]))
        self.threshold = float(np.float32(max(float(refine_threshold), float(epsilon))))
        self.grading = int(grading)
        self.mode = _MODES[grading_mode]
        self.dx_coarse = 1.0 / self.width
        self.dy_coarse = 1.0 / self.height
        self.dx_fine = self.dx_coarse / self.ratio
        self.dy_fine = self.dy_coarse / self.ratio
        denom = abs(self.velocity[0]) / self.dx_fine + abs(self.velocity[1]) / self.dy_fine
        self.dt = cfl / denom if denom > 0 else 0.0
        B, H, W, r = self.batch, self.height, self.width, self.ratio
        self.coarse = [c0.to(dtype).contiguous().clone(), torch.empty((B, H, W), dtype=dtype, device=self.device)]
        self.fine = [torch.empty((B, H * r, W * r), dtype=dtype, device=self.device) for _ in range(2)]
        self.actions = torch.zeros((B, H, W), dtype=torch.int8, device=self.device)
        self.tags = torch.empty((B, H, W), dtype=torch.uint8, device=self.device)
        self.cur = 0
        self.step_count = 0
        self.time = 0.0
        self._synced = False
        self._graphs = {}
        self._flips = {}  # regrid period -> whether its graph ends in the other pair of buffers
        # set_initial_field: actions from the initial gradient, then fine = prolong(coarse)
        self._regrid()
        keep = torch.zeros_like(self.actions)
        self._sync(keep)

    # ------------------------------------------------------------------ kernels
    def _stream(self) -> int:
        return stream_handle(self.device)

    def _regrid(self) -> None:
        lib = _lib.load()
        _check(lib.sx_amr_regrid_full(self.code, ptr(self.coarse[self.cur]), ptr(self.tags), ptr(self.actions),
                                      self.width, self.height, self.batch, self.threshold, self.grading, self.mode,
                                      self._stream()), "sx_amr_regrid_full")

    def _sync(self, actions: Optional[torch.Tensor] = None) -> None:
        lib = _lib.load()
        act = self.actions if actions is None else actions
        _check(lib.sx_amr_sync_full(self.code, ptr(self.coarse[self.cur]), ptr(self.fine[self.cur]), ptr(act),
                                    self.width, self.height, self.batch, self.ratio, self._stream()),
               "sx_amr_sync_full")

    def _advance(self) -> None:
        lib = _lib.load()
        a, b = self.velocity
        s = self._stream()
        nxt = 1 - self.cur
        _check(lib.sx_upwind_full(self.code, ptr(self.coarse[self.cur]), ptr(self.coarse[nxt]), self.width,
                                  self.height, self.batch, a, b, self.dt, self.dx_coarse, self.dy_coarse, s),
               "sx_upwind_full")
        _check(lib.sx_upwind_full(self.code, ptr(self.fine[self.cur]), ptr(self.fine[nxt]), self.width * self.ratio,
                                  self.height * self.ratio, self.batch, a, b, self.dt, self.dx_fine, self.dy_fine, s),
               "sx_upwind_full")
        self.cur = nxt

    def _fused_advance_sync(self) -> None:
        lib = _lib.load()
        a, b = self.velocity
        nxt = 1 - self.cur
        _check(lib.sx_amr_step_full(self.code, ptr(self.coarse[self.cur]), ptr(self.fine[self.cur]),
                                    ptr(self.coarse[nxt]), ptr(self.fine[nxt]), ptr(self.actions), self.width,
                                    self.height, self.batch, a, b, self.dt, self.dx_coarse, self.dy_coarse,
                                    self.dx_fine, self.dy_fine, self._stream()), "sx_amr_step_full")
        self.cur = nxt

    def _fused_steps(self, n: int) -> None:
        """``n`` steps on fixed actions, in as few launches as they allow, of nearly equal step counts."""
        lib = _lib.load()
        a, b = self.velocity
        launches = -(-n // _lib.AMR_MAX_STEPS)
        for i in range(launches):
            steps = n * (i + 1) // launches - n * i // launches
            if steps == 1:
                self._fused_advance_sync()
                continue
            nxt = 1 - self.cur
            _check(lib.sx_amr_steps_full(self.code, ptr(self.coarse[self.cur]), ptr(self.fine[self.cur]),
                                         ptr(self.coarse[nxt]), ptr(self.fine[nxt]), ptr(self.actions), self.width,
                                         self.height, self.batch, steps, a, b, self.dt, self.dx_coarse, self.dy_coarse,
                                         self.dx_fine, self.dy_fine, self._stream()), "sx_amr_steps_full")
            self.cur = nxt

    def _step_body(self, regrid: bool, n: int = 1) -> None:
        """``n`` steps, after a regrid when asked."""
        if regrid:
            self._regrid()
        if self.fused:
            self._fused_steps(n)
            return
        for _ in range(n):
            self._advance()
            self._sync()

    # ------------------------------------------------------------------ public
    def step(self, regrid_every: int = 1) -> None:
        """One step: synchronize; regrid when due; upwind both levels; synchronize."""
        if not self._synced:
            self._sync()
            self._synced = True
        self._step_body(self.step_count % max(1, int(regrid_every)) == 0)
        self.step_count += 1
        self.time += self.dt

    def _graph(self, regrid: bool, parity: int) -> torch.cuda.CUDAGraph:
        key = (regrid, parity)
        g = self._graphs.get(key)
        if g is None:
            saved = self.cur
            self.cur = parity
            s = torch.cuda.Stream(device=self.device)
            s.wait_stream(torch.cuda.current_stream(self.device))
            g = torch.cuda.CUDAGraph()
            with torch.cuda.stream(s):
                with torch.cuda.graph(g, stream=s):
                    self._step_body(regrid)
            torch.cuda.current_stream(self.device).wait_stream(s)
            self.cur = saved
            self._graphs[key] = g
        return g

    def _period_graph(self, period: int, parity: int) -> torch.cuda.CUDAGraph:
        """One graph for a whole regrid period: the regrid and ``period`` steps, from ping-pong side ``parity``."""
        key = ("period", period, parity)
        g = self._graphs.get(key)
        if g is None:
            saved = self.cur
            self.cur = parity
            s = torch.cuda.Stream(device=self.device)
            s.wait_stream(torch.cuda.current_stream(self.device))
            g = torch.cuda.CUDAGraph()
            with torch.cuda.stream(s):
                with torch.cuda.graph(g, stream=s):
                    self._step_body(True, period)
            torch.cuda.current_stream(self.device).wait_stream(s)
            self._flips[period] = self.cur ^ parity
            self.cur = saved
            self._graphs[key] = g
        return g

    def run(self, steps: int, regrid_every: int = 1, graph: bool = True) -> None:
        """Advance ``steps`` steps.

        With ``graph``, every whole regrid period (the regrid and its
        ``regrid_every`` steps) and every single step is one CUDA-graph
        replay; steps outside whole periods are launched as they come when
        one kernel takes several.  The launches, and so the results, are the
        same as without graphs.
        """
        period = max(1, int(regrid_every))
        if not self._synced:
            self._sync()
            self._synced = True
        left = int(steps)
        while left > 0:
            if graph and period > 1 and self.step_count % period == 0 and left >= period:
                self._period_graph(period, self.cur).replay()
                self.cur ^= self._flips[period]
                n = period
            else:
                regrid = self.step_count % period == 0
                n = min(left, period - self.step_count % period) if self.fused else 1
                if graph and n == 1:
                    self._graph(regrid, self.cur).replay()
                    self.cur = 1 - self.cur
                else:
                    self._step_body(regrid, n)
            for _ in range(n):
                self.step_count += 1
                self.time += self.dt
            left -= n

    def prepare_graphs(self, regrid_every: Optional[int] = None) -> None:
        """Capture the step graphs ahead of time (no work is done): the four
        single-step graphs and, given ``regrid_every``, the two whole-period graphs."""
        for regrid in (False, True):
            for parity in (0, 1):
                self._graph(regrid, parity)
        period = max(1, int(regrid_every or 1))
        if period > 1:
            for parity in (0, 1):
                self._period_graph(period, parity)

    # ---------------------------------------------------------------- results
    @property
    def coarse_values(self) -> torch.Tensor:
        return self.coarse[self.cur]

    @property
    def fine_values(self) -> torch.Tensor:
        return self.fine[self.cur]

    def refine_set(self, index: int = 0):
        """Refine region of batch entry ``index`` as an IntervalSet (as ``ActionField.refine_set``)."""
        from ..subsetix_cupy import create_interval_field, full_interval_set
        from .fields import _interval_field_value_intervals

        dom = full_interval_set(self.width, self.height)
        f = create_interval_field(dom, fill_value=0, dtype=np.int8)
        f.values.copy_(self.actions[index].reshape(-1))
        return _interval_field_value_intervals(f, 1)

    def mass(self, out: Optional[torch.Tensor] = None) -> torch.Tensor:
        """Compensated float64 integral of u over the domain, per batch entry (device tensor).

        After a synchronisation the refined coarse cells hold the mean of
        their fine blocks, so the coarse level carries the composite mass.
        """
        out = torch.empty(self.batch, dtype=torch.float64, device=self.device) if out is None else out
        area = self.dx_coarse * self.dy_coarse
        for b in range(self.batch):
            _core.mass_integral(self.coarse[self.cur][b].reshape(-1), area, self.device, out=out[b:b + 1])
        return out

    def restriction_defect(self) -> torch.Tensor:
        """Float64 mass of (coarse cell - fine block mean) over refined cells, per batch entry.

        Zero up to the rounding of the restriction; the compensated sums make
        the float32 rounding visible instead of hiding it under summation
        error.
        """
        r = self.ratio
        c = self.coarse[self.cur].to(torch.float64)
        f = self.fine[self.cur].to(torch.float64)
        B, H, W = c.shape
        block = f.reshape(B, H, r, W, r).sum(dim=(2, 4)) / (r * r)
        d = torch.where(self.actions != 0, c - block, torch.zeros_like(c))
        out = torch.empty(B, dtype=torch.float64, device=self.device)
        area = self.dx_coarse * self.dy_coarse
        for b in range(B):
            _core.mass_integral(d[b].reshape(-1).contiguous(), area, self.device, out=out[b:b + 1])
        return out


__all__ = ["FusedTwoLevelAMR"]
