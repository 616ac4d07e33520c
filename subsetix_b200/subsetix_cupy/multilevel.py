"""Multilevel sets and fields (drop-in for ``subsetix_cupy.multilevel``).

Names, arguments, checks and exceptions follow ``subsetix_cupy/multilevel.py``
of the reference.  The device work is new:

* ``prolong_set`` writes ``[b*r, e*r)`` on rows ``row*r + d`` directly at
  their final positions (``sx_prolong_set``): no repeat, sort or unique.
* ``restrict_set`` merges the coarsened intervals ``[floor(b/r), ceil(e/r))``
  of the ``r`` sub-rows under every coarse row in one launch for ratios 2 to 4
  (``sx_box_sweep``); other ratios and sparse rows align each group of ``r``
  fine rows onto its coarse row (``sx_align_rows`` with ``div = r``) and take
  one union-mode sweep.
* ``prolong_field`` and ``restrict_field`` run blocks of coarse rows and keep
  the reference's summation order (``sx_prolong_field``,
  ``sx_restrict_field``).  Float64 fields are kept in float64 when
  ``dtype=np.float64`` is requested, an addition of this package.  The
  reference always returns float32.
* Inputs outside the sweeps' contract take the reference's sort-and-merge
  order on the device.
"""

from __future__ import annotations

from dataclasses import dataclass
from typing import List, Optional

import numpy as np
import torch

from .. import _core, _lib
from .._runtime import like
from .expressions import IntervalSet, _t, evaluate, make_difference, make_input
from .interval_field import IntervalField, _is_packed, _offsets_of, _unset_interval_field, create_interval_field, torch_dtype
from .morphology import _box_restrict, _build_interval_set_from_rows, _empty_set, _wrap

I32 = torch.int32
_MAX_SUBROWS = 9  # leaves per union sweep
_REDUCER_CODES = {"mean": 0, "sum": 1, "min": 2, "max": 3}


def _default_ratios(n_levels: int, base: int) -> List[int]:
    """Ratios ``base**k`` of levels ``k = 0 .. n_levels-1`` relative to level 0."""
    if n_levels <= 0:
        raise ValueError(f"a hierarchy needs at least one level, got {n_levels}")
    if base < 2:
        raise ValueError(f"the refinement factor between levels must be at least 2, got {base}")
    return [int(base) ** k for k in range(int(n_levels))]


def _validate_ratios(ratios: List[int]) -> None:
    """Level 0 has ratio 1; each further ratio is a proper multiple of the one before."""
    if not ratios:
        raise ValueError("a hierarchy needs at least one ratio")
    if ratios[0] != 1:
        raise ValueError(f"level 0 must have ratio 1, got {ratios[0]}")
    for k, (lo, hi) in enumerate(zip(ratios, ratios[1:]), start=1):
        if hi <= lo:
            raise ValueError(f"ratio of level {k} ({hi}) does not exceed that of level {k - 1} ({lo})")
        if hi % lo:
            raise ValueError(f"ratio of level {k} ({hi}) is not a multiple of that of level {k - 1} ({lo})")


def _slot(items: list, level: int) -> int:
    """``level`` checked against the number of slots (IndexError outside)."""
    if not 0 <= level < len(items):
        raise IndexError(f"level {level} outside 0..{len(items) - 1}")
    return level


@dataclass
class MultiLevel2D:
    """One optional :class:`IntervalSet` per level, with each level's ratio to level 0 (``multilevel.py:48-87``)."""

    ratios: List[int]
    levels: List[Optional[IntervalSet]]

    @classmethod
    def create(cls, n_levels: int, base_ratio: int = 2) -> "MultiLevel2D":
        ratios = _default_ratios(n_levels, base_ratio)
        return cls(ratios=ratios, levels=[None for _ in ratios])

    @property
    def n_levels(self) -> int:
        return len(self.levels)

    def validate(self) -> None:
        _validate_ratios(self.ratios)
        if len(self.levels) != len(self.ratios):
            raise ValueError(f"{len(self.levels)} levels but {len(self.ratios)} ratios")

    def set_level(self, level: int, interval_set: Optional[IntervalSet]) -> None:
        self.levels[_slot(self.levels, level)] = interval_set

    def get_level(self, level: int) -> Optional[IntervalSet]:
        return self.levels[_slot(self.levels, level)]


@dataclass
class MultiLevelField2D:
    """One optional :class:`IntervalField` per level, on the ratios of a :class:`MultiLevel2D` (``multilevel.py:90-147``)."""

    ratios: List[int]
    fields: List[Optional[IntervalField]]

    @classmethod
    def empty_like(cls, ml: MultiLevel2D) -> "MultiLevelField2D":
        ml.validate()
        return cls(ratios=list(ml.ratios), fields=[None] * ml.n_levels)

    @classmethod
    def create_from_geometry(cls, ml: MultiLevel2D, *, fill_value: float = 0.0, dtype=None) -> "MultiLevelField2D":
        """A field on every level that has a set, filled with ``fill_value``."""
        ml.validate()
        return cls(ratios=list(ml.ratios),
                   fields=[s if s is None else create_interval_field(s, fill_value=fill_value, dtype=dtype)
                           for s in ml.levels])

    def validate_against(self, ml: MultiLevel2D) -> None:
        """Same ratios as ``ml``, and every field's row and interval counts equal to its level's set."""
        ml.validate()
        if len(self.fields) != ml.n_levels:
            raise ValueError(f"{len(self.fields)} field levels for {ml.n_levels} geometry levels")
        if list(self.ratios) != list(ml.ratios):
            raise ValueError(f"field ratios {list(self.ratios)} differ from geometry ratios {list(ml.ratios)}")
        for k, (f, s) in enumerate(zip(self.fields, ml.levels)):
            if f is None or s is None:
                continue
            fs = f.interval_set
            if (int(fs.row_offsets.shape[0]), int(fs.begin.shape[0])) != (int(s.row_offsets.shape[0]),
                                                                         int(s.begin.shape[0])):
                raise ValueError(f"level {k}: the field's rows or intervals differ from the level's set")

    def set_level_field(self, level: int, field: Optional[IntervalField]) -> None:
        self.fields[_slot(self.fields, level)] = field

    def get_level_field(self, level: int) -> Optional[IntervalField]:
        return self.fields[_slot(self.fields, level)]


# ---------------------------------------------------------------------------
# Sets
# ---------------------------------------------------------------------------

def _prolong_set_impl(interval_set: IntervalSet, ratio: int, cells: bool = False):
    """``[b*r, e*r)`` on rows ``row*r + 0..r-1`` of every occupied row (``multilevel.py:213-264``).

    With ``cells`` returns ``(set, cell offsets, cells, rising)``; rising: no
    row's begins fall, so fine interval ``o`` of a row is its coarse interval ``o``.
    """
    if ratio < 1:
        raise ValueError("ratio must be >= 1")
    s = interval_set
    r = int(ratio)
    device = _t(s.row_offsets).device
    R = s.row_count
    n = int(s.begin.shape[0])
    if r == 1 or R == 0 or n == 0:
        if r == 1:
            out = s
        else:
            if R > 0:
                rows_out = (_t(s.rows)[:, None] * r + torch.arange(r, dtype=I32, device=device)[None, :]).reshape(-1)
            else:
                rows_out = torch.zeros(0, dtype=I32, device=device)
            out = _empty_set(device, rows_out.to(I32), s.begin)
        return (out, *_offsets_of(out)[:2], False) if cells else out
    rows_out, off, ob, oe, unsorted, *more = _core.prolong_set(_t(s.rows), _t(s.row_offsets), _t(s.begin), _t(s.end), r,
                                                               device, cells=cells)
    if unsorted:
        # The reference sorts each output row by begin (a stable lexsort);
        # rows whose begins decrease need the same stable order here.
        per = torch.repeat_interleave(torch.arange(int(rows_out.numel()), device=device),
                                      (off[1:] - off[:-1]).to(torch.int64), output_size=int(ob.numel()))
        key = (per.to(torch.int64) << 32) | (ob.to(torch.int64) + (1 << 31))
        order = torch.sort(key, stable=True).indices
        ob, oe = ob[order], oe[order]
        if cells:
            more = _core.cell_offsets(ob, oe, device)
    out = _wrap(s.begin, ob, oe, off, rows_out)
    return (out, *more, not unsorted) if cells else out


def prolong_set(interval_set: IntervalSet, ratio: int) -> IntervalSet:
    """Refine by ``ratio``; ``ratio == 1`` returns the input object (``multilevel.py:267-269``)."""
    return _prolong_set_impl(interval_set, ratio)


def _restrict_reference_order(s: IntervalSet, r: int) -> IntervalSet:
    """Coarsen, sort and merge as the reference does (``multilevel.py:272-362``)."""
    per = _t(s.interval_rows())
    b, e = _t(s.begin), _t(s.end)
    crows = torch.div(per, r, rounding_mode="floor").to(I32)
    cb = torch.div(b, r, rounding_mode="floor").to(I32)
    ce = torch.div(e + (r - 1), r, rounding_mode="floor").to(I32)
    mask = ce > cb
    if not bool(mask.any()):
        return _empty_set(b.device, torch.unique(crows).to(I32), s.begin)
    return _build_interval_set_from_rows(crows[mask], cb[mask], ce[mask], kind=s.begin)


def restrict_set(interval_set: IntervalSet, ratio: int) -> IntervalSet:
    """Coarsen by ``ratio`` with floor/ceil bounds and merge (``multilevel.py:272-362``)."""
    if ratio < 1:
        raise ValueError("ratio must be >= 1")
    s = interval_set
    r = int(ratio)
    device = _t(s.row_offsets).device
    R = s.row_count
    if R == 0:
        return _empty_set(device, None, s.begin)
    if int(s.begin.shape[0]) == 0:
        return _empty_set(device, torch.unique(torch.div(_t(s.rows), r, rounding_mode="floor")).to(I32), s.begin)
    out = _box_restrict(s, r)
    if out is not None:
        return out
    if r > _MAX_SUBROWS:
        return _restrict_reference_order(s, r)
    rows, off = _t(s.rows), _t(s.row_offsets)
    host = torch.cat([rows[0:1], rows[-1:]]).cpu()
    lo = int(host[0]) // r
    hi = int(host[1]) // r
    lists = [(rows, off, 0, True, r, phase) for phase in range(r)]
    rows_out, starts, stops = _core.align_rows(lists, lo, hi, device, [True] * r, want_ends=[True] * r)
    R_out = int(rows_out.numel())
    b, e = _t(s.begin), _t(s.end)
    leaves = [(b, e, starts[p], 0, r, stops[p]) for p in range(r)]
    ob, oe, ooff, total, flags = _core.bool_eval(leaves, R_out, [0] * 8, _lib.MODE_UNION, device)
    if flags & _lib.FLAG_CONTRACT:
        return _restrict_reference_order(s, r)
    if flags & (_lib.FLAG_CAPACITY | _lib.FLAG_TIMEOUT):
        raise _lib.SubsetixError(f"restriction sweep failed (flags={flags})")
    return _wrap(s.begin, ob[:total].clone(), oe[:total].clone(), ooff, rows_out)


def _parts(s: IntervalSet) -> tuple:
    return _t(s.rows), _t(s.row_offsets), _t(s.begin), _t(s.end)


def _raise_misaligned(flags: int) -> None:
    """The reference's alignment errors, in its order (``multilevel.py:169-210,433-451``)."""
    if flags & 1:
        raise ValueError("fine set row count does not match coarse x ratio")
    if flags & 2:
        raise ValueError("fine set rows do not align with refinement ratio")
    if flags & 8:
        raise ValueError("fine field is not aligned with coarse geometry for restriction")


# ---------------------------------------------------------------------------
# Fields
# ---------------------------------------------------------------------------

def _value_dtype(dtype) -> torch.dtype:
    if dtype is None:
        return torch.float32
    t = torch_dtype(dtype)
    if t not in (torch.float32, torch.float64):
        raise TypeError("multilevel fields support float32 and float64")
    return t


def prolong_field(field: IntervalField, ratio: int, *, dtype=None) -> IntervalField:
    """Piecewise-constant injection onto ``prolong_set`` (``multilevel.py:365-407``).

    The result is float32 like the reference's; ``dtype=np.float64`` keeps
    double precision.
    """
    if ratio < 1:
        raise ValueError("ratio must be >= 1")
    out_t = _value_dtype(dtype)
    coarse = field.interval_set
    fine_set, fine_off, total, rising = _prolong_set_impl(coarse, ratio, cells=True)
    fine_field = _unset_interval_field(fine_set, out_t, fine_off, total)
    fv = _t(fine_field.values)
    cv = _t(field.values)
    if fv.numel() == 0:
        return fine_field
    if cv.numel() == 0:
        fv.zero_()
        return fine_field
    if ratio == 1:
        fv.copy_(cv.to(out_t))
        return fine_field
    n = int(coarse.begin.shape[0])
    if n == 0:
        fv.zero_()
        return fine_field
    device = fv.device
    # The reference's mapping check (multilevel.py:184-205) fails exactly
    # when a coarse row is empty: prolong_set then drops its r fine rows.
    # When the counts agree, the fine rows are coarse_row*r + d by construction.
    if int(fine_set.rows.shape[0]) != coarse.row_count * int(ratio):
        raise ValueError("fine set row count does not match coarse x ratio")
    if not (rising and _is_packed(field)):
        fv.zero_()  # fine intervals re-sorted within a row, or offsets of unknown origin: some cells may stay unwritten
    _core.prolong_field(_t(coarse.row_offsets), _t(field.interval_cell_offsets), n, _t(fine_set.row_offsets),
                        _t(fine_field.interval_cell_offsets), int(ratio), cv.to(out_t).contiguous(), fv, device)
    return fine_field


def restrict_field(field: IntervalField, ratio: int, *, reducer: str = "mean", dtype=None) -> IntervalField:
    """``ratio`` x ``ratio`` block reduction onto ``restrict_set`` (``multilevel.py:410-479``).

    ``mean`` is ``(sum over sub-rows, then columns) * (1 / r^2)`` as in the
    reference; also ``sum``, ``min``, ``max``.  Float32 unless
    ``dtype=np.float64``.
    """
    out_t = _value_dtype(dtype)
    fine_set = field.interval_set
    coarse_set = restrict_set(fine_set, ratio)
    r, n = int(ratio), int(coarse_set.begin.shape[0])
    device = _t(coarse_set.row_offsets).device
    check = 0
    if n and r > 1:  # the cell total and the alignment check come back in one read
        res = _core.empty_i32(3, device)
        off, _ = _core.cell_offsets(_t(coarse_set.begin), _t(coarse_set.end), device, sync=False, result=res)
        _core.coarse_fine_check(_parts(coarse_set), _parts(fine_set), r, device, flags=res[2:])
        total, scan_flags, check = res.tolist()
        _core.check_scan(scan_flags, "sx_cell_offsets")
        coarse_field = _unset_interval_field(coarse_set, out_t, off, total)
    else:
        coarse_field = _unset_interval_field(coarse_set, out_t)
    fv = _t(field.values)
    cv = _t(coarse_field.values)
    if cv.numel() == 0:
        return coarse_field
    if fv.numel() == 0:
        cv.zero_()
        return coarse_field
    if r <= 0:
        raise ValueError("ratio must be >= 1")
    if r == 1:
        # multilevel.py:421-423 names an undefined variable here
        raise NameError("name 'target_dtype' is not defined")
    code = _REDUCER_CODES.get(reducer)
    if code is None:
        raise ValueError(f"unsupported reducer '{reducer}'")
    _raise_misaligned(check)
    _core.restrict_field(_t(coarse_set.row_offsets), _t(coarse_field.interval_cell_offsets), n,
                         _t(fine_set.row_offsets), _t(field.interval_cell_offsets), r, code,
                         fv.to(out_t).contiguous(), cv, device)
    return coarse_field


# ---------------------------------------------------------------------------
# Level helpers
# ---------------------------------------------------------------------------

def _pair_ratio(ml: MultiLevel2D, level: int, what: str) -> int:
    """Ratio between ``level`` and ``level + 1`` of a valid hierarchy; IndexError when that pair does not exist."""
    ml.validate()
    if not 0 <= level < ml.n_levels - 1:
        raise IndexError(f"{what}: no level pair {level}/{level + 1} in {ml.n_levels} levels")
    return ml.ratios[level + 1] // ml.ratios[level]


def _defined(x, what: str):
    if x is None:
        raise ValueError(f"{what} is not defined")
    return x


def prolong_level_sets(ml: MultiLevel2D, level: int) -> IntervalSet:
    """Set of ``level + 1`` := prolongation of the set of ``level`` (``multilevel.py:482-492``)."""
    r = _pair_ratio(ml, level, "prolongation")
    ml.set_level(level + 1, prolong_set(_defined(ml.get_level(level), "base level interval set"), r))
    return ml.get_level(level + 1)


def restrict_level_sets(ml: MultiLevel2D, level: int) -> IntervalSet:
    """Set of ``level`` := restriction of the set of ``level + 1`` (``multilevel.py:495-505``)."""
    r = _pair_ratio(ml, level, "restriction")
    ml.set_level(level, restrict_set(_defined(ml.get_level(level + 1), "fine level interval set"), r))
    return ml.get_level(level)


def prolong_level_field(ml: MultiLevel2D, mf: MultiLevelField2D, level: int) -> IntervalField:
    """Field of ``level + 1`` := injection of the field of ``level`` (``multilevel.py:508-519``)."""
    mf.validate_against(ml)
    r = _pair_ratio(ml, level, "prolongation")
    mf.set_level_field(level + 1, prolong_field(_defined(mf.get_level_field(level), "base level field"), r))
    return mf.get_level_field(level + 1)


def restrict_level_field(ml: MultiLevel2D, mf: MultiLevelField2D, level: int, *, reducer: str = "mean"
                         ) -> IntervalField:
    """Field of ``level`` := ``reducer`` over the blocks of the field of ``level + 1`` (``multilevel.py:522-533``)."""
    mf.validate_against(ml)
    r = _pair_ratio(ml, level, "restriction")
    fine = _defined(mf.get_level_field(level + 1), "fine level field")
    mf.set_level_field(level, restrict_field(fine, r, reducer=reducer))
    return mf.get_level_field(level)


def covered_by_fine(ml: MultiLevel2D, level: int):
    """Cells of ``level`` under the set of ``level + 1`` (its restriction), or None when that set is unset."""
    r = _pair_ratio(ml, level, "covered_by_fine")
    fine = ml.get_level(level + 1)
    return None if fine is None else restrict_set(fine, r)


def coarse_only(coarse_set: IntervalSet, ml: MultiLevel2D, level: int):
    """``coarse_set`` minus the cells covered by ``level + 1`` (``coarse_set`` itself when nothing covers it)."""
    covered = covered_by_fine(ml, level)
    if covered is None or coarse_set is None:
        return coarse_set
    return evaluate(make_difference(make_input(coarse_set), make_input(covered)))


__all__ = [
    "MultiLevel2D",
    "MultiLevelField2D",
    "prolong_set",
    "restrict_set",
    "prolong_field",
    "restrict_field",
    "prolong_level_sets",
    "restrict_level_sets",
    "prolong_level_field",
    "restrict_level_field",
    "covered_by_fine",
    "coarse_only",
]
