"""Work that a user of subsetix_b200 has it do, as measurable cases over its public entry points.

Each case is one kind of call at one size.  ``listed()`` names the
representative ones, ``draw(rng)`` gives another case from the same ranges,
``prepare`` makes what a program holds before the call (inputs from the seed,
plans, hierarchies, engines), ``run`` is one pass, ``work`` the bytes and
operations that pass cannot do without, and ``exact`` the floating results in
float64 from plain torch.

Kinds:

* ``expr``       a fused set expression ``((A | B) - (C & D)) ^ E`` through
                 ``evaluate``, over random rows or over the round shapes and
                 checkerboards, stacked as copies on row bands
* ``batch_sets`` union and intersection of many uneven sets, one call each
* ``morph``      dilation, erosion or ghost zones of a set
* ``fields``     prolongation and restriction of an interval field
* ``sync``       two-level synchronisation of interval fields
* ``upwind``     one upwind step of an interval field
* ``upwind_batch`` one upwind step of many uneven sets, each with its spacing
* ``regrid``     gradient tagging and 2:1 grading of a whole-grid field
* ``amr``        steps of the two-level advection driver
* ``adjoint``    composite multi-level advection and its gradients

A case's ``geometry`` seeds the base geometry; the seed of ``prepare`` places
it (mirrored, flipped, shifted, rows rotated) and draws the field values, so
that results of one case have one size.
"""

import math
import random

import numpy as np
import torch

from subsetix_b200.adjoint import Hierarchy, advect_composite
from subsetix_b200.batch import SetBatch, batched_binary, batched_upwind
from subsetix_b200.subsetix_amr2 import (
    AMR2Simulation,
    SimulationConfig,
    enforce_two_level_grading_set,
    gradient_tag_set,
    synchronize_interval_fields,
)
from subsetix_b200.subsetix_amr2.fields import ActionField
from subsetix_b200.subsetix_amr2.regrid import (
    gradient_magnitude_interval_field,
    gradient_tag_threshold_interval_field,
)
from subsetix_b200.subsetix_cupy import (
    build_interval_set,
    create_interval_field,
    dilate_interval_set,
    erode_interval_set,
    evaluate,
    full_interval_set,
    ghost_zones,
    make_difference,
    make_input,
    make_intersection,
    make_symmetric_difference,
    make_union,
    prolong_field,
    prolong_set,
    restrict_field,
    step_upwind_interval,
)

_DEVICE = "cuda"
_DTYPES = {"f32": torch.float32, "f64": torch.float64}
_NUMPY = {"f32": np.float32, "f64": np.float64}
_SIDE_LO, _SIDE_HI = 128, 4096  # sides of the uneven sets of a batch


def listed():
    return [
        # Set algebra on one small grid (256 rows, about four intervals in each): a call in an interactive or
        # per-step host loop, where latency is what the user waits for.
        {"name": "expr_rows_256", "kind": "expr", "shapes": False, "size": 256, "copies": 1, "geometry": 1},
        # The headline workload: the five-leaf expression over 128 stacked copies of the 4096^2 shapes.
        {"name": "expr_shapes_4096x128", "kind": "expr", "shapes": True, "size": 4096, "copies": 128, "geometry": 1},
        # 256 uneven sets (sides 128 to 4096, lognormal interval counts, so skewed rows): union and intersection.
        {"name": "batch_sets_256", "kind": "batch_sets", "count": 256, "geometry": 1},
        # Halo of a many-interval geometry: 200 circles with a 64-pixel checkerboard, eight stacked 4096^2 copies.
        {"name": "dilate_4096x8", "kind": "morph", "op": "dilate", "size": 4096, "copies": 8, "hx": 1, "hy": 1,
         "geometry": 1},
        # Erosion of one geometry on an odd grid by an uneven box: a chain of clips, differences and one dilation.
        {"name": "erode_3001", "kind": "morph", "op": "erode", "size": 3001, "copies": 1, "hx": 2, "hy": 3,
         "geometry": 1},
        # Level transfer of a field on a 4096^2 geometry (about half of its cells): ratio 2, mean, float32.
        {"name": "fields_4096_f32", "kind": "fields", "size": 4096, "ratio": 2, "reducer": "mean", "dtype": "f32",
         "geometry": 1},
        # Two-level synchronisation of interval fields with partial refinement, odd size, float64.
        {"name": "sync_1001_f64", "kind": "sync", "size": 1001, "dtype": "f64"},
        # One upwind step of a float64 field on a ragged geometry of ordinary size, velocity against both axes.
        {"name": "upwind_2500_f64", "kind": "upwind", "size": 2500, "dtype": "f64", "a": -0.7, "b": 0.4,
         "geometry": 1},
        # One float32 upwind step of 256 uneven sets (about 240 M cells), each set with its own spacing and time step.
        {"name": "upwind_batch_256_f32", "kind": "upwind_batch", "count": 256, "dtype": "f32", "a": 1.0, "b": 0.5,
         "geometry": 1},
        # Regrid of a large whole-grid field: gradient tags and von Neumann 2:1 grading as interval sets.
        {"name": "regrid_4096", "kind": "regrid", "size": 4096, "tag": "threshold", "padding": 1,
         "mode": "von_neumann", "geometry": 1},
        # The two-level advection driver on the 1024^2 blob: two regrid periods of ten float32 steps.
        {"name": "amr_1024_f32", "kind": "amr", "size": 1024, "steps": 20, "every": 10, "dtype": "f32"},
        # Gradient of a three-level composite advection (base 2048^2, 50 float32 steps, checkpoints every 10).
        {"name": "adjoint_2048_f32", "kind": "adjoint", "base": 2048, "steps": 50, "every": 10, "dtype": "f32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    geometry = rng.randrange(1000)
    kind = rng.choice(["expr", "expr", "batch_sets", "morph", "morph", "fields", "sync", "upwind", "upwind_batch",
                       "regrid", "amr", "adjoint"])
    dtype = rng.choice(["f32", "f64"])
    a, b = rng.choice([-1, 1]) * rng.uniform(0.2, 1.0), rng.choice([-1, 1]) * rng.uniform(0.2, 1.0)
    if kind == "expr":
        if rng.random() < 0.5:
            return {"kind": kind, "shapes": False, "size": _log_int(rng, 64, 2048), "copies": 1,
                    "geometry": geometry}
        return {"kind": kind, "shapes": True, "size": _log_int(rng, 300, 4096), "copies": _log_int(rng, 1, 128),
                "geometry": geometry}
    if kind == "batch_sets":
        return {"kind": kind, "count": _log_int(rng, 8, 256), "geometry": geometry}
    if kind == "morph":
        return {"kind": kind, "op": rng.choice(["dilate", "erode", "ghost"]), "size": _log_int(rng, 300, 4096),
                "copies": _log_int(rng, 1, 8), "hx": rng.randint(0, 4), "hy": rng.randint(1, 4),
                "geometry": geometry}
    if kind == "fields":
        return {"kind": kind, "size": _log_int(rng, 200, 2048), "ratio": rng.choice([2, 2, 3, 4]),
                "reducer": rng.choice(["mean", "mean", "sum", "min", "max"]), "dtype": dtype, "geometry": geometry}
    if kind == "sync":
        return {"kind": kind, "size": _log_int(rng, 128, 2048), "dtype": dtype}
    if kind == "upwind":
        return {"kind": kind, "size": _log_int(rng, 128, 8192), "dtype": dtype, "a": a, "b": b,
                "geometry": geometry}
    if kind == "upwind_batch":
        return {"kind": kind, "count": _log_int(rng, 8, 256), "dtype": "f32", "a": a, "b": b,
                "geometry": geometry}
    if kind == "regrid":
        return {"kind": kind, "size": _log_int(rng, 200, 4096), "tag": rng.choice(["threshold", "fraction"]),
                "padding": rng.randint(1, 3), "mode": rng.choice(["von_neumann", "moore"]),
                "geometry": geometry}
    if kind == "amr":
        return {"kind": kind, "size": _log_int(rng, 100, 2048), "steps": 5 * rng.randint(2, 8),
                "every": rng.choice([5, 10]), "dtype": dtype}
    return {"kind": "adjoint", "base": 2 * _log_int(rng, 64, 512), "steps": rng.randint(10, 40),
            "every": rng.choice([5, 10]), "dtype": dtype}


# ----------------------------------------------------------------------------------------------------------------
# Inputs
# ----------------------------------------------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device=_DEVICE).manual_seed(int(seed))


def _runs(mask):
    """(row_offsets, begin, end) of a boolean mask, all rows kept."""
    h, w = mask.shape
    edge = torch.zeros((h, w + 1), dtype=torch.bool, device=mask.device)
    edge[:, 0] = mask[:, 0]
    edge[:, w] = mask[:, w - 1]
    edge[:, 1:w] = mask[:, 1:] ^ mask[:, :-1]
    at = torch.nonzero(edge)  # row-major: begins and ends alternate
    begin, end = at[0::2], at[1::2]
    off = torch.zeros(h + 1, dtype=torch.int64, device=mask.device)
    off[1:] = torch.cumsum(torch.bincount(begin[:, 0], minlength=h), 0)
    return off.to(torch.int32), begin[:, 1].to(torch.int32), end[:, 1].to(torch.int32)


def _turned(mask, seed):
    """The mask mirrored and flipped as the seed says."""
    axes = [a for a in (0, 1) if (seed >> a) & 1]
    return mask.flip(axes) if axes else mask


def _disk_mask(n, cx, cy, r):
    c = torch.arange(n, dtype=torch.float64, device=_DEVICE) + 0.5
    return ((c - cx) ** 2)[None, :] + ((c - cy) ** 2)[:, None] <= r * r


def _checker_mask(n, period, sx, sy):
    i = torch.arange(n, device=_DEVICE)
    return (((i + sx) // period)[None, :] + ((i + sy) // period)[:, None]) % 2 == 0


def _circles_mask(n, rng, count=200, r_min=20.0 / 4096, r_max=200.0 / 4096):
    mask = torch.zeros((n, n), dtype=torch.bool, device=_DEVICE)
    c = torch.arange(n, dtype=torch.float64, device=_DEVICE) + 0.5
    for _ in range(count):
        cx, cy, r = rng.uniform(0, n), rng.uniform(0, n), max(1.0, rng.uniform(r_min * n, r_max * n))
        x0, x1 = max(int(cx - r) - 1, 0), min(int(cx + r) + 2, n)
        y0, y1 = max(int(cy - r) - 1, 0), min(int(cy + r) + 2, n)
        mask[y0:y1, x0:x1] |= ((c[x0:x1] - cx) ** 2)[None, :] + ((c[y0:y1] - cy) ** 2)[:, None] <= r * r
    return mask


def _shape_masks(n, geometry):
    """Disk, annulus, checkerboard, circles and a shifted checkerboard on an ``n x n`` grid."""
    rng = random.Random(geometry)
    s = n / 4096.0
    period = max(1, int(64 * s))
    cx, cy = n / 2 + rng.uniform(-64, 64) * s, n / 2 + rng.uniform(-64, 64) * s
    sx, sy = rng.randrange(2 * period), rng.randrange(2 * period)
    yield _disk_mask(n, cx, cy, rng.uniform(1400, 1600) * s)
    yield _disk_mask(n, cx, cy, rng.uniform(1100, 1300) * s) & ~_disk_mask(n, cx, cy, rng.uniform(700, 900) * s)
    yield _checker_mask(n, period, sx, sy)
    yield _circles_mask(n, rng)
    yield _checker_mask(n, period, sx + max(1, period // 2), sy)


def _stacked(mask, copies, lowest_shift):
    """``copies`` of the mask's set on consecutive row bands, each shifted in x by a different amount."""
    off, b, e = _runs(mask)
    shift = (torch.arange(copies, device=_DEVICE) * 37) % 128 + lowest_shift
    shift = shift.to(torch.int32)[:, None]
    counts = (off[1:] - off[:-1]).repeat(copies)
    all_off = torch.zeros(counts.numel() + 1, dtype=torch.int64, device=_DEVICE)
    all_off[1:] = torch.cumsum(counts, 0)
    return build_interval_set(all_off.to(torch.int32), (b[None, :] + shift).reshape(-1),
                              (e[None, :] + shift).reshape(-1))


def _random_rows(n, g, order):
    """Rows (in ``order``) of min(Poisson(4), 8) intervals, gaps geometric with mean 8, lengths with mean 12."""
    k = torch.poisson(torch.full((n,), 4.0, device=_DEVICE), generator=g).clamp_max(8).to(torch.int64)
    step = torch.empty((n, 16), device=_DEVICE)
    step[:, 0::2].geometric_(1.0 / 8, generator=g)
    step[:, 1::2].geometric_(1.0 / 12, generator=g)
    k, at = k[order], torch.cumsum(step, 1).to(torch.int64)[order]
    b, e = at[:, 0::2], at[:, 1::2].clamp_max(n)
    keep = (torch.arange(8, device=_DEVICE)[None, :] < k[:, None]) & (b < n)
    off = torch.zeros(n + 1, dtype=torch.int64, device=_DEVICE)
    off[1:] = torch.cumsum(keep.sum(1), 0)
    return build_interval_set(off.to(torch.int32), b[keep].to(torch.int32), e[keep].to(torch.int32))


def _sides(count):
    rng = random.Random(3)
    return [_log_int(rng, _SIDE_LO, _SIDE_HI) for _ in range(count)]


def _uneven(sides, geometry, seed):
    """Per set, (row_offsets, begin, end): lognormal(1.5, 1) intervals per row from 2k distinct points of the side.

    The seed rotates the rows of every set and mirrors all of them or none.
    """
    g, turn = _generator(geometry), random.Random(seed)
    side = torch.repeat_interleave(torch.tensor(sides, device=_DEVICE), torch.tensor(sides, device=_DEVICE))
    k = torch.empty(side.numel(), device=_DEVICE).log_normal_(1.5, 1.0, generator=g).round().to(torch.int64)
    k = torch.minimum(k, side // 2)
    row = torch.repeat_interleave(torch.arange(side.numel(), device=_DEVICE), 2 * k)
    start = torch.cumsum(2 * k, 0) - 2 * k
    nth = torch.arange(row.numel(), device=_DEVICE) - start[row]
    free = (side + 2 - 2 * k)[row]  # sorted draws from [0, side + 1 - 2k] plus their rank are distinct points
    u = torch.minimum((torch.rand(row.numel(), device=_DEVICE, generator=g, dtype=torch.float64) * free).long(),
                      free - 1)
    point = (torch.sort((row << 32) | u).values & 0xFFFFFFFF) + nth
    rows = [0]
    for s in sides:
        rows.append(rows[-1] + s)
    to = torch.cat([torch.arange(s, device=_DEVICE).add_(turn.randrange(s)).remainder_(s) + r
                    for s, r in zip(sides, rows)])  # the row that each row is moved to
    if seed & 1:
        point = side[row] - point
    point = torch.sort((to[row] << 32) | point).values & 0xFFFFFFFF
    counts = torch.empty_like(k)
    counts[to] = k
    begin, end = point[0::2].to(torch.int32), point[1::2].to(torch.int32)
    off = torch.zeros(side.numel() + 1, dtype=torch.int64, device=_DEVICE)
    off[1:] = torch.cumsum(counts, 0)
    cut = off[torch.tensor(rows, device=_DEVICE)].tolist()
    return [((off[r0:r1 + 1] - lo).to(torch.int32), begin[lo:hi], end[lo:hi])
            for r0, r1, lo, hi in zip(rows, rows[1:], cut, cut[1:])]


def _batch(sides, parts):
    return SetBatch.from_sets([build_interval_set(*p) for p in parts], sides)


def _mask_of(part, side):
    off, b, e = (x.long() for x in part)
    row = torch.repeat_interleave(torch.arange(side, device=_DEVICE), off[1:] - off[:-1])
    edge = torch.zeros((side, side + 1), dtype=torch.int8, device=_DEVICE)
    edge[row, b] += 1
    edge[row, e] -= 1
    return torch.cumsum(edge, 1, dtype=torch.int8)[:, :side] > 0


def _values(count, dtype, g):
    """Values of order one, smooth along the storage order with noise on top."""
    x = torch.arange(count, device=_DEVICE, dtype=dtype)
    phase = torch.rand(1, device=_DEVICE, generator=g, dtype=dtype)
    return torch.sin(x.mul_(1e-3).add_(6.28 * phase)).add_(
        torch.rand(count, device=_DEVICE, generator=g, dtype=dtype), alpha=0.25)


def _blob(n, seed, dtype, blobs=1, width=0.05):
    """Gaussian blobs on the unit square, placed by the seed."""
    rng = random.Random(seed)
    c = (torch.arange(n, dtype=torch.float64, device=_DEVICE) + 0.5) / n
    u = torch.zeros((n, n), dtype=torch.float64, device=_DEVICE)
    for _ in range(blobs):
        cx, cy = rng.uniform(0.3, 0.7), rng.uniform(0.3, 0.7)
        u += torch.exp(-((c - cy) ** 2) / (2 * width ** 2))[:, None] * torch.exp(-((c - cx) ** 2) / (2 * width ** 2))
    return u.to(dtype)


def _geometry_mask(case, seed):
    """Ragged geometry of a field: circles and a large disk."""
    n, rng = case["size"], random.Random(case["geometry"])
    return _turned(_circles_mask(n, rng) | _disk_mask(n, n * rng.uniform(0.4, 0.6), n * rng.uniform(0.4, 0.6),
                                                      0.3 * n), seed)


def _regrid_field(case, seed):
    """Six blobs that vanish towards the edges, moved by up to a sixteenth of the grid and turned by the seed."""
    n, rng = case["size"], random.Random(seed)
    u = _blob(n, case["geometry"], torch.float32, blobs=6)
    u = torch.where(u < 1e-3, torch.zeros_like(u), u)
    return _turned(u.roll((rng.randint(-(n // 16), n // 16), rng.randint(-(n // 16), n // 16)), (0, 1)),
                   seed).contiguous()


def _occupied_set(mask):
    """Set of a mask on its occupied rows only, and those rows."""
    rows = torch.nonzero(mask.any(1)).reshape(-1)
    off, b, e = _runs(mask[rows])
    return build_interval_set(off, b, e, rows=rows.to(torch.int32)), rows


def _level_masks(base):
    """Nested levels: the whole base grid and two centred disks, each made of whole blocks of the level above."""
    masks, n = [torch.ones((base, base), dtype=torch.bool, device=_DEVICE)], base
    for radius in (0.3, 0.15):
        d = _disk_mask(n, n / 2, n / 2, radius * n)
        masks.append(d.repeat_interleave(2, 0).repeat_interleave(2, 1))
        n *= 2
    return masks


def _adjoint_inputs(case, seed):
    g, dtype = _generator(seed), _DTYPES[case["dtype"]]
    masks = _level_masks(case["base"])
    cells = [int(m.sum()) for m in masks]
    return masks, [_values(c, dtype, g) for c in cells], [_values(c, dtype, g) for c in cells]


_VELOCITY = (1.0, 0.5)


def _adjoint_dt(case):
    finest = 1.0 / (4 * case["base"])
    return 0.5 * finest / (abs(_VELOCITY[0]) + abs(_VELOCITY[1]))


# ----------------------------------------------------------------------------------------------------------------
# The cases
# ----------------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind, g = case["kind"], _generator(seed)
    if kind == "expr":
        n, turn = case["size"], random.Random(seed)
        if case["shapes"]:
            shift, roll = turn.randrange(256) - 128, turn.randrange(n)
            sets = [_stacked(_turned(m, seed).roll(roll, 0), case["copies"], shift)
                    for m in _shape_masks(n, case["geometry"])]
        else:
            order, g = torch.randperm(n, device=_DEVICE, generator=g), _generator(case["geometry"])
            sets = [_random_rows(n, g, order) for _ in range(5)]
        return {"case": case, "sets": sets}
    if kind == "batch_sets":
        sides = _sides(case["count"])
        return {"case": case, "A": _batch(sides, _uneven(sides, 2 * case["geometry"], seed)),
                "B": _batch(sides, _uneven(sides, 2 * case["geometry"] + 1, seed))}
    if kind == "morph":
        n = case["size"]
        rng = random.Random(case["geometry"])
        mask = _circles_mask(n, rng) | _checker_mask(n, max(1, int(64 * n / 4096)), rng.randrange(64), 0)
        margin = 8 + seed % 64  # the halo stays inside the domain's columns
        return {"case": case, "set": _stacked(_turned(mask, seed >> 6), case["copies"], margin), "width": n + 256,
                "height": n * case["copies"]}
    if kind == "fields":
        dtype = _DTYPES[case["dtype"]]
        s, _ = _occupied_set(_geometry_mask(case, seed))
        coarse = create_interval_field(s, 0.0, dtype=dtype)
        coarse.values.copy_(_values(coarse.values.numel(), dtype, g))
        fine = create_interval_field(prolong_set(s, case["ratio"]), 0.0, dtype=dtype)
        fine.values.copy_(_values(fine.values.numel(), dtype, g))
        return {"case": case, "coarse": coarse, "fine": fine}
    if kind == "sync":
        n, dtype = case["size"], _DTYPES[case["dtype"]]
        coarse = create_interval_field(full_interval_set(n, n), 0.0, dtype=dtype)
        coarse.values.copy_(_values(n * n, dtype, g))
        fine = create_interval_field(full_interval_set(2 * n, 2 * n), 0.0, dtype=dtype)
        fine.values.copy_(_values(4 * n * n, dtype, g))
        actions = ActionField.full_grid(n, n, 2)
        actions.set_from_interval_set(build_interval_set(*_runs(_circles_mask(n, random.Random(seed)))))
        return {"case": case, "coarse": coarse, "fine": fine, "actions": actions}
    if kind == "upwind":
        dtype = _DTYPES[case["dtype"]]
        s, _ = _occupied_set(_geometry_mask(case, seed))
        field = create_interval_field(s, 0.0, dtype=dtype)
        field.values.copy_(_values(field.values.numel(), dtype, g))
        return {"case": case, "field": field}
    if kind == "upwind_batch":
        sides = _sides(case["count"])
        batch = _batch(sides, _uneven(sides, case["geometry"], seed))
        plan = batch.stencil_plan()
        return {"case": case, "sides": sides, "batch": batch,
                "values": _values(plan.cells, _DTYPES[case["dtype"]], g)}
    if kind == "regrid":
        n = case["size"]
        field = create_interval_field(full_interval_set(n, n), 0.0, dtype=np.float32)
        field.values.copy_(_regrid_field(case, seed).reshape(-1))
        return {"case": case, "field": field}
    if kind == "amr":
        n = case["size"]
        u0 = _blob(n, seed, _DTYPES[case["dtype"]])
        sim = AMR2Simulation(SimulationConfig(coarse_resolution=n, velocity=_VELOCITY, cfl=0.5,
                                              refine_threshold=0.05 / n))
        field = create_interval_field(full_interval_set(n, n), 0.0, dtype=_NUMPY[case["dtype"]])
        field.values.copy_(u0.reshape(-1))
        sim.set_initial_field(field)
        sim.engine.prepare_graphs(case["every"])
        fine0 = u0.repeat_interleave(2, 0).repeat_interleave(2, 1).reshape(-1)
        return {"case": case, "sim": sim, "u0": u0.reshape(-1), "fine0": fine0}
    masks, u0, w = _adjoint_inputs(case, seed)
    sets = [_occupied_set(m)[0] for m in masks]
    h = Hierarchy(sets, case["base"], case["base"])
    return {"case": case, "hierarchy": h, "u0": [u.requires_grad_(True) for u in u0], "w": w,
            "velocity": torch.tensor(_VELOCITY, dtype=torch.float64, device=_DEVICE, requires_grad=True)}


def _set_out(s):
    return [s.begin, s.end, s.row_offsets, s.rows]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "expr":
        A, B, C, D, E = (make_input(s) for s in state["sets"])
        return _set_out(evaluate(make_symmetric_difference(
            make_difference(make_union(A, B), make_intersection(C, D)), E)))
    if kind == "batch_sets":
        return {m: _set_out(batched_binary(state["A"], state["B"], m).combined) for m in ("union", "intersection")}
    if kind == "morph":
        s, hx, hy = state["set"], case["hx"], case["hy"]
        if case["op"] == "dilate":
            return _set_out(dilate_interval_set(s, halo_x=hx, halo_y=hy))
        op = erode_interval_set if case["op"] == "erode" else ghost_zones
        return _set_out(op(s, halo_x=hx, halo_y=hy, width=state["width"], height=state["height"]))
    if kind == "fields":
        dtype = _NUMPY[case["dtype"]]
        up = prolong_field(state["coarse"], case["ratio"], dtype=dtype)
        down = restrict_field(state["fine"], case["ratio"], reducer=case["reducer"], dtype=dtype)
        return {"up": up.values, "up_set": _set_out(up.interval_set), "down": down.values,
                "down_set": _set_out(down.interval_set)}
    if kind == "sync":
        coarse, fine = synchronize_interval_fields(state["coarse"], state["fine"], state["actions"], ratio=2)
        return {"coarse": coarse.values, "fine": fine.values}
    if kind == "upwind":
        n, a, b = case["size"], case["a"], case["b"]
        dt = 0.5 / n / (abs(a) + abs(b))
        return step_upwind_interval(state["field"], width=n, height=n, a=a, b=b, dt=dt, dx=1.0 / n, dy=1.0 / n)
    if kind == "upwind_batch":
        a, b = case["a"], case["b"]
        dx = [1.0 / s for s in state["sides"]]
        dt = [0.5 * d / (abs(a) + abs(b)) for d in dx]
        return batched_upwind(state["batch"], state["values"], width=state["sides"], a=a, b=b, dt=dt, dx=dx, dy=dx)
    if kind == "regrid":
        n, field = case["size"], state["field"]
        out = {}
        if case["tag"] == "threshold":
            tags = gradient_tag_threshold_interval_field(field, width=n, height=n, threshold=0.05 / n)
        else:
            grad = gradient_magnitude_interval_field(field, width=n, height=n)
            out["gradient"] = grad.values
            tags = gradient_tag_set(grad, width=n, height=n, frac_high=0.1)
        graded = enforce_two_level_grading_set(tags, padding=case["padding"], mode=case["mode"], width=n, height=n)
        return {**out, "tags": _set_out(tags), "graded": _set_out(graded)}
    if kind == "amr":
        sim = state["sim"]
        view = sim.state  # a live view: what is written to its fields feeds the next step
        view.coarse_field.values.copy_(state["u0"])
        view.fine_field.values.copy_(state["fine0"])
        view, _ = sim.run(steps=case["steps"], regrid_every=case["every"])
        return {"coarse": view.coarse_field.values, "fine": view.fine_field.values,
                "actions": view.actions.field.values}
    out = advect_composite(state["velocity"], state["hierarchy"], state["u0"], dt=_adjoint_dt(case),
                           steps=case["steps"], checkpoint_every=case["every"])
    grads = torch.autograd.grad(out, [state["velocity"], *state["u0"]], grad_outputs=state["w"])
    return {"out": [o.detach() for o in out], "velocity": grads[0], "u0": list(grads[1:])}


def _size(case):
    return 8 if case["dtype"] == "f64" else 4


def work(case):
    """Each input and each output once (int32 interval arrays, field values), from the distributions of the inputs."""
    kind = case["kind"]
    if kind == "expr":
        rows = case["size"] * case["copies"]
        n_in, n_out = (72 * rows, 40 * rows) if case["shapes"] else (18 * rows, 9 * rows)
        return {"bytes": 8.0 * (n_in + n_out) + 4.0 * 6 * rows, "flops": 0.0}
    if kind == "batch_sets":
        rows = sum(_sides(case["count"]))
        return {"bytes": 8.0 * 2 * (2 * 7.4 * rows) + 4.0 * 4 * rows, "flops": 0.0}
    if kind == "morph":
        rows = case["size"] * case["copies"]
        return {"bytes": 8.0 * 2 * 34 * rows + 4.0 * 2 * rows, "flops": 0.0}
    if kind == "fields":
        cells, r2 = 0.5 * case["size"] ** 2, case["ratio"] ** 2
        return {"bytes": 2.0 * (1 + r2) * cells * _size(case), "flops": r2 * cells}
    if kind == "sync":
        n2 = case["size"] ** 2
        return {"bytes": 2.0 * 5 * n2 * _size(case), "flops": 4.0 * n2}
    if kind == "upwind":
        cells = 0.5 * case["size"] ** 2
        return {"bytes": 2.0 * cells * _size(case), "flops": 9.0 * cells}
    if kind == "upwind_batch":
        cells = 0.5 * sum(s * s for s in _sides(case["count"]))
        return {"bytes": 2.0 * cells * _size(case), "flops": 9.0 * cells}
    if kind == "regrid":
        n2 = case["size"] ** 2
        gradient = 8.0 * n2 if case["tag"] == "fraction" else 4.0 * n2
        return {"bytes": gradient + 8.0 * 4 * 2 * case["size"], "flops": 6.0 * n2}
    if kind == "amr":
        n2 = case["size"] ** 2
        return {"bytes": (n2 * (10.0 * _size(case) + 1)) * case["steps"] + n2 * 6.0 * case["steps"] / case["every"],
                "flops": 9.0 * 2 * n2 * case["steps"]}
    cells = case["base"] ** 2 * (1 + 4 * math.pi * 0.09 + 16 * math.pi * 0.0225)
    return {"bytes": cells * _size(case) * case["steps"] * (2.0 + 2.0 + 3.0), "flops": 30.0 * cells * case["steps"]}


# ----------------------------------------------------------------------------------------------------------------
# The floating results in float64, from plain torch on dense grids
# ----------------------------------------------------------------------------------------------------------------

def _dense_upwind(u, a, b, dt, dx, dy):
    """Upwind update on a dense grid that is zero outside the geometry (no masking of the result)."""
    h, v = torch.zeros_like(u), torch.zeros_like(u)
    if a >= 0:
        h[:, 1:] = u[:, :-1]
        du = (u - h) / dx
    else:
        h[:, :-1] = u[:, 1:]
        du = (h - u) / dx
    if b >= 0:
        v[1:] = u[:-1]
        dv = (u - v) / dy
    else:
        v[:-1] = u[1:]
        dv = (v - u) / dy
    return u - dt * (a * du + b * dv)


def _spread(mask, values):
    u = torch.zeros(mask.shape, dtype=torch.float64, device=_DEVICE)
    u[mask] = values.double()
    return u


def _dense_gradient(u):
    """Half central differences inside, one-sided at the edges."""
    gx, gy = torch.zeros_like(u), torch.zeros_like(u)
    gx[:, 1:-1] = (u[:, 2:] - u[:, :-2]) * 0.5
    gx[:, 0], gx[:, -1] = u[:, 1] - u[:, 0], u[:, -1] - u[:, -2]
    gy[1:-1] = (u[2:] - u[:-2]) * 0.5
    gy[0], gy[-1] = u[1] - u[0], u[-1] - u[-2]
    return torch.sqrt(gx * gx + gy * gy)


def _blocks(fine):
    h, w = fine.shape
    return fine.reshape(h // 2, 2, w // 2, 2).sum(dim=(1, 3)) * 0.25


def _double(u):
    return u.repeat_interleave(2, 0).repeat_interleave(2, 1)


def _exact_amr(case, seed):
    n = case["size"]
    dx, (a, b) = 1.0 / n, _VELOCITY
    dt = 0.5 / (abs(a) / (dx / 2) + abs(b) / (dx / 2))
    coarse = _blob(n, seed, _DTYPES[case["dtype"]]).double()
    fine = _double(coarse)
    refined = None
    for k in range(case["steps"]):
        if k % case["every"] == 0:
            tag = _dense_gradient(coarse.float()) >= float(np.float32(0.05 / n))
            refined = tag.clone()
            refined[:, 1:] |= tag[:, :-1]
            refined[:, :-1] |= tag[:, 1:]
            refined[1:] |= tag[:-1]
            refined[:-1] |= tag[1:]
        coarse = _dense_upwind(coarse, a, b, dt, dx, dx)
        fine = _dense_upwind(fine, a, b, dt, dx / 2, dx / 2)
        coarse = torch.where(refined, _blocks(fine), coarse)
        fine = torch.where(_double(refined), fine, _double(coarse))
    return {"coarse": coarse.reshape(-1), "fine": fine.reshape(-1), "actions": None}


def _composite_step(u, masks, rings, base, ab, dt):
    """One composite step on dense grids: ghost rings from the parents, upwind everywhere, means under finer levels."""
    u = list(u)
    for k in range(1, len(u)):
        u[k] = torch.where(rings[k], _double(u[k - 1]), u[k])
    new = []
    for k, x in enumerate(u):
        d = 1.0 / (base * 2 ** k)
        h = torch.nn.functional.pad(x[:, :-1], (1, 0))  # both velocities of this workload are positive
        v = torch.nn.functional.pad(x[:-1], (0, 0, 1, 0))
        y = x - dt * (ab[0] * ((x - h) / d) + ab[1] * ((x - v) / d))
        new.append(torch.where(masks[k], y, torch.zeros_like(y)))
    for k in range(len(u) - 1, 0, -1):
        new[k - 1] = torch.where(masks[k][::2, ::2], _blocks(new[k]), new[k - 1])
    return new


def _exact_adjoint(case, seed):
    masks, u0, w = _adjoint_inputs(case, seed)
    rings = []
    for m in masks:
        near = m.clone()
        near[:, 1:] |= m[:, :-1]
        near[:, :-1] |= m[:, 1:]
        near[1:] |= m[:-1]
        near[:-1] |= m[1:]
        rings.append(near & ~m)
    dt, base = _adjoint_dt(case), case["base"]
    ab = torch.tensor(_VELOCITY, dtype=torch.float64, device=_DEVICE)
    states = [[_spread(m, u) for m, u in zip(masks, u0)]]
    for _ in range(case["steps"]):
        states.append(_composite_step(states[-1], masks, rings, base, ab, dt))
    out = [s[m] for s, m in zip(states.pop(), masks)]
    bar = [_spread(m, x) for m, x in zip(masks, w)]
    grad_ab = torch.zeros_like(ab)
    while states:
        ins = [x.requires_grad_(True) for x in states.pop()]
        v = ab.clone().requires_grad_(True)
        new = _composite_step(ins, masks, rings, base, v, dt)
        got = torch.autograd.grad(new, [v, *ins], grad_outputs=bar)
        grad_ab += got[0]
        bar = list(got[1:])
    return {"out": out, "velocity": grad_ab, "u0": [x[m] for x, m in zip(bar, masks)]}


def exact(case, seed):
    kind, g = case["kind"], _generator(seed)
    if kind == "fields":
        r, dtype = case["ratio"], _DTYPES[case["dtype"]]
        mask = _geometry_mask(case, seed)
        rows = torch.nonzero(mask.any(1)).reshape(-1)
        mask = mask[rows]
        coarse = _values(int(mask.sum()), dtype, g)
        fine_mask = mask.repeat_interleave(r, 0).repeat_interleave(r, 1)
        fine = _values(int(fine_mask.sum()), dtype, g)
        up = _spread(mask, coarse).repeat_interleave(r, 0).repeat_interleave(r, 1)[fine_mask]
        blocks = _spread(fine_mask, fine).reshape(mask.shape[0], r, mask.shape[1], r)
        reduce = {"mean": lambda x: x.sum(dim=(1, 3)) / (r * r), "sum": lambda x: x.sum(dim=(1, 3)),
                  "min": lambda x: x.amin(dim=(1, 3)), "max": lambda x: x.amax(dim=(1, 3))}[case["reducer"]]
        return {"up": up, "up_set": [None] * 4, "down": reduce(blocks)[mask], "down_set": [None] * 4}
    if kind == "sync":
        n, dtype = case["size"], _DTYPES[case["dtype"]]
        coarse = _values(n * n, dtype, g).double().reshape(n, n)
        fine = _values(4 * n * n, dtype, g).double().reshape(2 * n, 2 * n)
        refined = _circles_mask(n, random.Random(seed))
        coarse = torch.where(refined, _blocks(fine), coarse)
        fine = torch.where(_double(refined), fine, _double(coarse))
        return {"coarse": coarse.reshape(-1), "fine": fine.reshape(-1)}
    if kind == "upwind":
        n, a, b = case["size"], case["a"], case["b"]
        mask = _geometry_mask(case, seed)
        u = _spread(mask, _values(int(mask.sum()), _DTYPES[case["dtype"]], g))
        return _dense_upwind(u, a, b, 0.5 / n / (abs(a) + abs(b)), 1.0 / n, 1.0 / n)[mask]
    if kind == "upwind_batch":
        a, b, sides = case["a"], case["b"], _sides(case["count"])
        parts = _uneven(sides, case["geometry"], seed)
        cells = [int((e - b_).sum()) for _, b_, e in parts]
        values = _values(sum(cells), _DTYPES[case["dtype"]], g)
        out, at = [], 0
        for side, part, n in zip(sides, parts, cells):
            mask = _mask_of(part, side)
            u = _spread(mask, values[at:at + n])
            out.append(_dense_upwind(u, a, b, 0.5 / side / (abs(a) + abs(b)), 1.0 / side, 1.0 / side)[mask])
            at += n
        return torch.cat(out)
    if kind == "regrid" and case["tag"] == "fraction":
        u = _regrid_field(case, seed).double()
        return {"gradient": _dense_gradient(u).reshape(-1), "tags": [None] * 4, "graded": [None] * 4}
    if kind == "amr":
        return _exact_amr(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    return None
