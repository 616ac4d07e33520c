"""Synchronisation of whole-grid fields by the dense kernel against the interval kernels, bit for bit."""

import numpy as np
import pytest
import torch

from subsetix_b200.subsetix_amr2 import fields as F
from subsetix_b200.subsetix_cupy import IntervalField, build_interval_set, create_interval_field, full_interval_set

pytestmark = pytest.mark.gpu


def _field(w, h, dtype, rng):
    f = create_interval_field(full_interval_set(w, h), 0.0, dtype=dtype)
    f.values.copy_(torch.as_tensor(rng.standard_normal(w * h), device="cuda"))
    return f


def _actions(w, h, ratio, kind, rng):
    act = F.ActionField.full_grid(h, w, ratio, default=F.Action.REFINE if kind == "default" else F.Action.KEEP)
    if kind == "default":  # the bytes say REFINE, the cached refine set is empty, as in the reference
        return act
    if kind == "values":   # written as bytes, the set derived from them
        act.values().copy_(torch.as_tensor(rng.integers(-1, 2, w * h).astype(np.int8), device="cuda"))
        act._refresh_from_values()
        return act
    mask = rng.random((h, w)) < {"some": 0.3, "none": 0.0, "all": 1.1}[kind]
    e = np.diff(np.pad(mask, ((0, 0), (1, 1))).astype(np.int8), axis=1)
    off = np.concatenate([[0], np.cumsum((e == 1).sum(1))])
    act.set_from_interval_set(build_interval_set(off, np.nonzero(e == 1)[1], np.nonzero(e == -1)[1]))
    if kind == "some":  # later writes to the bytes do not change the cached refine set
        act.values().fill_(1)
    return act


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ratio", [2, 3])
@pytest.mark.parametrize("kind", ["some", "none", "all", "values", "default"])
@pytest.mark.parametrize("w,h", [(1, 1), (7, 5), (256, 3), (257, 9)])
def test_whole_grid_sync_equals_interval_kernels(cuda_device, monkeypatch, dtype, ratio, kind, w, h):
    rng = np.random.default_rng(w + h)
    coarse, fine = _field(w, h, dtype, rng), _field(w * ratio, h * ratio, dtype, rng)
    act = _actions(w, h, ratio, kind, rng)
    taken = []
    whole = F._synchronize_whole_grids
    monkeypatch.setattr(F, "_synchronize_whole_grids", lambda *a: taken.append(whole(*a)) or taken[-1])
    before = coarse.values.clone(), fine.values.clone()
    got = F.synchronize_interval_fields(coarse, fine, act, ratio=ratio)
    assert taken[-1] is not None
    assert torch.equal(coarse.values, before[0]) and torch.equal(fine.values, before[1])
    place = F.clone_interval_field(coarse), F.clone_interval_field(fine)
    F.synchronize_interval_fields(*place, act, ratio=ratio, copy=False)
    assert taken[-1] is not None
    monkeypatch.setattr(F, "_synchronize_whole_grids", lambda *a: None)
    ref = F.synchronize_interval_fields(coarse, fine, act, ratio=ratio)
    for a, b, c in zip(got, place, ref):
        assert torch.equal(a.values, c.values) and torch.equal(b.values, c.values)
        assert torch.equal(a.interval_cell_offsets, c.interval_cell_offsets)


def test_other_fields_keep_the_interval_kernels(cuda_device):
    rng = np.random.default_rng(1)
    coarse, fine, act = _field(8, 6, np.float32, rng), _field(16, 12, np.float32, rng), _actions(8, 6, 2, "some", rng)
    assert F._synchronize_whole_grids(coarse, fine, act, 2, True) is not None
    own = IntervalField(interval_set=coarse.interval_set, values=coarse.values,
                        interval_cell_offsets=coarse.interval_cell_offsets)
    assert F._synchronize_whole_grids(own, fine, act, 2, True) is None      # offsets of unknown origin
    coarse.interval_cell_offsets.add_(0)
    assert F._synchronize_whole_grids(coarse, fine, act, 2, True) is None   # offsets modified since
    coarse = _field(8, 6, np.float32, rng)
    act._refine_set_cache = act._refine_set_cache.copy()
    assert F._synchronize_whole_grids(coarse, fine, act, 2, True) is None   # a refine set put in from outside
    coarse.values.requires_grad_(True)
    assert F._synchronize_whole_grids(coarse, fine, _actions(8, 6, 2, "all", rng), 2, True) is None
