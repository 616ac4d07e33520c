"""Fields made under torch.inference_mode(), whose tensors track no versions."""

import numpy as np
import pytest
import torch

from subsetix_b200.subsetix_cupy.interval_field import IntervalField, _is_packed, _packed_field


def test_inference_offsets_are_not_known_to_be_packed():
    with torch.inference_mode():
        off = torch.tensor([0, 3], dtype=torch.int32)
        assert not _is_packed(_packed_field(None, torch.zeros(3), off))
    field = _packed_field(None, torch.zeros(3), torch.tensor([0, 3], dtype=torch.int32))
    assert _is_packed(field)
    with torch.inference_mode():
        assert _is_packed(field)
        assert not _is_packed(IntervalField(interval_set=None, values=torch.zeros(3), interval_cell_offsets=off))


@pytest.mark.gpu
def test_field_calls_under_inference_mode(cuda_device):
    from subsetix_b200.subsetix_amr2.fields import ActionField, synchronize_interval_fields
    from subsetix_b200.subsetix_cupy import (build_interval_set, create_interval_field, full_interval_set,
                                             prolong_field, restrict_field)

    def calls():
        domain = full_interval_set(12, 8)
        coarse = create_interval_field(domain, 0.0, dtype=np.float32)
        coarse.values.copy_(torch.arange(96, device="cuda", dtype=torch.float32))
        fine = prolong_field(coarse, 2)
        fine.values.mul_(torch.linspace(1.0, 2.0, 384, device="cuda"))
        back = restrict_field(fine, 2)
        actions = ActionField.full_grid(8, 12, 2)
        actions.set_from_interval_set(build_interval_set([0, 1, 2], [2, 2], [7, 9], rows=[3, 4]))
        out = synchronize_interval_fields(coarse, fine, actions, ratio=2)
        return [f.values for f in (fine, back, *out)]

    want = calls()
    with torch.inference_mode():
        got = calls()
    for g, w in zip(got, want):
        assert torch.equal(g.clone(), w)
