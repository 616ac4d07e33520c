"""Adjoint passes over one geometry on several streams: every pass counts its blocks in its own scratch."""

import pytest
import torch

from subsetix_b200 import _core, adjoint
from subsetix_b200.subsetix_cupy import full_interval_set
from tests.test_gpu_adjoint import _hierarchy

pytestmark = pytest.mark.gpu


def test_passes_and_segments_do_not_share_counters(cuda_device, monkeypatch):
    """No launch: the scratch that each adjoint would get is recorded."""
    used = []
    monkeypatch.setattr(_core.FlatPlan, "adjoint", lambda self, w, u, out, a, b, dt, dx, dy, grad, scratch, device:
                        (used.append((torch.cuda.current_stream().cuda_stream, scratch)), out.copy_(w)))
    lvl = adjoint.Level(full_interval_set(64, 48), 64, 48, 1.0 / 64, 1.0 / 48)
    H, _ = _hierarchy()
    x, grad = torch.rand(64 * 48, device="cuda"), torch.zeros(2, dtype=torch.float64, device="cuda")
    for stream in (torch.cuda.Stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            lvl.adjoint(x, x, 0.5, 0.5, 1e-3, grad)
            vel = torch.tensor([0.5, 0.5], device="cuda", requires_grad=True)
            adjoint.advect(vel, [lvl], [x], dt=1e-3, steps=2)[0].sum().backward()
            u = [torch.rand(n, device="cuda") for n in H.inner_cells]
            for graphs, steps in ((False, 2), (True, 2), (True, 3)):
                sum(o.sum() for o in adjoint.advect_composite(vel, H, u, dt=1e-3, steps=steps, graphs=graphs)).backward()
    streams = {}
    for stream, scratch in used:
        streams.setdefault(scratch.data_ptr(), set()).add(stream)
    assert len(used) > 20 and all(len(s) == 1 for s in streams.values())


def test_overlapping_passes(cuda_device):
    """Passes that overlap on two streams give the gradients of passes run alone, and leave later ones right."""
    n = 512
    lvl = adjoint.Level(full_interval_set(n, n), n, n, 1.0 / n, 1.0 / n)
    gen = torch.Generator(device="cuda").manual_seed(1)
    w, u = (torch.rand(lvl.cells, dtype=torch.float64, device="cuda", generator=gen) for _ in range(2))

    def passes(scratch):
        grad = torch.zeros(2, dtype=torch.float64, device="cuda")
        for _ in range(20):
            out = lvl.adjoint(w, u, 0.7, -0.2, 1e-4, grad, scratch=scratch)
        return grad, out

    want = passes(None)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for s in streams:
        with torch.cuda.stream(s):
            got.append(passes(lvl.adjoint_scratch()))
    torch.cuda.synchronize()
    got.append(passes(None))
    for grad, out in got:
        assert torch.equal(grad, want[0]) and torch.equal(out, want[1])
