"""Capture of a composite segment that fails: out of memory once, and another error (both raised on the host)."""

import pytest
import torch

from subsetix_b200 import adjoint
from tests.test_gpu_adjoint import _hierarchy

pytestmark = pytest.mark.gpu


def _run(H, graphs):
    gen = torch.Generator(device="cuda").manual_seed(5)
    vel = torch.tensor([0.4, -0.3], dtype=torch.float64, device="cuda", requires_grad=True)
    u = [torch.rand(n, dtype=torch.float64, device="cuda", generator=gen).requires_grad_() for n in H.inner_cells]
    out = adjoint.advect_composite(vel, H, u, dt=2e-3, steps=7, checkpoint_every=4, graphs=graphs)
    return [x.detach().clone() for x in (*out, *torch.autograd.grad(sum(x.square().sum() for x in out), [vel, *u]))]


def _fail_once(monkeypatch, at, error):
    """Level.step raises ``error`` at its call number ``at`` and works from then on."""
    step, calls = adjoint.Level.step, []

    def failing(self, *args):
        calls.append(torch.cuda.is_current_stream_capturing())
        if len(calls) == at:
            raise error
        return step(self, *args)

    monkeypatch.setattr(adjoint.Level, "step", failing)
    return calls


@pytest.mark.parametrize("at", [1, 5, 16])  # the first graph's first and later launches, the second graph's
def test_out_of_memory_once(cuda_device, monkeypatch, at):
    H, _ = _hierarchy()
    want = _run(H, False)
    emptied = []
    empty_cache = torch.cuda.empty_cache
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: (emptied.append(1), empty_cache()))
    calls = _fail_once(monkeypatch, at, torch.OutOfMemoryError("planned"))
    got = _run(H, True)
    assert len(calls) > at and all(calls) and emptied
    for g, w in zip(got, want):
        assert torch.equal(g, w)


def test_other_errors_come_through(cuda_device, monkeypatch):
    H, _ = _hierarchy()
    want = _run(H, False)
    calls = _fail_once(monkeypatch, 5, ValueError("planned"))
    with pytest.raises(ValueError, match="planned"):
        _run(H, True)
    assert len(calls) == 5
    for g, w in zip(_run(H, True), want):
        assert torch.equal(g, w)
