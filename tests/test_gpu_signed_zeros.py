"""Zeros keep their sign: the kernels that divide by a known spacing against those that divide, bits compared."""

import numpy as np
import pytest
import torch

from subsetix_b200 import _core, _lib
from subsetix_b200 import adjoint as adj
from subsetix_b200._runtime import ptr, stream_handle
from tests.gpu_util import dev_set
from tests.test_gpu_amr_steps import _inputs, _one_by_one
from tests.test_gpu_flat_stencil import _geometries, _plan

pytestmark = pytest.mark.gpu

ZEROS = [0.0, -0.0, -0.0, -0.0, 1.0, -0.25]


def _bits(t):
    return t.view(torch.int64 if t.dtype == torch.float64 else torch.int32)


def _draw(rng, n, dtype, values=ZEROS):
    return torch.as_tensor(rng.choice(np.asarray(values), n), device="cuda").to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("a,b", [(0.6, 0.3), (-0.4, 0.9), (0.6, -0.3), (0.0, -0.0)])
def test_flat_step_and_adjoint(cuda_device, dtype, a, b):
    rng = np.random.default_rng(4)
    code = _lib.SX_F64 if dtype == torch.float64 else _lib.SX_F32
    signs = 0
    for h in _geometries():
        (bg, e, off, rows), H, coff, cells, lookup, plan = _plan(h, cuda_device)
        v, w = _draw(rng, cells, dtype), _draw(rng, cells, dtype)
        ref, got = torch.empty_like(v), torch.empty_like(v)
        _core.upwind(rows, off, bg, e, coff, cells, lookup, v, ref, plan.hi, H, a, b, 1e-3, 1e-2, 1.0 / 777, False,
                     cuda_device)
        plan.step(v, got, a, b, 1e-3, 1e-2, 1.0 / 777, cuda_device)
        assert torch.equal(_bits(got), _bits(ref))
        signs += int((torch.signbit(ref) & (ref == 0)).sum())
        lvl = adj.Level(dev_set(h), plan.hi, H, 1e-2, 1.0 / 777)
        g_ref, g = torch.empty(2, dtype=torch.float64, device="cuda"), torch.zeros(2, dtype=torch.float64, device="cuda")
        got = lvl.adjoint(w, v, a, b, 1e-3, g)
        _lib.check(_lib.load().sx_upwind_adjoint(code, ptr(rows), ptr(off), int(rows.numel()), ptr(bg), ptr(e), ptr(coff),
                                                 int(bg.numel()), cells, ptr(lookup), ptr(w), ptr(v), ptr(ref), plan.hi,
                                                 H, a, b, 1e-3, lvl.dx, lvl.dy, 0, ptr(g_ref), ptr(lvl.scratch),
                                                 int(lvl.scratch.numel()), stream_handle(cuda_device)),
                   "sx_upwind_adjoint")
        assert torch.equal(_bits(got), _bits(ref))
    assert signs > 0


@pytest.mark.parametrize("dtype,tail", [(torch.float32, 1.0), (torch.float32, 1e-30), (torch.float32, 1e-41),
                                        (torch.float64, 1.0), (torch.float64, 1e-300)])
@pytest.mark.parametrize("a,b", [(1.0, 0.5), (-1.0, 0.5), (0.7, -0.3), (0.0, -0.0)])
def test_amr_steps(cuda_device, dtype, tail, a, b):
    """``tail`` scales some values so that the scaled, the float64 and the dividing forms run as well."""
    rng = np.random.default_rng(6)
    w, h, n = 150, 60, 5
    code = _lib.SX_F64 if dtype == torch.float64 else _lib.SX_F32
    c, f, act = _inputs(cuda_device, w, h, 1, dtype, "blocks", 5)
    c.copy_(_draw(rng, c.numel(), dtype, ZEROS + [tail]).view(c.shape))
    f.copy_(_draw(rng, f.numel(), dtype, ZEROS + [tail]).view(f.shape))
    args = (a, b, 1e-3, 0.013, 1.0 / 777, 0.0065, 0.5 / 777)
    want = _one_by_one(code, c, f, act, n, args)
    co, fo = torch.empty_like(c), torch.empty_like(f)
    _lib.check(_lib.load().sx_amr_steps_full(code, ptr(c), ptr(f), ptr(co), ptr(fo), ptr(act), w, h, 1, n, *args,
                                             stream_handle(cuda_device)), "sx_amr_steps_full")
    assert torch.equal(_bits(co), _bits(want[0])) and torch.equal(_bits(fo), _bits(want[1]))
