"""Several AMR steps in one pass (sx_amr_steps_full) against the same steps one at a time: equal, bit for bit.

Widths around the edges of a warp's strip (64 columns in float32, 32 in
float64, less the columns worked out twice), odd widths, one column, heights
around a band of rows, every pair of velocity signs, spacings with and
without exact reciprocals, refined sets from empty to full.
"""

import pytest
import torch

from subsetix_b200 import _lib
from subsetix_b200._runtime import ptr, stream_handle

pytestmark = pytest.mark.gpu


def _inputs(device, width, height, batch, dtype, refined, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    c = torch.randn((batch, height, width), generator=g, dtype=torch.float64).to(dtype).to(device)
    f = torch.randn((batch, 2 * height, 2 * width), generator=g, dtype=torch.float64).to(dtype).to(device)
    if refined == "blocks":
        x, y = torch.arange(width), torch.arange(height)
        act = (((x[None, :] // 70) + (y[:, None] // 5)) % 2).to(torch.int8).expand(batch, -1, -1).contiguous()
    else:
        act = (torch.rand((batch, height, width), generator=g) < refined).to(torch.int8)
    return c, f, act.to(device)


def _one_by_one(code, c, f, act, n, args):
    b, h, w = c.shape
    lib = _lib.load()
    for _ in range(n):
        co, fo = torch.empty_like(c), torch.empty_like(f)
        _lib.check(lib.sx_amr_step_full(code, ptr(c), ptr(f), ptr(co), ptr(fo), ptr(act), w, h, b, *args,
                                        stream_handle(c.device)), "sx_amr_step_full")
        c, f = co, fo
    return c, f


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("width,height,batch", [(1, 1, 1), (2, 3, 2), (31, 9, 1), (58, 17, 1), (63, 8, 2), (64, 40, 1),
                                                (65, 7, 1), (122, 70, 1), (123, 33, 3), (300, 129, 1)])
@pytest.mark.parametrize("a,b", [(1.0, 0.5), (-1.0, 0.5), (0.7, -0.3), (-0.2, -0.9), (0.0, -0.0)])
def test_steps_equal_single_steps(cuda_device, dtype, width, height, batch, a, b):
    code = _lib.SX_F64 if dtype == torch.float64 else _lib.SX_F32
    lib = _lib.load()
    for n, refined, dx in ((2, 0.5, 1.0 / 64), (3, "blocks", 0.013), (4, 0.0, 1.0 / 64), (5, "blocks", 1.0 / 64),
                           (5, 1.0, 0.013), (5, 0.02, 1.0 / 64)):
        c, f, act = _inputs(cuda_device, width, height, batch, dtype, refined, 7 * n + width)
        args = (a, b, 0.2 * dx, dx, 1.5 * dx if dx == 0.013 else dx, dx / 2, dx / 2)
        want = _one_by_one(code, c, f, act, n, args)
        co, fo = torch.full_like(c, float("nan")), torch.full_like(f, float("nan"))
        _lib.check(lib.sx_amr_steps_full(code, ptr(c), ptr(f), ptr(co), ptr(fo), ptr(act), width, height, batch, n,
                                         *args, stream_handle(cuda_device)), "sx_amr_steps_full")
        assert torch.equal(co, want[0]), (n, refined)
        assert torch.equal(fo, want[1]), (n, refined)


@pytest.mark.parametrize("dtype,values", [
    (torch.float32, (0.0, -0.0, 1.0, 1e-22, 1e-24, 3e-30, 1e-41, 2e38)),
    (torch.float32, (0.5, 3e38, float("inf"), float("nan"), 1e-38)),
    (torch.float64, (0.0, -0.0, 1.0, 1e-252, 1e-254, 1e-300, 5e-324, 1e308)),
    (torch.float64, (0.5, 1.7e308, float("inf"), float("nan"), 1e-308))])
@pytest.mark.parametrize("dx", [0.013, 1.0 / 777, 1e-25, 3e7])
def test_steps_with_small_large_and_special_values(cuda_device, dtype, values, dx):
    """Quotients that leave the range of the division by a known divisor, mixed with ordinary ones."""
    w, h, n = 150, 60, 5
    g = torch.Generator(device="cpu").manual_seed(11)
    code = _lib.SX_F64 if dtype == torch.float64 else _lib.SX_F32
    c, f, act = _inputs(cuda_device, w, h, 1, dtype, 0.4, 5)
    pool = torch.tensor(values, dtype=dtype)
    for t, share in ((c, 0.3), (f, 0.02)):
        which = torch.rand(t.shape, generator=g) < share
        t.copy_(torch.where(which, pool[torch.randint(len(values), t.shape, generator=g)], t.cpu()))
        t[:, : t.shape[1] // 3] *= 1e-30
    args = (1.0, -0.5, 0.1, dx, dx, dx / 2, dx / 2)
    want = _one_by_one(code, c, f, act, n, args)
    co, fo = torch.empty_like(c), torch.empty_like(f)
    _lib.check(_lib.load().sx_amr_steps_full(code, ptr(c), ptr(f), ptr(co), ptr(fo), ptr(act), w, h, 1, n, *args,
                                             stream_handle(cuda_device)), "sx_amr_steps_full")
    for got, exp in ((co, want[0]), (fo, want[1])):
        torch.testing.assert_close(got, exp, rtol=0.0, atol=0.0, equal_nan=True)


@pytest.mark.parametrize("offset", [1, 2])
def test_steps_on_unaligned_arrays(cuda_device, offset):
    w, h, n = 66, 20, 5
    c, f, act = _inputs(cuda_device, w, h, 1, torch.float32, 0.3, 3)
    args = (1.0, 0.5, 0.01, 0.1, 0.1, 0.05, 0.05)
    want = _one_by_one(_lib.SX_F32, c, f, act, n, args)

    def moved(t):
        x = torch.empty(t.numel() + offset, dtype=t.dtype, device=t.device)[offset:].view(t.shape)
        return x.copy_(t)

    ins = [moved(t) for t in (c, f, act)]
    outs = [moved(c), moved(f)]
    _lib.check(_lib.load().sx_amr_steps_full(_lib.SX_F32, ptr(ins[0]), ptr(ins[1]), ptr(outs[0]), ptr(outs[1]),
                                             ptr(ins[2]), w, h, 1, n, *args, stream_handle(cuda_device)),
               "sx_amr_steps_full")
    assert torch.equal(outs[0], want[0]) and torch.equal(outs[1], want[1])


@pytest.mark.parametrize("steps,every", [(7, 3), (13, 6), (23, 11), (5, 1), (4, 10)])
@pytest.mark.parametrize("graph", [False, True])
def test_runs_in_any_portions_agree(cuda_device, steps, every, graph):
    from subsetix_b200.subsetix_amr2.fused import FusedTwoLevelAMR

    x = torch.linspace(0, 1, 48, device=cuda_device)
    u0 = torch.exp(-((x[None, :] - 0.4) ** 2 + (x[:, None] - 0.5) ** 2) / 0.02)
    one, many, two = (FusedTwoLevelAMR(u0, velocity=(0.8, -0.6), cfl=0.5, refine_threshold=0.02) for _ in range(3))
    for _ in range(steps):
        one.step(every)
    many.run(steps, every, graph=graph)
    two.run(steps // 2, every, graph=graph)
    two.run(steps - steps // 2, every, graph=graph)
    for eng in (many, two):
        assert (eng.step_count, eng.time) == (one.step_count, one.time)
        assert torch.equal(eng.coarse_values, one.coarse_values)
        assert torch.equal(eng.fine_values, one.fine_values)
        assert torch.equal(eng.actions, one.actions)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("padding", [0, 1, 2, 3, 8, 9])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("width,height,batch", [(1, 1, 1), (1, 40, 1), (28, 16, 1), (29, 17, 2), (57, 33, 1), (130, 50, 1)])
def test_tag_and_grade_against_dense_masks(cuda_device, dtype, padding, mode, width, height, batch):
    """Fields of small whole numbers, whose gradients are exact: tags and actions equal those of dense masks."""
    g = torch.Generator(device="cpu").manual_seed(width + padding)
    u = torch.randint(0, 20, (batch, height, width), generator=g).clamp_max(1).sub(1).mul(-4).to(torch.float64)
    gx, gy = torch.zeros_like(u), torch.zeros_like(u)
    if width > 1:
        gx[:, :, 1:-1] = (u[:, :, 2:] - u[:, :, :-2]) / 2
        gx[:, :, 0], gx[:, :, -1] = u[:, :, 1] - u[:, :, 0], u[:, :, -1] - u[:, :, -2]
    if height > 1:
        gy[:, 1:-1] = (u[:, 2:] - u[:, :-2]) / 2
        gy[:, 0], gy[:, -1] = u[:, 1] - u[:, 0], u[:, -1] - u[:, -2]
    tag = (gx * gx + gy * gy) >= 4.0
    p, pool = padding, torch.nn.functional.max_pool2d
    t = tag.to(torch.float32)[:, None]
    if p == 0:
        on = t
    elif mode == 1:
        on = pool(t, 2 * p + 1, stride=1, padding=p)
    else:
        on = torch.maximum(pool(t, (1, 2 * p + 1), stride=1, padding=(0, p)),
                           pool(t, (2 * p + 1, 1), stride=1, padding=(p, 0)))
    v = u.to(dtype).to(cuda_device).contiguous()
    tags = torch.full((batch, height, width), 7, dtype=torch.uint8, device=cuda_device)
    act = torch.full((batch, height, width), 7, dtype=torch.int8, device=cuda_device)
    code = _lib.SX_F64 if dtype == torch.float64 else _lib.SX_F32
    _lib.check(_lib.load().sx_amr_regrid_full(code, ptr(v), ptr(tags), ptr(act), width, height, batch, 2.0, padding,
                                              mode, stream_handle(cuda_device)), "sx_amr_regrid_full")
    assert torch.equal(tags.cpu().bool(), tag)
    assert torch.equal(act.cpu().bool(), on[:, 0].bool())
