"""Kernels that are launched early read global memory by ordinary loads only.

Such a kernel is alive while the kernels before it write its inputs; the
read-only path (``__ldg``, or a ``const __restrict__`` parameter that the
compiler turns into it) is for data that nobody writes during the kernel.
"""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "subsetix_b200", "csrc")


def _block(src: str, at: int) -> str:
    """``src`` from ``at`` to the closing brace of the first block after it."""
    depth, i = 0, src.index("{", at)
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[at:j + 1]
    raise AssertionError("unbalanced braces")


def test_early_launched_kernels_use_ordinary_loads():
    seen = set()
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        src = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", src)
        functions = {m.group(1): _block(src, m.start()) for m in
                     re.finditer(r"(?:__global__|__device__)[^;{}=]*?\b(\w+)\s*\((?=[^;{]*\)\s*\{)", src)}
        kernels = set(re.findall(r"sx_launch_early\(\s*(\w+)", src))
        todo = list(kernels)
        reached = set()
        while todo:  # the kernels and the device functions of the file that they call
            name = todo.pop()
            if name in reached:
                continue
            reached.add(name)
            assert name in functions, f"{path}: {name} not found"
            todo += [f for f in functions if re.search(rf"\b{f}\b", functions[name]) and f != name]
        for name in reached:
            assert "__ldg" not in functions[name] and "ld.global.nc" not in functions[name], (path, name)
            assert not re.search(r"const\s+\w+(\s+\w+)?\s*\*\s*__restrict__", functions[name]), (path, name)
        for name in kernels:
            assert "sx_after_previous()" in functions[name], (path, name)
        seen |= kernels
    assert {"flat_step_kernel", "flat_adjoint_kernel", "index_copy_kernel", "segment_add_kernel",
            "run_block_mean_kernel", "run_block_mean_adj_kernel"} <= seen


@pytest.mark.gpu
def test_replayed_chain_equals_one_kernel_at_a_time(cuda_device, monkeypatch):
    """Chains of early-launched kernels on buffers that are used again and again, against the same launches run singly."""
    import torch

    from subsetix_b200 import _lib, adjoint
    from tests.test_gpu_adjoint import _hierarchy

    H, _ = _hierarchy()
    gen = torch.Generator(device="cuda").manual_seed(3)
    vel = torch.tensor([0.9, -0.4], dtype=torch.float64, device="cuda", requires_grad=True)
    u0 = [torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) for n in H.inner_cells]

    def run(graphs):
        u = [x.clone().requires_grad_() for x in u0]
        out = adjoint.advect_composite(vel, H, u, dt=2e-3, steps=40, checkpoint_every=8, graphs=graphs)
        grads = torch.autograd.grad(sum(x.square().sum() for x in out), [vel, *u])
        return [x.detach().clone() for x in (*out, *grads)]

    replayed = [run(True) for _ in range(25)]
    check = _lib.check
    monkeypatch.setattr(_lib, "check", lambda rc, what: (check(rc, what), torch.cuda.synchronize()))
    single = run(False)
    for got in replayed:
        for g, s in zip(got, single):
            assert torch.equal(g, s)
