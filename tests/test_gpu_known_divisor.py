"""The flat step with a known divisor against divisions: fields whose quotients leave its range, mixed with ordinary ones.

The generic kernel divides every difference; results must be equal, bit for
bit up to the sign of zero.
"""

import numpy as np
import pytest
import torch

from subsetix_b200 import _core
from tests.test_gpu_flat_stencil import _geometries, _plan

pytestmark = pytest.mark.gpu

ORDINARY = (1.0, -0.3, 0.7)
F32 = ((0.0, -0.0, 1e-29, 1e-31, 3e-38, 1e-42, 1e18, 1e19, 2e38) + ORDINARY,
       (float("inf"), float("nan"), 3.4e38) + 8 * ORDINARY)
F64 = ((0.0, -0.0, 1e-270, 1e-272, 1e-307, 5e-324, 1e270, 1e272, 1e308) + ORDINARY,
       (float("inf"), float("nan"), 1.7e308) + 8 * ORDINARY)


@pytest.mark.parametrize("dtype,values", [(torch.float32, v) for v in F32] + [(torch.float64, v) for v in F64])
@pytest.mark.parametrize("dx,dy", [(1e-2, 1.0 / 777), (3.3e5, 0.1), (1e-17, 1e-2), (1e-25, 3e7), (0.75, 1.0)])
def test_flat_step_equals_divisions(cuda_device, dtype, values, dx, dy):
    rng = np.random.default_rng(9)
    for h in _geometries():
        (b, e, off, rows), H, coff, cells, lookup, plan = _plan(h, cuda_device)
        picked = rng.choice(np.asarray(values), cells)
        v = torch.as_tensor(np.where(rng.random(cells) < 0.5, picked, rng.standard_normal(cells)),
                            device=cuda_device).to(dtype)
        for a_, b_ in ((0.6, 0.3), (-0.4, 0.9), (0.6, -0.3)):
            ref, got = torch.empty_like(v), torch.empty_like(v)
            _core.upwind(rows, off, b, e, coff, cells, lookup, v, ref, plan.hi, H, a_, b_, 1e-3, dx, dy, False,
                         cuda_device)
            plan.step(v, got, a_, b_, 1e-3, dx, dy, cuda_device)
            torch.testing.assert_close(got, ref, rtol=0.0, atol=0.0, equal_nan=True)
