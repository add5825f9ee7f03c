"""The per-op momentum exchange of a field with an infinite or NaN population at a
link: the two entry points sum the same terms."""

import ctypes
import math

import pytest
import torch

from lbm_jax_autodiff_gb300 import _native as nat
from lbm_jax_autodiff_gb300.core.forces import momentum_exchange

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
@pytest.mark.parametrize("direction", [1, 4, 5, 9, 12, 17])
def test_nonfinite_population_at_a_link(cuda, dtype, value, direction):
    dims = (8, 9, 10)
    f = torch.full((19, *dims), 0.05, dtype=dtype, device="cuda")
    q = torch.full_like(f, -1.0)
    q[direction, 3, 4, 5] = 0.25
    q[7, 5, 2, 1] = 0.75
    f[direction, 3, 4, 5] = value
    force = momentum_exchange(f, f, q)
    other = torch.zeros(3, dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    nat.call("lbm_momentum_exchange_noalloc", nat.LBM_F64 if dtype == torch.float64 else nat.LBM_F32,
             p(f), p(f), p(q), p(other), *dims,
             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert torch.equal(torch.nan_to_num(force, nan=7.0), torch.nan_to_num(other.to(dtype), nan=7.0))
    # 0 * inf is NaN on the axes that the direction has no component along
    assert not force.isfinite().any()
