"""The transposed per-op stream where only the cotangent of f is wanted: the same
values as with dJ/dq, to the bit."""

import pytest
import torch

from lbm_jax_autodiff_gb300.core.streaming import stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("grid", [(5, 4, 6), (17, 9, 11)])
@pytest.mark.parametrize("periodic", [True, False])
def test_cotangent_of_f_alone(cuda, dtype, grid, periodic):
    gen = torch.Generator(device="cuda").manual_seed(2)
    f = torch.rand((19, *grid), generator=gen, device="cuda", dtype=dtype)
    q = torch.rand(f.shape, generator=gen, device="cuda", dtype=dtype) * 2.4 - 1.2
    g = torch.randn(f.shape, generator=gen, device="cuda", dtype=dtype)
    f1, f2, q2 = f.clone().requires_grad_(), f.clone().requires_grad_(), q.clone().requires_grad_()
    (alone,) = torch.autograd.grad(stream(f1, q, periodic), f1, g)
    both, gq = torch.autograd.grad(stream(f2, q2, periodic), (f2, q2), g)
    assert torch.equal(alone, both)
    assert (gq[q < 0] == 0).all() and gq.abs().max() > 0
