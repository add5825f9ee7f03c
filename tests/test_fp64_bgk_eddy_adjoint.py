"""FP64-storage gradients of BGK with the eddy viscosity, on both sides of the size
that chooses between the adjoint's register budgets, with cells inside and outside
the fixed-point range: dense cotangents of f_0 and q against FP32 storage."""

import pytest
import torch

import lbm_jax_autodiff_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(33, 17, 12), (80, 44, 46), (131, 64, 65)])
@pytest.mark.parametrize("porosity", ["hard", "soft"])
@pytest.mark.parametrize("dense", [1.0, 2.5])        # density of half of the domain
def test_gradient_against_fp32(cuda, grid, porosity, dense):
    n = 3

    def grads(storage):
        sim = L.Simulation(*grid, 0.6, collision="bgk", storage=storage, use_smagorinsky=True)
        sim.set_sphere(0.8, center=(0.013, 0.017, -0.011), kind="sigmoid", porosity=porosity,
                       sharpness=10.0)
        f0 = sim.equilibrium_state().cuda().double()
        gen = torch.Generator(device="cuda").manual_seed(1)
        f0 = f0 * (1.0 + 0.01 * torch.randn(f0.shape, generator=gen, device="cuda",
                                            dtype=torch.float64))
        f0[:, :grid[0] // 2] *= dense
        sim.set_state(f0.float().to(sim.dtype).contiguous())
        out = sim.cd_and_grad(n, checkpoint_every=n, dcd_dq=True, dcd_df0=True)
        sim.close()
        return out

    cd, dr, ex = grads("fp32")
    cd64, dr64, ex64 = grads("fp64")
    # some 20 roundings a step on values of order one (df0); dq and dr multiply
    # differences of populations a hundred times smaller than the populations
    eps = n * 20 * torch.finfo(torch.float32).eps
    assert abs(cd - cd64) <= 100 * eps * abs(cd64)
    err = (ex["dcd_df0"].double() - ex64["dcd_df0"]).abs().max()
    assert err <= 10 * eps * ex64["dcd_df0"].abs().max()
    err = (ex["dcd_dq"].double() - ex64["dcd_dq"]).abs().max()
    assert err <= 100 * eps * ex64["dcd_dq"].abs().max()
    assert abs(dr - dr64) <= 100 * eps * ex64["dcd_dq"].abs().sum()
