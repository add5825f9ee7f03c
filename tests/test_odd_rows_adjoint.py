"""FP32-arithmetic gradients on odd nz (rows start at either parity, pairs
straddle rows, an odd cell count leaves one cell without a partner): dense
cotangents of f_0 and q against the FP64-storage solver."""

import pytest
import torch

import lbm_jax_autodiff_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(24, 12, 5), (25, 13, 7), (24, 11, 13), (33, 17, 33), (9, 16, 3)])
@pytest.mark.parametrize("porosity,periodic,collision", [("hard", True, "mrt"), ("soft", False, "mrt"),
                                                         ("soft", True, "bgk")])
def test_gradient_on_odd_rows(cuda, grid, porosity, periodic, collision):
    n = 10

    def grads(storage):
        sim = L.Simulation(*grid, 0.6, collision=collision, storage=storage, periodic_yz=periodic,
                           use_smagorinsky=True)
        # off centre: a link of a centred sphere may cross at exactly half a link, where dq's
        # two one-sided formulas meet and q in FP32 and in FP64 may fall on different sides
        sim.set_sphere(0.8, center=(0.013, 0.017, -0.011), kind="sigmoid", porosity=porosity,
                       sharpness=10.0)
        f0 = sim.equilibrium_state().cuda().double()
        gen = torch.Generator(device="cuda").manual_seed(1)
        f0 = f0 * (1.0 + 0.01 * torch.randn(f0.shape, generator=gen, device="cuda",
                                            dtype=torch.float64))
        sim.set_state(f0.float().to(sim.dtype).contiguous())
        return sim.cd_and_grad(n, checkpoint_every=4, dcd_dq=True, dcd_df0=True)

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
