"""The forms of the fused step on both sides of the grid size that chooses
between them: a run whose every step is sampled (256-thread blocks of the general
kernel) against one without samples."""

import pytest
import torch

import lbm_jax_autodiff_gb300 as L

pytestmark = pytest.mark.gpu


# (152 * 1024 cells is the last size of the small grids' form)
@pytest.mark.parametrize("grid", [(3, 5, 7), (16, 8, 1), (33, 17, 15), (76, 64, 32), (77, 64, 32),
                                  (79, 45, 43), (81, 45, 43)])
@pytest.mark.parametrize("streaming,storage", [("ab", "fp32"), ("aa", "fp32"), ("ab", "fp16"),
                                               ("ab", "bf16")])
@pytest.mark.parametrize("porosity,periodic,collision", [("hard", True, "mrt"), ("soft", False, "bgk")])
def test_sampled_and_plain_steps(cuda, grid, streaming, storage, porosity, periodic, collision):
    n = 6
    states = []
    for every in (1, 0):
        sim = L.Simulation(*grid, 0.6, collision=collision, storage=storage,
                           periodic_yz=periodic or streaming == "aa",   # (in place: periodic only)
                           use_smagorinsky=True, guard="pre")
        sim.set_sphere(0.8, center=(0.013, 0.017, -0.011), kind="sigmoid", porosity=porosity,
                       sharpness=10.0)
        if streaming == "aa":
            sim.set_streaming("aa")
        f0 = sim.equilibrium_state().cuda().double()
        gen = torch.Generator(device="cuda").manual_seed(1)
        f0 = f0 * (1.0 + 0.01 * torch.randn(f0.shape, generator=gen, device="cuda",
                                            dtype=torch.float64))
        sim.set_state(f0.float().contiguous())
        sim.run(n, sample_every=every)
        states.append(sim.get_state().double())
        sim.close()
    # some 20 roundings a step of the arithmetic's type, and one of the storage's on
    # the deviation from the stored offset (a tenth of f at most)
    store = {"fp32": 0.0, "fp16": 0.1 * 2.0**-11, "bf16": 0.1 * 2.0**-8}[storage]
    bar = n * (20 * torch.finfo(torch.float32).eps + store) * states[0].abs().max()
    assert (states[0] - states[1]).abs().max() <= bar
