"""16-bit MRT steps on clamped sides and odd nz, above the small grids' form: their
boundary cells go through a call.  Random wall links on every edge and face and
across the storage-offset box, plain steps against sampled ones, whose
kernel has the same arithmetic inlined."""

import pytest
import torch

import lbm_jax_autodiff_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(81, 45, 43), (121, 1441, 1), (260, 200, 3)])
@pytest.mark.parametrize("storage", ["fp16", "bf16"])
@pytest.mark.parametrize("soft", [False, True])
def test_plain_and_sampled_steps(cuda, grid, storage, soft):
    n = 4
    gen = torch.Generator(device="cuda").manual_seed(grid[2])
    q = torch.rand((19, *grid), generator=gen, device="cuda")
    q = torch.where(torch.rand(q.shape, generator=gen, device="cuda") < 0.9,
                    torch.full_like(q, -1.0), q)
    q[0] = -1.0
    solid = torch.zeros(grid, dtype=torch.int32, device="cuda")
    solid[grid[0] // 3:grid[0] // 2, grid[1] // 4:grid[1] // 2] = 1
    por = torch.rand(grid, generator=gen, device="cuda") if soft else None
    states = []
    for every in (1, 0):
        sim = L.Simulation(*grid, 0.6, collision="mrt", storage=storage, periodic_yz=False,
                           use_smagorinsky=True)
        sim.set_mask(solid, q=q, porosity=por)
        f0 = sim.equilibrium_state().cuda()
        gen2 = torch.Generator(device="cuda").manual_seed(1)
        f0 = f0 * (1.0 + 0.01 * torch.randn(f0.shape, generator=gen2, device="cuda"))
        sim.set_state(f0.contiguous())
        sim.run(n, sample_every=every)
        states.append(sim.get_state().double())
        sim.close()
    # some 20 roundings a step of the arithmetic's type, and one of the storage's on
    # the deviation from the stored offset (a tenth of f at most)
    store = {"fp16": 0.1 * 2.0**-11, "bf16": 0.1 * 2.0**-8}[storage]
    bar = n * (20 * torch.finfo(torch.float32).eps + store) * states[0].abs().max()
    assert (states[0] - states[1]).abs().max() <= bar
