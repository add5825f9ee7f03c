"""FP64-storage steps on cells inside and outside the fixed-point range
(csrc/fixed64.cuh), side by side in one grid: densities from 0.3 to 1000,
fast cells, empty directions, NaN, solid and porous cells, guards.  One step
against the FP64 oracle."""

import pytest
import torch

import lbm_jax_autodiff_gb300 as L
from oracle import drivers, ops

pytestmark = pytest.mark.gpu
DT = torch.float64


def _cells(nx, ny, nz, nan):
    gen = torch.Generator().manual_seed(nx)
    rho = torch.tensor([1.0, 0.9, 1.3, 0.55, 1.9, 0.3, 2.5, 1000.0], dtype=DT)
    rho = rho[torch.randint(0, 8, (nx, ny, nz), generator=gen)]
    u = 0.12 * torch.randn((3, nx, ny, nz), generator=gen, dtype=DT)
    f = ops.equilibrium(rho, u)
    f = f * (1.0 + 0.1 * torch.randn(f.shape, generator=gen, dtype=DT))
    f = torch.where(torch.rand(f.shape, generator=gen) < 0.02, torch.zeros_like(f), f)
    if nan:
        f[3, 2, 1, 1] = float("nan")
    return f


@pytest.mark.parametrize("collision", ["bgk", "mrt"])
@pytest.mark.parametrize("smag", [False, True])
@pytest.mark.parametrize("solid_kind,guard,nan", [("none", "off", True), ("hard", "pre", False),
                                                  ("soft", "post", False)])
@pytest.mark.parametrize("tau", [0.501, 0.9])
def test_one_step(cuda, collision, smag, solid_kind, guard, nan, tau):
    nx, ny, nz = 11, 9, 10
    f0 = _cells(nx, ny, nz, nan)
    gen = torch.Generator().manual_seed(7)
    solid = (torch.rand((nx, ny, nz), generator=gen) < 0.2).to(torch.int32)
    por = torch.rand((nx, ny, nz), generator=gen, dtype=DT) * 1.3 - 0.1    # also beyond [0, 1]
    q = torch.full((19, nx, ny, nz), -1.0, dtype=DT)
    cfg = drivers.StepConfig(tau=tau, inlet=(0.05, 0.0, 0.0), collision=collision, guard=guard,
                             smagorinsky_cs=0.1 if smag else None)
    kw = {}
    sim = L.Simulation(nx, ny, nz, tau, collision=collision, storage="fp64", use_smagorinsky=smag,
                       guard=guard)
    if solid_kind == "soft":
        kw["porosity"] = por
        sim.set_mask(torch.zeros_like(solid).cuda(), q=q.cuda(), porosity=por.cuda())
    else:
        kw["solid"] = solid if solid_kind == "hard" else torch.zeros_like(solid)
        sim.set_mask(kw["solid"].cuda(), q=q.cuda())
    f_ref = drivers.initial_state(nx, ny, nz, 0.05, DT)
    want, _, _ = drivers.step(f0, q, cfg, f_ref=f_ref, **kw)
    sim.set_state(f0.cuda())
    sim.run(1)
    got = sim.get_state().cpu()
    # a collision sums 19 populations with factors up to 30 and divides by the density:
    # some hundred ulp of the cell's largest value
    scale = f0.nan_to_num().abs().amax(0).clamp(min=1.0).expand(19, nx, ny, nz).contiguous()
    scale = ops.zou_he_outlet(ops.zou_he_inlet(ops.stream(scale, q), (0.0, 0.0, 0.0)))
    scale = torch.maximum(scale.abs().amax(0), torch.ones(1, dtype=DT))
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    err = ((got - want).abs() / scale).nan_to_num()
    assert err.max() <= 400 * torch.finfo(DT).eps, err.max()
