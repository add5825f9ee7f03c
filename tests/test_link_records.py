"""Boundary-cell records with every kind of link: random wall distances on
all cells and directions (q >= 0.5, q < 0.5, q > 1, ties at 0, 0.5 and 1, no
wall), so links meet x faces, clamped and wrapped y / z edges, and the second
fluid cell of a q < 0.5 link lies beyond the domain edge (streaming.py:148-183
wraps it in every axis).  Steps and the transposed step against the oracle."""

import pytest
import torch

import lbm_jax_autodiff_gb300 as L
from oracle import drivers, ops

pytestmark = pytest.mark.gpu

GRIDS = [(5, 4, 6, True), (7, 5, 8, False), (6, 3, 7, True), (3, 6, 4, False), (4, 33, 10, True)]


def _inputs(nx, ny, nz, dt):
    gen = torch.Generator().manual_seed(nx * 100 + ny * 10 + nz)
    q = torch.rand((19, nx, ny, nz), generator=gen, dtype=torch.float64) * 1.2
    ties = torch.tensor([0.0, 0.5, 1.0], dtype=torch.float64)
    pick = torch.randint(0, 12, q.shape, generator=gen)
    q = torch.where(pick < 3, ties[pick.clamp(max=2)], q)
    q = torch.where(pick >= 8, torch.full_like(q, -1.0), q)
    q[0] = -1.0
    solid = (torch.rand((nx, ny, nz), generator=gen) < 0.2).to(torch.int32)
    f = drivers.initial_state(nx, ny, nz, 0.05, torch.float64)
    f = f * (1.0 + 0.02 * torch.randn(f.shape, generator=gen, dtype=torch.float64))
    return f.to(dt), q.to(dt), solid


@pytest.mark.parametrize("nx,ny,nz,periodic", GRIDS)
@pytest.mark.parametrize("storage", ["fp32", "fp64"])
@pytest.mark.parametrize("streaming", ["ab", "aa"])
def test_steps_with_random_links(cuda, nx, ny, nz, periodic, storage, streaming):
    if streaming == "aa" and not periodic:
        pytest.skip("in-place streaming needs periodic y / z")
    dt = torch.float64 if storage == "fp64" else torch.float32
    f0, q, solid = _inputs(nx, ny, nz, dt)
    cfg = drivers.StepConfig(tau=0.8, inlet=(0.05, 0.0, 0.0), periodic_yz=periodic)
    f, _, _ = drivers.run(f0.double(), q.double(), cfg, 3, solid=solid)
    sim = L.Simulation(nx, ny, nz, 0.8, collision="bgk", storage=storage, periodic_yz=periodic)
    sim.set_streaming(streaming)
    sim.set_mask(solid.cuda(), q=q.cuda())
    sim.set_state(f0.cuda())
    s = sim.run(3, sample_every=1)
    # a step's sums of 19 populations of a cell (rho ~ 1) round by at most 20 ulp
    tol = 3 * 20 * torch.finfo(dt).eps
    assert (sim.get_state().cpu().double() - f).abs().max() <= tol
    f2, fp, _ = drivers.run(f0.double(), q.double(), cfg, 2, solid=solid)
    force = ops.momentum_exchange(fp, f2, q.double())
    links = int((q[1:] >= 0).sum())
    assert (s[1, :3].cpu() - force).abs().max() <= links * tol


@pytest.mark.parametrize("nx,ny,nz,periodic", GRIDS)
def test_transposed_steps_with_random_links(cuda, nx, ny, nz, periodic):
    f0, q, solid = _inputs(nx, ny, nz, torch.float64)
    # (jax's and this solver's half cotangent at a tie of clip is autograd's in the oracle;
    # the functional API holds a velocity tuple in FP32, so it gets an FP64 tensor)
    fo, qo = f0.clone().requires_grad_(), q.clone().requires_grad_()
    cfg = drivers.StepConfig(tau=0.8, inlet=(0.05, 0.0, 0.0), periodic_yz=periodic)
    out, _, _ = drivers.run(fo, qo, cfg, 3, solid=solid)
    gen = torch.Generator().manual_seed(5)
    g = torch.randn(out.shape, generator=gen, dtype=torch.float64)
    gf, gq = torch.autograd.grad(out, (fo, qo), g)
    fc, qc = f0.cuda().requires_grad_(), q.cuda().requires_grad_()
    res = L.simulate(L.LBMState(fc, solid.cuda(), qc),
                     L.LBMParams(tau=0.8, periodic_yz=periodic,
                                 inlet_velocity=torch.tensor([0.05, 0.0, 0.0],
                                                             dtype=torch.float64)), 3)
    hf, hq = torch.autograd.grad(res.f, (fc, qc), g.cuda())
    # sums of some dozens of terms a step, in 64 bits
    assert (hf.cpu() - gf).abs().max() <= 1e-12 * gf.abs().max()
    links = q >= 0
    assert (hq.cpu() - gq)[links].abs().max() <= 1e-12 * gq.abs().max()
