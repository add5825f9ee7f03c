"""The geometry of a handle: records built straight from the sphere against
those built from the dense solid and q of the same sphere, for bodies that
touch wrapped and clamped domain edges, and buffers reused and grown over a
sequence of radii against a fresh handle.  Same cells, links and steps, to
the bit."""

import pytest
import torch

import lbm_jax_autodiff_gb300 as L
from lbm_jax_autodiff_gb300.geometry.primitives import create_sphere

pytestmark = pytest.mark.gpu

BODIES = [
    # grid, periodic, centre, radius
    ((16, 12, 10), True, (0.0, 0.0, 0.0), 0.9),
    ((16, 12, 10), True, (0.3, 1.5, -1.6), 1.1),       # second fluid cells across the y / z wrap
    ((15, 11, 9), False, (-3.4, -1.7, 1.5), 0.8),      # clamped edges and the x = 0 face, odd sizes
    ((40, 8, 6), True, (3.5, 0.0, 0.0), 1.4),          # x = nx - 1 face, few cells across
    ((33, 70, 130), True, (0.0, 0.5, 0.0), 1.0),       # many blocks of the pair list's scan
]


def _sim(grid, storage, periodic):
    return L.Simulation(*grid, 0.7, collision="mrt", storage=storage, periodic_yz=periodic)


def _three_steps(sim, f0):
    sim.set_state(f0)
    s = sim.run(3, sample_every=1)
    return sim.get_state(), s


@pytest.mark.parametrize("grid,periodic,center,radius", BODIES)
@pytest.mark.parametrize("storage", ["fp32", "fp64", "bf16"])
def test_sphere_equals_its_dense_fields(cuda, grid, periodic, center, radius, storage):
    dt = torch.float64 if storage == "fp64" else torch.float32
    solid, q = create_sphere(*grid, center, radius, dtype=dt)
    a, b = _sim(grid, storage, periodic), _sim(grid, storage, periodic)
    a.set_sphere(radius, center=center, kind="dist")
    b.set_mask(solid.to(torch.int32), q=q)
    assert a.link_count == b.link_count and a.projected_area == b.projected_area
    f0 = a.equilibrium_state()
    (fa, sa), (fb, sb) = _three_steps(a, f0), _three_steps(b, f0)
    assert torch.equal(fa, fb) and torch.equal(sa, sb)


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
def test_rebuilt_geometry_equals_a_fresh_one(cuda, storage):
    grid = (48, 24, 24)
    one = _sim(grid, storage, True)
    f0 = one.equilibrium_state()
    for radius, porosity in ((0.3, "hard"), (0.9, "soft"), (0.35, "soft"), (1.2, "hard")):
        kw = dict(kind="sigmoid", porosity=porosity, sharpness=10.0)
        one.set_sphere(radius, **kw)
        two = _sim(grid, storage, True)
        two.set_sphere(radius, **kw)
        assert one.link_count == two.link_count and one.projected_area == two.projected_area
        (f1, s1), (f2, s2) = _three_steps(one, f0), _three_steps(two, f0)
        assert torch.equal(f1, f2) and torch.equal(s1, s2)
        one.set_state(f0)
        two.set_state(f0)
        assert one.cd_and_grad(6) == two.cd_and_grad(6)
    none = _sim(grid, storage, True)
    none.set_mask(torch.zeros(grid, dtype=torch.int32, device="cuda"))
    assert none.link_count == (0, 0) and none.projected_area == 0.0
