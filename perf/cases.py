"""The calls whose speed counts: what a user of the solver has it do.

Each case is one call sequence through the public entry points, over the sizes
that the repository's configurations, tests and benchmark use.  A case is a
dict of plain values; ``kind`` names the entry point:

  run       Simulation.set_state / run / get_state: a forward simulation
  grad      Simulation.set_sphere / cd_and_grad: one shape-gradient evaluation
            of an optimisation loop (each iteration has a new radius)
  simulate  state.simulate and its backward for f_0 and q (the functional API)
  ops       one time step composed of the per-op functions, and its backward
  batch     Batch.set_spheres / set_equilibrium / optimize: one optimisation
            iteration over many domains

``exact`` restates the same calculation in plain torch in 64 bits.
"""

import math

import torch

from lbm_jax_autodiff_gb300 import Simulation
from lbm_jax_autodiff_gb300.batch import Batch
from lbm_jax_autodiff_gb300.core.boundary import zou_he_inlet, zou_he_outlet
from lbm_jax_autodiff_gb300.core.collision import mrt, smagorinsky_tau
from lbm_jax_autodiff_gb300.core.forces import drag_coefficient, momentum_exchange
from lbm_jax_autodiff_gb300.core.streaming import stream
from lbm_jax_autodiff_gb300.geometry.primitives import create_sphere
from lbm_jax_autodiff_gb300.geometry.smooth import soft_bounce_back
from lbm_jax_autodiff_gb300.state import LBMParams, LBMState, simulate

U = 0.05

# defaults of the fields that a case leaves out
_DEFAULTS = dict(storage="fp32", collision="mrt", smag=False, guard="off", periodic=True,
                 geometry="sphere", mask="dist", q_mode="bouzidi", porosity="hard", alpha=20.0,
                 radius=0.5, tau=0.548, sample=0, checkpoint=0, streaming="ab", dense=False,
                 count=0)


def _full(case):
    return {**_DEFAULTS, **case}


def listed():
    return [
        # the smallest domain in use: the plane-channel validation run (walls at y = 0 and
        # ny - 1, parabolic inlet), where launches and latency count
        dict(name="channel_64x21x8", kind="run", nx=64, ny=21, nz=8, steps=100, tau=0.8,
             collision="bgk", geometry="channel"),
        # a small sphere domain, Cd sampled now and then, as in the optimisation examples
        dict(name="sphere_64x32x32", kind="run", nx=64, ny=32, nz=32, steps=100, sample=25,
             guard="pre"),
        # double precision: the mode that the other storages are validated against
        dict(name="sphere_96x48x48_fp64", kind="run", nx=96, ny=48, nz=48, steps=60, sample=20,
             storage="fp64", guard="pre"),
        # the drag-convergence run at its full resolution, with the eddy viscosity
        dict(name="sphere_256x128x128", kind="run", nx=256, ny=128, nz=128, steps=100, sample=50,
             smag=True, guard="pre"),
        # the same with 16-bit populations
        dict(name="sphere_256x128x128_fp16", kind="run", nx=256, ny=128, nz=128, steps=100,
             sample=50, smag=True, guard="pre", storage="fp16"),
        # one iteration of a shape optimisation with a sigmoid-soft sphere, at the
        # optimisation example's size, with the dense dCd/dq and dCd/df_0
        dict(name="grad_96x48x48_soft", kind="grad", nx=96, ny=48, nz=48, steps=200,
             mask="sigmoid", porosity="soft", radius=0.5, tau=0.536, dense=True),
        # the shape gradient at full resolution; half of the window's forward steps are
        # recomputed, as in the 2000-step window that does not fit the device
        dict(name="grad_256x128x128", kind="grad", nx=256, ny=128, nz=128, steps=60, smag=True,
             checkpoint=30, dense=True),
        # the same with 16-bit populations
        dict(name="grad_256x128x128_fp16", kind="grad", nx=256, ny=128, nz=128, steps=60,
             smag=True, checkpoint=30, storage="fp16"),
        # the gradient check in double precision
        dict(name="grad_64x32x32_fp64", kind="grad", nx=64, ny=32, nz=32, steps=40,
             mask="sigmoid", storage="fp64", dense=True, checkpoint=20),
        # the functional API, differentiated for the initial state and the wall distances,
        # on a ragged domain with clamped sides
        dict(name="simulate_101x51x47", kind="simulate", nx=101, ny=51, nz=47, steps=80, smag=True,
             periodic=False),
        # a step written with the per-op functions, and its backward
        dict(name="ops_128x64x64", kind="ops", nx=128, ny=64, nz=64, steps=1, smag=True,
             porosity="soft"),
        # one optimisation iteration over domains of mixed sizes and boundary modes
        dict(name="batch_12", kind="batch", nx=128, ny=64, nz=64, count=12, steps=300,
             checkpoint=75),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "grad", "grad", "simulate", "ops", "batch"])
    nx, ny, nz = _log(rng, 32, 256), _log(rng, 16, 128), _log(rng, 16, 128)
    if rng.random() < 0.5:      # usual domains have nz a multiple of 8, ragged ones do not
        nz = max(16, nz // 8 * 8)
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, radius=rng.uniform(0.35, 0.7),
             tau=rng.uniform(0.53, 0.7), smag=rng.random() < 0.5,
             collision=rng.choice(["mrt", "mrt", "bgk"]))
    cells = nx * ny * nz
    if kind == "run":
        c["storage"] = rng.choice(["fp32", "fp32", "fp64", "fp16", "bf16"])
        c["steps"] = min(_log(rng, 20, 200), 100 * 256 * 128 * 128 // cells)
        c["sample"] = rng.choice([0, 10])
        c["guard"] = rng.choice(["off", "pre", "post"])
        c["periodic"] = rng.random() < 0.75
        if c["storage"] == "fp32" and c["periodic"] and rng.random() < 0.25:
            c["streaming"] = "aa"
        if rng.random() < 0.2:
            c.update(geometry="channel", tau=0.8)
        elif rng.random() < 0.4:
            c.update(mask="sigmoid", porosity="soft")
        if c["storage"] == "fp64":
            c["steps"] = min(c["steps"], max(8, 24_000_000 // cells))
    elif kind == "grad":
        c["storage"] = rng.choice(["fp32", "fp32", "fp32", "fp64", "fp16", "bf16"])
        c["steps"] = min(_log(rng, 20, 200), max(20, 60 * 256 * 128 * 128 // cells))
        c["q_mode"] = rng.choice(["bouzidi", "bouzidi", "halfway"])
        c["mask"] = rng.choice(["dist", "sigmoid"])
        if c["mask"] == "sigmoid" and rng.random() < 0.5:
            c["porosity"] = "soft"
        if rng.random() < 0.5:
            c["checkpoint"] = max(4, c["steps"] // 2)
        c["dense"] = rng.random() < 0.5
        if c["storage"] == "fp64":
            c["steps"] = min(c["steps"], max(8, 12_000_000 // cells))
    elif kind == "simulate":
        c["steps"] = min(_log(rng, 20, 100), max(20, 30 * 256 * 128 * 128 // cells))
        c["periodic"] = rng.random() < 0.5
        c["storage"] = "fp32"
    elif kind == "ops":
        c.update(steps=1, collision="mrt", smag=True, porosity="soft")
    else:
        c.update(nx=128, ny=64, nz=64, count=rng.randint(3, 16), smag=False, collision="mrt",
                 steps=_log(rng, 50, 250))
        c["checkpoint"] = max(10, c["steps"] // 4)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_EX = (0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0)
_EY = (0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 0, 0, 0, 0, 1, -1, 1, -1)
_EZ = (0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1)
_OPP = (0, 2, 1, 4, 3, 6, 5, 10, 9, 8, 7, 14, 13, 12, 11, 18, 17, 16, 15)


def _f32(v):
    return float(torch.tensor(v, dtype=torch.float32))


# the lattice weights and relaxation rates as the solver holds them by default
_W = tuple(_f32(v) for v in (1 / 3,) + (1 / 18,) * 6 + (1 / 36,) * 12)
_RATE = tuple(_f32(v) for v in (0, 1.19, 1.4, 0, 1.2, 0, 1.2, 0, 1.2, 0, 1.4, 0, 1.4, 0, 0, 0,
                                1.98, 1.98, 1.98))


def _equilibrium(rho, ux, uy, uz):
    usq = ux * ux + uy * uy + uz * uz
    out = []
    for i in range(19):
        eu = _EX[i] * ux + _EY[i] * uy + _EZ[i] * uz
        out.append(_W[i] * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * usq))
    return torch.stack(out)


def _initial(c, seed, dtype, ux):
    """A developed state: the free stream with smooth density and velocity waves."""
    gen = torch.Generator().manual_seed(seed)
    ph = torch.rand(4, 3, generator=gen) * (2 * math.pi)
    amp = 0.02 * (0.5 + torch.rand(4, generator=gen))
    axes = [torch.arange(n, device="cuda", dtype=torch.float64) * (2 * math.pi / n)
            for n in (c["nx"], c["ny"], c["nz"])]
    x, y, z = (a.reshape([-1 if k == j else 1 for k in range(3)]) for j, a in enumerate(axes))
    waves = [float(amp[k]) * torch.sin(x + float(ph[k, 0])) * torch.cos(y + float(ph[k, 1])) *
             torch.cos(z + float(ph[k, 2])) for k in range(4)]
    f = _equilibrium(1.0 + 0.1 * waves[0], ux * (1.0 + waves[1]), U * waves[2], U * waves[3])
    return f.to(dtype).contiguous()


def _dtype(c):
    return torch.float64 if c["storage"] == "fp64" else torch.float32


def _radius(c, seed):
    return _f32(c["radius"] * (1.0 + 0.02 * math.sin(1.0 + seed)))


def _walls(c):
    solid = torch.zeros((c["nx"], c["ny"], c["nz"]), dtype=torch.int32, device="cuda")
    solid[:, 0] = 1
    solid[:, -1] = 1
    return solid


def _profile(c, seed):
    """Parabolic inlet between the channel's walls, (3, ny, nz)."""
    s = torch.arange(c["ny"], device="cuda", dtype=torch.float64) - 0.5
    h = float(c["ny"] - 2)
    p = U * (1.0 + 0.02 * math.sin(1.0 + seed)) * 4.0 * s * (h - s) / (h * h)
    p[0] = p[-1] = 0.0
    u = torch.zeros((3, c["ny"], c["nz"]), device="cuda", dtype=torch.float64)
    u[0] = p[:, None]
    return u


def _cotangent(c, seed, dtype):
    gen = torch.Generator(device="cuda").manual_seed(1000 + seed)
    return torch.randn((19, c["nx"], c["ny"], c["nz"]), generator=gen, device="cuda",
                       dtype=torch.float32).to(dtype)


def _batch(c, seed):
    """(instances, spheres): the three grids of the batched workload in turn, radius 4 to 8
    cells per 32, modes and alpha in turn, tau from Re 50."""
    gen = torch.Generator().manual_seed(seed)
    radii = (4.0 + 4.0 * torch.rand(c["count"], generator=gen)).tolist()
    grids = [(c["nx"], c["ny"], c["nz"]), (c["nx"] * 3 // 4, c["ny"] * 3 // 4, c["nz"] * 3 // 4),
             (c["nx"] // 2, c["ny"] // 2, c["nz"] // 2)]
    instances, spheres = [], []
    for i in range(c["count"]):
        nx, ny, nz = grids[i % 3]
        cells = radii[i] * ny / 32.0
        instances.append(dict(nx=nx, ny=ny, nz=nz, tau=3.0 * U * 2.0 * cells / 50.0 + 0.5,
                              inlet_velocity=(U, 0.0, 0.0)))
        spheres.append(dict(radius=cells / (ny / 4.0), sharpness=(5.0, 10.0, 20.0)[i // 3 % 3],
                            kind="sigmoid", q_mode=("halfway", "bouzidi")[i % 2],
                            porosity=("hard", "soft")[i // 2 % 2]))
    return instances, spheres


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def _sphere_args(c):
    return dict(sharpness=c["alpha"], kind=c["mask"], q_mode=c["q_mode"], porosity=c["porosity"])


def prepare(case, seed):
    c = _full(case)
    kind, dt = c["kind"], _dtype(c)
    st = {"case": c}
    if kind in ("run", "grad"):
        st["f0"] = _initial(c, seed, dt, U if c["geometry"] == "sphere" else 0.3 * U)
        st["radius"] = _radius(c, seed)
        sim = Simulation(c["nx"], c["ny"], c["nz"], c["tau"], collision=c["collision"],
                         storage=c["storage"], use_smagorinsky=c["smag"],
                         periodic_yz=c["periodic"], guard=c["guard"], inlet_velocity=(U, 0.0, 0.0))
        if c["geometry"] == "channel":
            sim.set_mask(_walls(c))
            sim.set_inlet_profile(_profile(c, seed).to(dt))
        else:
            sim.set_sphere(st["radius"], **_sphere_args(c))
        if c["streaming"] == "aa":
            sim.set_streaming("aa")
        st["sim"] = sim
    elif kind == "simulate":
        solid, q = create_sphere(c["nx"], c["ny"], c["nz"], (0.0, 0.0, 0.0), _radius(c, seed))
        st["solid"], st["q"] = solid.to(torch.int32), q.to(dt).requires_grad_()
        st["f0"] = _initial(c, seed, dt, U).requires_grad_()
        st["g"] = _cotangent(c, seed, dt)
        st["params"] = LBMParams(tau=c["tau"], inlet_velocity=(U, 0.0, 0.0),
                                 collision_mode=int(c["collision"] == "mrt"),
                                 use_smagorinsky=int(c["smag"]), periodic_yz=c["periodic"])
    elif kind == "ops":
        g = _geometry(c, torch.tensor(_radius(c, seed), dtype=torch.float64, device="cuda"))
        st["area"] = g["area"]
        st["q"] = g["q"].to(dt).contiguous().requires_grad_()
        st["p"] = g["p"].to(dt).contiguous().requires_grad_()
        st["f0"] = _initial(c, seed, dt, U).requires_grad_()
        st["g"] = _cotangent(c, seed, dt)
    else:
        instances, st["spheres"] = _batch(c, seed)
        st["batch"] = Batch(instances)
    return st


def run(st):
    c = st["case"]
    if c["kind"] == "run":
        sim = st["sim"]
        sim.set_state(st["f0"])
        out = {}
        samples = sim.run(c["steps"], sample_every=c["sample"])
        if c["sample"]:
            # (Fx, Fy, Fz, Cd): FP64 sums over the run's populations, no more exact than these
            out["samples"] = samples.to(sim.dtype)
        out["f"] = sim.get_state()
        return out
    if c["kind"] == "grad":
        sim = st["sim"]
        sim.set_sphere(st["radius"], **_sphere_args(c))
        sim.set_state(st["f0"])
        got = sim.cd_and_grad(c["steps"], checkpoint_every=c["checkpoint"], dcd_dq=c["dense"],
                              dcd_df0=c["dense"])
        out = {"cd": got[0], "dcd_dr": got[1]}
        if c["dense"]:
            out.update(got[2])
        return out
    if c["kind"] == "simulate":
        f = simulate(LBMState(st["f0"], st["solid"], st["q"]), st["params"], c["steps"]).f
        gf, gq = torch.autograd.grad(f, (st["f0"], st["q"]), st["g"])
        return {"f": f.detach(), "g_f0": gf, "g_q": gq}
    if c["kind"] == "ops":
        f, q, p = st["f0"], st["q"], st["p"]
        post = soft_bounce_back(mrt(f, smagorinsky_tau(f, c["tau"], 0.1)), p)
        new = zou_he_outlet(zou_he_inlet(stream(post, q), (U, 0.0, 0.0)))
        cd = drag_coefficient(momentum_exchange(post, new, q), U, st["area"])
        gf, gq, gp = torch.autograd.grad((new, cd), (f, q, p), (st["g"], torch.ones_like(cd)))
        return {"f": new.detach(), "cd": cd.detach(), "g_f": gf, "g_q": gq, "g_p": gp}
    b = st["batch"]
    b.set_spheres(st["spheres"])
    b.set_equilibrium()
    h = b.optimize(1, c["steps"], lr=0.01, r_min=0.3, r_max=1.2,
                   checkpoint_every=c["checkpoint"])
    # histories of FP32 domains, to the precision of their arithmetic
    return {k: torch.from_numpy(v).float() for k, v in sorted(h.items())}


# ---------------------------------------------------------------------------
# the work
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the inputs read once and the outputs written once.  Operations: per cell and
    step 230 (BGK) or 320 (MRT) for the moments, the relaxation and the streaming, 70 for the
    eddy viscosity; a gradient's adjoint step, which needs the forward values again, twice that."""
    c = _full(case)
    cells = c["nx"] * c["ny"] * c["nz"]
    step = (320 if c["collision"] == "mrt" else 230) + (70 if c["smag"] else 0)
    size = 8 if c["storage"] == "fp64" else 4
    pop = 19 * size
    if c["kind"] == "batch":
        grids = [1.0, 27.0 / 64.0, 1.0 / 8.0]
        cells = int(cells * sum(grids[i % 3] for i in range(c["count"])))
        return {"bytes": cells * pop, "flops": 3 * step * cells * c["steps"]}
    if c["kind"] == "run":
        return {"bytes": 2 * cells * pop, "flops": step * cells * c["steps"]}
    if c["kind"] == "grad":
        return {"bytes": (3 if c["dense"] else 1) * cells * pop,
                "flops": 3 * step * cells * c["steps"]}
    if c["kind"] == "simulate":
        return {"bytes": cells * (6 * pop + 4), "flops": 3 * step * cells * c["steps"]}
    return {"bytes": cells * (6 * pop + 2 * size), "flops": 3 * step * cells}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _mrt_basis(device):
    """The moment matrix (rows k, columns i) of the d'Humieres basis."""
    rows = [[] for _ in range(19)]
    for x, y, z in zip(_EX, _EY, _EZ):
        s = x * x + y * y + z * z
        vals = [1, 19 * s - 30, (21 * s * s - 53 * s + 24) // 2, x, (5 * s - 9) * x, y,
                (5 * s - 9) * y, z, (5 * s - 9) * z, 3 * x * x - s,
                (3 * s - 5) * (3 * x * x - s), y * y - z * z, (3 * s - 5) * (y * y - z * z),
                x * y, y * z, x * z, (y * y - z * z) * x, (z * z - x * x) * y,
                (x * x - y * y) * z]
        for k in range(19):
            rows[k].append(float(vals[k]))
    return torch.tensor(rows, dtype=torch.float64, device=device)


def _collide(f, c):
    rho = f.sum(0)
    e = torch.tensor([_EX, _EY, _EZ], dtype=torch.float64, device=f.device)
    j = (e @ f.reshape(19, -1)).reshape((3,) + f.shape[1:])
    ux, uy, uz = j[0] / rho, j[1] / rho, j[2] / rho
    tau = c["tau"]
    feq = _equilibrium(rho, ux, uy, uz) if c["smag"] or c["collision"] == "bgk" else None
    if c["smag"]:
        pairs = torch.stack([e[a] * e[b] for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2),
                                                       (1, 2))])
        s = (pairs @ (f - feq).reshape(19, -1)).reshape((6,) + f.shape[1:])
        pi = torch.sqrt((s[:3] ** 2).sum(0) + 2.0 * (s[3:] ** 2).sum(0))
        tau = 0.5 * (tau + torch.sqrt(tau * tau + 18.0 * 0.01 * pi / (rho + 1e-10)))
    if c["collision"] == "bgk":
        return f - (f - feq) / tau
    m_all = _mrt_basis(f.device)
    m = (m_all @ f.reshape(19, -1)).reshape(f.shape)
    u2 = ux * ux + uy * uy + uz * uz
    pxx, pww = 3.0 * ux * ux - u2, uy * uy - uz * uz
    zero = torch.zeros_like(rho)
    meq = torch.stack([rho, rho * (-11.0 + 19.0 * u2), rho * (3.0 - 5.5 * u2), j[0], -2 / 3 * j[0],
                       j[1], -2 / 3 * j[1], j[2], -2 / 3 * j[2], rho * pxx, -0.5 * rho * pxx,
                       rho * pww, -0.5 * rho * pww, rho * ux * uy, rho * uy * uz, rho * ux * uz,
                       zero, zero, zero])
    omega = 1.0 / tau + zero
    rate = torch.stack([omega if k in (9, 11, 13, 14, 15) else zero + _RATE[k] for k in range(19)])
    d = rate * (m - meq)
    back = (m_all / (m_all * m_all).sum(1, keepdim=True)).t().contiguous()
    return f - (back @ d.reshape(19, -1)).reshape(f.shape)


def _edge(c, i, device):
    """Cells whose source x - e_i lies outside: they keep their own value."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    m = torch.zeros((nx, ny, nz), dtype=torch.bool, device=device)
    if _EX[i]:
        m[0 if _EX[i] > 0 else nx - 1] = True
    if not c["periodic"]:
        if _EY[i]:
            m[:, 0 if _EY[i] > 0 else ny - 1] = True
        if _EZ[i]:
            m[:, :, 0 if _EZ[i] > 0 else nz - 1] = True
    return m


def _stream(s, q, c):
    out = [s[0]]
    for i in range(1, 19):
        o, sh = _OPP[i], (_EX[i], _EY[i], _EZ[i])
        moved = torch.where(_edge(c, i, s.device), s[i], torch.roll(s[i], sh, (0, 1, 2)))
        a = 1.0 / (2.0 * q[o].clamp(0.5, 1.0))
        b = 2.0 * q[o].clamp(0.0, 0.5)
        ahead = torch.roll(s[o], tuple(-k for k in sh), (0, 1, 2))
        wall = torch.where(q[o] >= 0.5, a * s[o] + (1.0 - a) * s[i], b * s[o] + (1.0 - b) * ahead)
        out.append(torch.where(q[o] >= 0.0, wall, moved))
    return torch.stack(out)


def _inlet_outlet(f, face):
    ux, uy, uz = face
    a, b = f[:, 0], f[:, -1]
    side = (0, 3, 4, 5, 6, 15, 16, 17, 18)
    rho = (sum(a[i] for i in side) + 2.0 * sum(a[i] for i in (2, 8, 10, 12, 14))) / (1.0 - ux)
    new = {1: a[2] + rho * ux / 3.0, 7: a[10] + rho * (ux + uy) / 6.0,
           9: a[8] + rho * (ux - uy) / 6.0, 11: a[14] + rho * (ux + uz) / 6.0,
           13: a[12] + rho * (ux - uz) / 6.0}
    first = torch.stack([new.get(i, a[i]) for i in range(19)])
    v = -1.0 + sum(b[i] for i in side) + 2.0 * sum(b[i] for i in (1, 7, 9, 11, 13))
    new = {2: b[1] - v / 3.0, 10: b[7] - v / 6.0, 8: b[9] - v / 6.0, 14: b[11] - v / 6.0,
           12: b[13] - v / 6.0}
    last = torch.stack([new.get(i, b[i]) for i in range(19)])
    return torch.cat([first[:, None], f[:, 1:-1], last[:, None]], 1)


def _geometry(c, radius):
    """solid, q, porosity (or None), projected area of the case's body."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    dev = radius.device
    scale = (nx / 8.0, ny / 4.0, nz / 4.0)
    w = [((torch.arange(n, device=dev, dtype=torch.float64) + 0.5) / s - off).reshape(
        [-1 if k == j else 1 for k in range(3)]) for j, (n, s, off) in
        enumerate(zip((nx, ny, nz), scale, (4.0, 2.0, 2.0)))]
    d2 = w[0] ** 2 + w[1] ** 2 + w[2] ** 2
    p = torch.sigmoid(c["alpha"] * (radius - torch.sqrt(d2)))
    if c["geometry"] == "channel":
        solid = _walls(c).to(dev)
    else:
        solid = (d2 <= radius * radius) if c["mask"] == "dist" else (p > 0.5)
    body = torch.nn.functional.pad((solid > 0).double(), (1, 1, 1, 1, 1, 1)) > 0
    q = [torch.full((nx, ny, nz), -1.0, dtype=torch.float64, device=dev)]
    for i in range(1, 19):
        nb = body[1 + _EX[i]:1 + _EX[i] + nx, 1 + _EY[i]:1 + _EY[i] + ny,
                  1 + _EZ[i]:1 + _EZ[i] + nz]
        link = (solid == 0) & nb
        if c["geometry"] == "channel" or c["q_mode"] == "halfway":
            qv = torch.full_like(d2, 0.5)
        else:
            r = [e / s for e, s in zip((_EX[i], _EY[i], _EZ[i]), scale)]
            a = sum(v * v for v in r)
            b = 2.0 * sum(x * v for x, v in zip(w, r))
            disc = b * b - 4.0 * a * (d2 - radius * radius)
            t = (-b - torch.sqrt(disc.clamp_min(1e-10))) / (2.0 * a)
            ok = (disc >= 0.0) & (t > 0.0) & (t <= 1.0)
            qv = torch.where(ok, t, torch.full_like(t, 0.5)).clamp(0.01, 0.99)
        q.append(torch.where(link, qv, torch.full_like(qv, -1.0)))
    area = max(float((solid == 1).any(0).sum()), 1.0)
    return {"solid": solid, "q": torch.stack(q), "p": p, "area": area}


def _post(f, c, solid, p):
    s = _collide(f, c)
    t = s[list(_OPP)]
    if c["porosity"] == "soft":
        return (1.0 - p) * s + p * t
    return torch.where(solid >= 1, t, s)


def _force(s, f, q):
    total = torch.where(q >= 0.0, s + f[list(_OPP)], torch.zeros_like(s)).sum((1, 2, 3))
    e = torch.tensor([_EX, _EY, _EZ], dtype=torch.float64, device=s.device)
    return e @ total


def _drag(force, area):
    return force[0].abs() / (0.5 * U * U * area + 1e-10)


def exact(case, seed):
    c = _full(case)
    cells = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "batch" or c["kind"] == "grad" and cells * c["steps"] > 1.5e8:
        return None         # autograd through every step: more than some seconds
    c64 = {**c, "storage": "fp64"}
    f = _initial(c, seed, _dtype(c), U if c["geometry"] == "sphere" else 0.3 * U).double()
    radius = torch.tensor(_radius(c, seed), dtype=torch.float64, device="cuda", requires_grad=True)
    geo = _geometry(c64, radius)
    q, p, solid, area = geo["q"], geo["p"], geo["solid"], geo["area"]
    face = (U, 0.0, 0.0)
    if c["geometry"] == "channel":
        face = tuple(_profile(c, seed).to(_dtype(c)).double())

    def step(f, q, p):
        s = _post(f, c, solid, p)
        return s, _inlet_outlet(_stream(s, q, c), face)

    if c["kind"] == "run":
        rows = []
        with torch.no_grad():
            for k in range(1, c["steps"] + 1):
                s, f = step(f, q, p)
                if c["sample"] and k % c["sample"] == 0:
                    force = _force(s, f, q)
                    rows.append(torch.cat([force, _drag(force, area)[None]]))
        if not c["sample"]:
            return {"f": f}
        return {"samples": torch.stack(rows) if rows else torch.zeros(1, 4), "f": f}
    if c["kind"] == "ops":
        f, q, p = (t.detach().to(_dtype(c)).double().requires_grad_() for t in (f, q, p))
        s, new = step(f, q, p)
        cd = _drag(_force(s, new, q), area)
        gf, gq, gp = torch.autograd.grad((new, cd), (f, q, p),
                                         (_cotangent(c, seed, torch.float64),
                                          torch.ones_like(cd)))
        return {"f": new.detach(), "cd": cd.detach(), "g_f": gf, "g_q": gq, "g_p": gp}

    # gradients through the run: every state kept, one step's graph at a time
    states, last = [f], None
    with torch.no_grad():
        for _ in range(c["steps"]):
            last, f = step(f, q, p)
            states.append(f)
    gq, gp = torch.zeros_like(q), torch.zeros_like(p)
    qd, pd = q.detach().requires_grad_(), p.detach().requires_grad_()
    cd = None
    g = None if c["kind"] == "grad" else _cotangent(c, seed, torch.float64)
    for k in range(c["steps"] - 1, -1, -1):
        fk = states[k].detach().requires_grad_()
        s, new = step(fk, qd, pd)
        if g is None:
            out, seedg = _drag(_force(s, new, qd), area), None
            cd = out.detach()
        else:
            out, seedg = new, g
        got = torch.autograd.grad(out, (fk, qd, pd), seedg, allow_unused=True)
        g = got[0]
        gq += got[1] if got[1] is not None else 0.0
        gp += got[2] if got[2] is not None else 0.0
        states[k + 1] = None if k + 1 < c["steps"] else states[k + 1]
    if c["kind"] == "simulate":
        return {"f": states[-1], "g_f0": g, "g_q": gq}
    soft = c["porosity"] == "soft"
    (gr,) = torch.autograd.grad((q, p), radius, (gq, gp if soft else torch.zeros_like(gp)))
    out = {"cd": float(cd), "dcd_dr": float(gr)}
    if c["dense"]:
        out.update(dcd_dq=gq, dcd_df0=g)
    return out
