"""Chained launches (a step or an adjoint step starts while its predecessor still
writes): how their kernels load what the chain writes, and runs against the same
launches made one at a time."""

import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lbm_jax_autodiff_gb300", "csrc")
# the translation units and headers of the kernels that launch_chained starts
CHAINED = ("lbm_core.cuh", "vec2.cuh", "sim.cuh", "batch.cuh", "step.cu", "step_aa.cu",
           "adjoint.cuh", "adjoint_pair.cuh", "adjoint_batch.cu")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def _calls(code, name):
    for m in re.finditer(r"\b%s\(" % name, code):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(code[k], 0)
            k += 1
        yield code[m.end():k - 1]


@pytest.mark.parametrize("name", CHAINED)
def test_non_coherent_loads_read_geometry_only(name):
    code = _code(name)
    assert "global.nc" not in code
    for arg in _calls(code, "__ldg"):
        assert re.match(r"(a\.tag|a\.spec_pairs|A\.s\.spec_pairs|&r\.(w|nbw|gc)\[)", arg), arg


@pytest.mark.parametrize("name", CHAINED)
def test_global_loads_in_asm_are_ordered(name):
    code = _code(name)
    for m in re.finditer(r"asm\s*(volatile)?\s*\(", code):
        stmt = code[m.start():code.index(";", code.index('"', m.end()))]
        body = code[m.end():code.index(");", m.end())]
        if '"ld.global' in body:
            assert m.group(1) and '"memory"' in body, stmt


_SCRIPT = """
import hashlib, sys
import torch
import lbm_jax_autodiff_gb300 as L

def digest(*ts):
    h = hashlib.sha256()
    for t in ts:
        h.update(t.contiguous().view(torch.uint8).cpu().numpy().tobytes()
                 if torch.is_tensor(t) else repr(t).encode())
    return h.hexdigest()

# below and above one wave of blocks; even and odd nz
for grid in ((24, 13, 9), (64, 32, 32), (130, 66, 63), (160, 96, 96)):
    for storage in ("fp32", "fp64", "fp16", "bf16"):
        for streaming in ("ab", "aa"):
            if streaming == "aa" and storage in ("fp16", "bf16"):
                continue
            sim = L.Simulation(*grid, 0.55, collision="mrt", storage=storage,
                               use_smagorinsky=True)
            sim.set_sphere(0.7, kind="sigmoid", porosity="soft", sharpness=10.0)
            sim.set_streaming(streaming)
            f0 = sim.equilibrium_state().cuda()
            gen = torch.Generator(device="cuda").manual_seed(3)
            f0 = (f0 * (1.0 + 0.01 * torch.randn(f0.shape, generator=gen, device="cuda",
                                                 dtype=f0.dtype))).contiguous()
            sim.set_state(f0)
            s = sim.run(60, sample_every=25)
            print(grid, storage, streaming, digest(sim.get_state(), s))
            if streaming == "ab":
                sim.set_state(f0)
                cd, dr, ex = sim.cd_and_grad(24, checkpoint_every=10, dcd_dq=True, dcd_df0=True)
                print(grid, storage, "grad", digest(cd, dr, ex["dcd_dq"], ex["dcd_df0"]))
            sim.close()
"""


@pytest.mark.gpu
def test_chained_equals_one_at_a_time(cuda):
    # CUDA_LAUNCH_BLOCKING: every launch is waited for before the next is made
    out = []
    for blocking in ("0", "1"):
        env = dict(os.environ, CUDA_LAUNCH_BLOCKING=blocking)
        r = subprocess.run([sys.executable, "-c", _SCRIPT], cwd=ROOT, env=env, text=True,
                           capture_output=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        out.append(r.stdout.splitlines())
    assert len(out[0]) == 40
    assert out[0] == out[1]
