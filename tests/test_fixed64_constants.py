"""Which constants the fixed-point FP64 collision (csrc/fixed64.cuh) takes: one that
is not finite, or beyond the range of its roots' FP32 seeds, runs the FP64 form."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SRC = r"""
#include <cstdio>
#include "fixed64.cuh"
using namespace lbm;
int main() {
  Consts<double> K;
  for (int i = 0; i < Q; ++i) {
    K.w[i] = i == 0 ? 1.0 / 3 : (i < 7 ? 1.0 / 18 : 1.0 / 36);
    K.rate[i] = 1.2;
  }
  for (double tau : {0.5000001, 0.55, 1.0, 40.0, 1e6})
    for (double c : {0.0, 0.18, 18.0, 1e3})
      if (!make_fix_consts(K, tau, c).ok) return printf("refused %g %g\n", tau, c), 1;
  for (double c : {(double)NAN, (double)INFINITY, -0.18, 1e30})
    if (make_fix_consts(K, 0.55, c).ok) return printf("taken: constant %g\n", c), 1;
  for (double tau : {(double)NAN, (double)INFINITY, 0.5, 0.1, -1.0, 1e20})
    if (make_fix_consts(K, tau, 0.18).ok) return printf("taken: tau %g\n", tau), 1;
  printf("ok\n");
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs the CUDA compiler")
def test_constants_of_the_fixed_point_form(tmp_path):
    src, exe = tmp_path / "consts.cu", tmp_path / "consts"
    src.write_text(SRC)
    r = subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr",
                        "-I" + os.path.join(ROOT, "lbm_jax_autodiff_gb300", "csrc"), "-gencode",
                        "arch=compute_103a,code=sm_103a", str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("collision", ["bgk", "mrt"])
def test_a_nan_constant_gives_nan(cuda, collision):
    import lbm_jax_autodiff_gb300 as L
    sim = L.Simulation(8, 6, 6, 0.6, collision=collision, storage="fp64", use_smagorinsky=True,
                       smagorinsky_cs=float("nan"))
    sim.set_sphere(0.6)
    f = sim.equilibrium_state().cuda() * 1.0
    f[1] *= 1.01
    sim.set_state(f)
    sim.run(2)
    assert sim.get_state().isnan().any()
    # unused, it changes nothing
    out = []
    for cs in (float("nan"), 0.1):
        sim = L.Simulation(8, 6, 6, 0.6, collision=collision, storage="fp64", smagorinsky_cs=cs)
        sim.set_sphere(0.6)
        sim.set_state(f)
        sim.run(2)
        out.append(sim.get_state())
    assert out[0].isfinite().all() and bool((out[0] == out[1]).all())
