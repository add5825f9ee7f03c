"""A geometry whose buffers were too small runs again; one that never settles is an
error, not a handle without a geometry behind a success code."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SRC = r"""
#include <cstdio>
#include "sim_handle.cuh"
namespace lbm { int set_error(int status, const char*) { return status; } }
int main() {
  for (int need = 1; need < 8; ++need) {     // passes until nothing is left to do
    int n = 0;
    const int rc = settle_geometry([&](bool* more) -> int {
      *more = ++n < need;
      return LBM_OK;
    });
    const bool good = need <= 3 ? (rc == LBM_OK && n == need) : (rc == LBM_ERR_STATE && n == 3);
    if (!good) return printf("%d passes: %d after %d\n", need, rc, n), 1;
  }
  int n = 0;
  if (settle_geometry([&](bool*) -> int { ++n; return LBM_ERR_NOMEM; }) != LBM_ERR_NOMEM || n != 1)
    return printf("an error of a pass\n"), 1;
  printf("ok\n");
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs the CUDA compiler")
def test_passes_of_a_geometry(tmp_path):
    src, exe = tmp_path / "passes.cu", tmp_path / "passes"
    src.write_text(SRC)
    r = subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr",
                        "-I" + os.path.join(ROOT, "lbm_jax_autodiff_gb300", "csrc"),
                        "-I" + os.path.join(ROOT, "include"), "-gencode",
                        "arch=compute_103a,code=sm_103a", str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
