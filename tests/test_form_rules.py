"""The size rules of the kernels' forms: counted in the device's SMs, and each line
where the measured times put it."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

# us a step of a run and its adjoint, one / two blocks per SM, on 152 SMs
# (soft, eddy, mrt): {blocks: (one, two)}
TIMES = {
    (0, 0, 1): {256: (44.8, 50.2), 500: (55.9, 58.4), 666: (66.6, 70.1), 864: (82.8, 84.5),
                1099: (99.9, 96.9), 1372: (119.8, 109.4), 2048: (162.8, 141.7)},
    (0, 0, 0): {256: (45.9, 51.8), 500: (59.8, 62.2), 666: (69.2, 72.9), 864: (87.8, 90.7),
                1099: (105.6, 102.8), 1372: (126.5, 116.9), 2048: (171.5, 149.7)},
    (0, 1, 1): {256: (62.5, 74.5), 500: (84.9, 97.1), 666: (97.1, 113.3), 864: (119.0, 128.8),
                1099: (141.1, 146.8), 1372: (167.5, 165.0), 2048: (226.4, 208.6)},
    (1, 0, 1): {256: (55.7, 61.6), 500: (86.5, 77.7), 666: (106.8, 94.6), 864: (136.2, 114.3),
                1099: (167.0, 136.4), 1372: (202.4, 163.3), 2048: (285.4, 222.4)},
    (1, 0, 0): {256: (58.8, 62.9), 500: (91.4, 81.7), 666: (112.8, 99.6), 864: (143.8, 121.1),
                1099: (175.9, 145.0), 1372: (212.8, 173.2), 2048: (299.0, 235.2)},
    (1, 1, 1): {256: (78.8, 87.0), 500: (120.9, 115.0), 666: (148.1, 141.6), 864: (183.0, 166.4),
                1099: (226.1, 199.0), 1372: (273.0, 239.4), 2048: (383.7, 328.6)},
    (0, 1, 0): {256: (89.8, 114.8), 500: (125.7, 149.5), 666: (142.5, 171.5), 864: (166.3, 187.1),
                1099: (190.2, 212.5), 1372: (218.7, 238.5), 2048: (295.5, 303.6)},
    (1, 1, 0): {256: (107.9, 137.9), 500: (155.7, 174.6), 666: (186.9, 202.4), 864: (227.8, 228.1),
                1099: (275.3, 263.4), 1372: (331.4, 303.8), 2048: (464.1, 411.8)},
}

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "sim.cuh"
int main(int, char** v) {
  for (long long n; scanf("%lld", &n) == 1;) {
    int sms, soft, eddy, mrt;
    if (scanf("%d %d %d %d", &sms, &soft, &eddy, &mrt) != 4) return 1;
    printf("%d %d\n", int(lbm::one_block_per_sm(int(n), sms, soft, eddy, mrt)),
           int(lbm::roomy_cells(n, sms)));
  }
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs the CUDA compiler")
def test_lines_lie_where_they_were_measured(tmp_path):
    src, exe = tmp_path / "rules.cu", tmp_path / "rules"
    src.write_text(SRC)
    r = subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr",
                        "-I" + os.path.join(ROOT, "lbm_jax_autodiff_gb300", "csrc"), "-gencode",
                        "arch=compute_103a,code=sm_103a", str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    ask = [(nb, 152, *form) for form, t in TIMES.items() for nb in t]
    # half of the SMs: the lines move with them
    ask += [(nb // 2, 76, *form) for nb, _, *form in ask]
    cells = [(n, s, 0, 0, 1) for s in (76, 152) for n in (1024 * s, 1024 * s + 1)]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60,
                       input="\n".join(" ".join(map(str, a)) for a in ask + cells))
    assert r.returncode == 0
    got = [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    for (nb, sms, *form), (one, _) in zip(ask, got):
        t = TIMES[tuple(form)]
        times = t[nb if sms == 152 else min(t, key=lambda b: abs(b - 2 * nb))]
        assert times[0 if one else 1] <= 1.02 * min(times), (nb, sms, form, one)
    assert [roomy for _, roomy in got[len(ask):]] == [1, 0, 1, 0]
