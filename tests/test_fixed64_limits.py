"""The fixed-point FP64 collision and its transpose (csrc/fixed64.cuh) at the limits
of the cells that they take, where an intermediate that did not fit would wrap:
densities at 1/2 and 2, momenta at 1/4 in every combination of signs, populations at
their bounds with either sign.  Against extended precision on the host, with the
device's wrapping integers; and the device's square root and reciprocal."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
CSRC = os.path.join(ROOT, "lbm_jax_autodiff_gb300", "csrc")

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
namespace lbm {
inline long double lbm_rcp(long double x) { return 1.0L / x; }
inline long double lbm_sqrt(long double x) { return sqrtl(x); }
}
#include "fixed64.cuh"
using namespace lbm;

std::mt19937_64 g(1);
std::uniform_real_distribution<double> U(-1, 1);
double sign() { return (g() & 1) ? 1.0 : -1.0; }

// A cell at the limits: populations at their bounds or anywhere in them; kinds 1 to 3
// are moved onto a density and momentum at the edge of what is accepted.
void cell(int kind, double f[Q]) {
  const double w[3] = {1. / 3, 1. / 18, 1. / 36};
  for (int i = 0; i < Q; ++i) {
    const double top = i == 0 ? 0.5 : 0.25;
    f[i] = kind == 0 ? sign() * top * (1 - 1e-9 * fabs(U(g)))
           : kind == 3 ? 0.7 * sign() * top : 0.6 * top * U(g);
  }
  if (kind == 0) return;
  double rho = 0, j[3] = {0, 0, 0};
  for (int i = 0; i < Q; ++i) {
    rho += f[i];
    j[0] += ex(i) * f[i];
    j[1] += ey(i) * f[i];
    j[2] += ez(i) * f[i];
  }
  const double edge = (g() & 1) ? 1e-12 : 1e-3 * fabs(U(g));
  const double r = (g() & 1) ? 0.5 + edge : 2.0 - edge;
  double jt[3];
  for (int a = 0; a < 3; ++a) jt[a] = kind == 2 && (g() & 1) ? 0.2 * U(g) : sign() * (0.25 - edge);
  for (int i = 0; i < Q; ++i) {
    const double wi = w[i == 0 ? 0 : (i < 7 ? 1 : 2)];
    f[i] += wi * ((r - rho) + 3 * (ex(i) * (jt[0] - j[0]) + ey(i) * (jt[1] - j[1]) +
                                   ez(i) * (jt[2] - j[2])));
  }
}

int main() {
  const double w[3] = {1. / 3, 1. / 18, 1. / 36};
  const double r[Q] = {0.0, 1.19, 1.4, 0.0, 1.2, 0.0, 1.2, 0.0, 1.2, 0.0,
                       1.4, 0.0,  1.4, 0.0, 0.0, 0.0, 1.98, 1.98, 1.98};
  // a wrapped integer is off by 2^-7 and more; roundings are some dozens of units of
  // 2^-58 (forward) and of 2^-57 of the cell's largest cotangent (transposed)
  const double bar = 300 * ldexp(1.0, -58), bar_t = 300 * ldexp(1.0, -57);
  for (int exact = 0; exact < 2; ++exact) {
    Consts<double> K;
    Consts<long double> KL;
    for (int i = 0; i < Q; ++i) {
      const double wi = w[i == 0 ? 0 : (i < 7 ? 1 : 2)];
      K.w[i] = exact ? wi : double(float(wi));
      K.rate[i] = exact ? r[i] : double(float(r[i]));
      KL.w[i] = K.w[i];
      KL.rate[i] = K.rate[i];
    }
    for (int kind = 0; kind < 4; ++kind)
      for (double tau : {0.5000001, 0.503, 0.8, 40.0})
        for (double c18 : {0.0, 0.18, 0.72}) {
          const FixConsts C = make_fix_consts(K, tau, c18);
          const bool smag = c18 > 0;
          int n = 0, nt = 0, ne = 0;
          for (int t = 0; t < 400000 && n < 1500; ++t) {
            double f[Q], mu[Q], of[Q];
            long double fl[Q], o[Q], ml[Q];
            cell(kind, f);
            FixCell c;
            if (!fixed_load(f, c)) continue;
            ++n;
            for (int i = 0; i < Q; ++i) fl[i] = f[i];
            for (int mrt = 0; mrt < 2; ++mrt) {
              auto sink = [&](int i, fix v) { of[i] = mrt ? from_fix<61>(v) : from_fix<59>(v); };
              if (mrt) fixed_collide<true>(c, smag, C, sink);
              else fixed_collide<false>(c, smag, C, sink);
              collide_cell<long double>(fl, (long double)tau, mrt, smag, (long double)c18, KL, o);
              for (int i = 0; i < Q; ++i)
                if (!(fabs(double(of[i] - o[i])) <= bar))
                  return printf("forward: mrt %d tau %g c %g kind %d f[%d] %g for %g\n", mrt, tau,
                                c18, kind, i, of[i], double(o[i])), 1;
            }
            // cotangents: one size and random sign, all equal, aligned with one moment
            for (int m = 0; m < 3; ++m) {
              const int row = 1 + int(g() % 18);
              const double size = ldexp(1 - 1e-9 * fabs(U(g)), int(g() % 40) - 20);
              for (int i = 0; i < Q; ++i)
                mu[i] = size * (m == 0 ? sign() : m == 1 ? 1.0 : mrow(row, i) < 0 ? -1.0 : 1.0);
              fix F[Q];
              int sh;
              if (!fixed_load_T(mu, F, sh)) return printf("cotangents refused\n"), 1;
              for (int mrt = smag; mrt < 2; ++mrt) {
                FixEddyT ed;
                if (smag) {
                  ++nt;
                  if (!fixed_eddy_T(c, C, sh, F, ed)) continue;
                  ++ne;
                  fixed_collide_T<true, true>(c, C, sh, F, of, &ed);
                } else if (mrt) {
                  fixed_collide_T<true>(c, C, sh, F, of);
                } else {
                  fixed_collide_T<false>(c, C, sh, F, of);
                }
                for (int i = 0; i < Q; ++i) ml[i] = mu[i];
                CellScalars<long double> cl;
                cell_scalars<long double>(fl, cl);
                collide_vjp_s<long double>(cl, fl, ml, (long double)tau, mrt, smag,
                                           (long double)c18, KL, nullptr);
                for (int i = 0; i < Q; ++i)
                  if (!(fabs(double(of[i] - ml[i])) <= bar_t * size))
                    return printf("transposed: mrt %d tau %g c %g kind %d m %d g[%d] %g for %g (%g)\n",
                                  mrt, tau, c18, kind, m, i, of[i], double(ml[i]), size), 1;
              }
            }
          }
          if (n < 500 || (smag && ne * 2 < nt))
            return printf("tau %g c %g kind %d: %d cells, %d of %d eddy\n", tau, c18, kind, n, ne,
                          nt), 1;
        }
  }
  printf("ok\n");
  return 0;
}
"""

SRC_ROOTS = r"""
#include <cstdio>
#include "fixed64.cuh"
using namespace lbm;
// worst error of newton_sqrt and newton_rcp in ulp of the result
__global__ void k_roots(double lo, double hi, int n, double* worst) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  unsigned long long h = (t + 1) * 0x9e3779b97f4a7c15ull;
  h ^= h >> 29;
  h *= 0xbf58476d1ce4e5b9ull;
  h ^= h >> 32;
  const double u = double(h >> 11) * 1.1102230246251565e-16;      // 2^-53
  const double x = lo * exp(log(hi / lo) * u);
  const double s = sqrt(x), r = 1.0 / x;
  const double es = fabs(newton_sqrt(x) - s) / (nextafter(s, 1e300) - s);
  const double er = fabs(newton_rcp(x) - r) / (nextafter(r, 1e300) - r);
  if (es > 1.0 || er > 1.0 || es != es || er != er) {
    worst[0] = x;
    worst[1] = es;
    worst[2] = er;
  }
}
int main() {
  double *d, h[3] = {0, 0, 0};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return printf("no memory\n"), 1;
  cudaMemcpy(d, h, sizeof(h), cudaMemcpyHostToDevice);
  const int n = 1 << 20;
  // squared stresses, tau^2 + 18 Cs^2 |stress| / rho, and relaxation times
  const double range[4][2] = {{1e-32, 1e-20}, {1e-20, 64.0}, {0.2, 8.0}, {8.0, 1e13}};
  for (auto& q : range) k_roots<<<n / 256, 256>>>(q[0], q[1], n, d);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return printf("copy\n"), 1;
  if (h[0] != 0) return printf("x %.17g: sqrt %g ulp, reciprocal %g ulp\n", h[0], h[1], h[2]), 1;
  printf("ok\n");
  return 0;
}
"""


def _run(tmp_path, text, *flags):
    src, exe = tmp_path / "fixed.cu", tmp_path / "fixed"
    src.write_text(text)
    r = subprocess.run([NVCC, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-I" + CSRC,
                        "-Xcompiler", "-ffp-contract=off", *flags, "-gencode",
                        "arch=compute_103a,code=sm_103a", str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs the CUDA compiler")
def test_cells_at_the_limits(tmp_path):
    _run(tmp_path, SRC, "-Xcompiler", "-fwrapv")


@pytest.mark.gpu
def test_roots_on_the_device(cuda, tmp_path):
    # a seed of 22 bits, two steps, one rounding of the last: within an ulp
    _run(tmp_path, SRC_ROOTS)
