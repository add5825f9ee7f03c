"""The fixed-point FP64 collision and its transpose (csrc/fixed64.cuh) on the
host: conversions, the range tests, and its error against extended precision beside that of the
FP64 form that it stands in for, over relaxation times, speeds and departures
from equilibrium.  Compiled with the CUDA compiler, run on the CPU."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

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

#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); exit(1); } } while (0)

int main() {
  std::mt19937_64 g(1);
  std::normal_distribution<double> N(0, 1);
  std::uniform_real_distribution<double> U(-1, 1);
  // conversions: exact from 2^-6 up, within 2^-58 below; back to the nearest double
  CHECK(from_fix(0) == 0.0 && from_fix(to_fix(0.0)) == 0.0 && to_fix(-0.0) == 0);
  for (int k = 0; k < 400000; ++k) {
    const double v = U(g) * ldexp(1.0, -(k % 40));
    const double r = from_fix(to_fix(v));
    CHECK(fabs(r - v) <= ldexp(1.0, -58));
    if (fabs(v) >= 1.0 / 64) CHECK(r == v);
    const fix x = fix(g()) >> (2 + k % 60);
    CHECK(from_fix(x) == double((long double)x * ldexpl(1.0L, -58)));
    CHECK(from_fix<61>(x) == double((long double)x * ldexpl(1.0L, -61)));
  }
  // cells out of the range are refused
  FixCell c;
  double f[Q];
  const double bad[] = {0.25, -0.25, 1.0, 1e300, INFINITY, -INFINITY, NAN};
  for (double b : bad)
    for (int i = 1; i < Q; ++i) {
      for (int j = 0; j < Q; ++j) f[j] = j == 0 ? 1.0 / 3 : (j < 7 ? 1.0 / 18 : 1.0 / 36);
      CHECK(fixed_load(f, c));
      f[i] = b;
      CHECK(!fixed_load(f, c));
    }
  for (double s : {0.0, 0.49, 2.1, -1.0, 1e-300}) {
    for (int j = 0; j < Q; ++j) f[j] = s * (j == 0 ? 1.0 / 3 : (j < 7 ? 1.0 / 18 : 1.0 / 36));
    CHECK(!fixed_load(f, c));
  }
  // error of every population over the range, all corners of it included
  const double w[3] = {1. / 3, 1. / 18, 1. / 36};
  const double r[Q] = {0.0, 1.19, 1.4, 0.0, 1.2, 0.0, 1.2, 0.0, 1.2, 0.0,
                       1.4, 0.0,  1.4, 0.0, 0.0, 0.0, 1.98, 1.98, 1.98};
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
    for (int mrt = 0; mrt < 2; ++mrt)
      for (int smag = 0; smag < 2; ++smag)
        for (double tau : {0.5000001, 0.503, 0.548, 0.8, 2.0, 40.0})
          for (double speed : {0.0, 0.1, 0.2})
            for (double dens : {0.0, 0.05, 0.28})
              for (double amp : {0.0, 1e-6, 1e-2, 0.6}) {
                const FixConsts C = make_fix_consts(K, tau, 18 * 0.01);
                CHECK(C.ok);
                double e64 = 0, efx = 0, top = 0;
                int n = 0;
                for (int t = 0; t < 200; ++t) {
                  double feq[Q], od[Q], of[Q];
                  long double fl[Q], o[Q];
                  equilibrium<double>(1 + dens * U(g), speed * U(g), speed * U(g), speed * U(g), K.w,
                                      feq);
                  for (int i = 0; i < Q; ++i) fl[i] = f[i] = feq[i] + amp * K.w[i] * N(g);
                  if (!fixed_load(f, c)) continue;
                  auto sink = [&](int i, fix v) { of[i] = mrt ? from_fix<61>(v) : from_fix<59>(v); };
                  if (mrt) fixed_collide<true>(c, smag, C, sink);
                  else fixed_collide<false>(c, smag, C, sink);
                  collide_cell<long double>(fl, (long double)tau, mrt, smag,
                                            (long double)C.c18cs2, KL, o);
                  collide_cell<double>(f, tau, mrt, smag, C.c18cs2, K, od);
                  for (int i = 0; i < Q; ++i) {
                    const double a = double(od[i] - o[i]), b = double(of[i] - o[i]);
                    e64 += a * a;
                    efx += b * b;
                    top = fmax(top, fabs(b));
                    ++n;
                  }
                }
                if (n < 100) continue;
                // rounding of the result itself (rms 5e-18 over these populations) counts
                // in both; at rest with no noise the FP64 form may happen to be exact
                if (!(efx <= e64 * 1.1 || sqrt(efx / n) < 8e-18) || top > 2e-16) {
                  printf("exact %d mrt %d smag %d tau %g u %g rho %g amp %g: %g %g top %g\n", exact,
                         mrt, smag, tau, speed, dens, amp, sqrt(e64 / n), sqrt(efx / n), top);
                  return 1;
                }
              }
  }
  printf("ok\n");
  return 0;
}
"""


SRC_T = SRC[:SRC.index("int main()")] + r"""
int main() {
  std::mt19937_64 g(1);
  std::normal_distribution<double> N(0, 1);
  std::uniform_real_distribution<double> U(-1, 1);
  fix F[Q];
  int sh;
  double mu[Q];
  // extreme, non-finite and all-zero cotangents are refused, mixed ones are not
  const double bad[] = {INFINITY, -INFINITY, NAN, 1e300, 1e-300};
  for (double b : bad) {
    for (int i = 0; i < Q; ++i) mu[i] = 0.0;
    CHECK(all_zero(mu) && !fixed_load_T(mu, F, sh));
    mu[7] = 1e-30;
    CHECK(!all_zero(mu) && fixed_load_T(mu, F, sh));
    mu[7] = b;
    CHECK(!fixed_load_T(mu, F, sh));
  }
  const double w[3] = {1. / 3, 1. / 18, 1. / 36};
  const double r[Q] = {0.0, 1.19, 1.4, 0.0, 1.2, 0.0, 1.2, 0.0, 1.2, 0.0,
                       1.4, 0.0,  1.4, 0.0, 0.0, 0.0, 1.98, 1.98, 1.98};
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
    for (int form = 0; form < 3; ++form)      // BGK, MRT, MRT with the eddy viscosity
      for (double tau : {0.5000001, 0.503, 0.548, 0.8, 2.0, 40.0})
        for (double speed : {0.0, 0.1, 0.24})
          for (double dens : {0.0, 0.4})
            // cotangents: random, nearly equal, of mixed size, of one size and random sign
            // (the largest sums), 400 decades between the cells
            for (int kind = 0; kind < 5; ++kind) {
              const bool mrt = form > 0, smag = form == 2;
              const FixConsts C = make_fix_consts(K, tau, smag ? 0.18 : 0.0);
              double e64 = 0, efx = 0, top = 0;
              int n = 0;
              for (int t = 0; t < 300; ++t) {
                double f[Q], of[Q], od[Q];
                long double fl[Q], ml[Q];
                equilibrium<double>(1 + dens * U(g), speed * U(g), speed * U(g), speed * U(g), K.w, f);
                const double sc = pow(10.0, kind == 4 ? 200 * U(g) : 6 * U(g));
                double big = 0;
                for (int i = 0; i < Q; ++i) {
                  f[i] += 1e-4 * K.w[i] * N(g);
                  mu[i] = sc * (kind == 1 ? 1 + 0.01 * N(g)
                                : kind == 2 ? N(g) * pow(10.0, -2 * fabs(N(g)))
                                : kind == 3 ? ((g() & 1) ? 1.0 : -1.0) : N(g));
                  big = fmax(big, fabs(mu[i]));
                  ml[i] = od[i] = mu[i];
                  fl[i] = f[i];
                }
                FixCell c;
                if (!fixed_load(f, c)) continue;
                CHECK(fixed_load_T(mu, F, sh));
                FixEddyT ed;
                if (smag) {
                  CHECK(fixed_eddy_T(c, C, sh, F, ed));
                  fixed_collide_T<true, true>(c, C, sh, F, of, &ed);
                } else if (mrt) fixed_collide_T<true>(c, C, sh, F, of);
                else fixed_collide_T<false>(c, C, sh, F, of);
                CellScalars<long double> cl;
                cell_scalars<long double>(fl, cl);
                collide_vjp_s<long double>(cl, fl, ml, (long double)tau, mrt, smag,
                                           (long double)C.c18cs2, KL, nullptr);
                CellScalars<double> cd;
                cell_scalars<double>(f, cd);
                collide_vjp_s<double>(cd, f, od, tau, mrt, smag, C.c18cs2, K, nullptr);
                for (int i = 0; i < Q; ++i) {
                  const double a = double(od[i] - ml[i]) / big, b = double(of[i] - ml[i]) / big;
                  e64 += a * a;
                  efx += b * b;
                  top = fmax(top, fabs(b));
                  ++n;
                }
              }
              if (n < 100) continue;
              // (at rest the FP64 form skips its velocity terms' roundings)
              if (!(efx <= e64 * 1.1 || (speed == 0.0 && sqrt(efx / n) < 8e-17)) || top > 1.5e-15) {
                printf("exact %d form %d tau %g u %g rho %g kind %d: %g %g top %g\n", exact, form, tau,
                       speed, dens, kind, sqrt(e64 / n), sqrt(efx / n), top);
                return 1;
              }
            }
  }
  printf("ok\n");
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs the CUDA compiler")
@pytest.mark.parametrize("which", ["forward", "transposed"])
def test_fixed_point_collision_on_the_host(tmp_path, which):
    src, exe = tmp_path / "fixed.cu", tmp_path / "fixed"
    src.write_text(SRC if which == "forward" else SRC_T)
    inc = os.path.join(ROOT, "lbm_jax_autodiff_gb300", "csrc")
    r = subprocess.run([NVCC, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-I" + inc,
                        "-Xcompiler", "-ffp-contract=off", "-gencode",
                        "arch=compute_103a,code=sm_103a", str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
