// FP64-storage collision on 64-bit integers.
//
// sm_103a executes about two FP64 operations per clock and SM, a 64th of its
// FP32 rate, and the ~350 of a collision made the FP64 step 15 times longer
// than its bytes (2.2 to 2.7 ms against 0.19 ms at 256x128x128).  Its integer
// units are full rate.  So a cell's collision runs in fixed point, 58 bits
// after the point: populations f < 1/2 are multiples of 2^-58 or of a coarser
// unit as soon as they are above 2^-6 (a double holds 53 bits), so the
// conversion is exact for those and off by less than 2^-58 = 3.5e-18 below,
// sums are exact, and a product is off by one unit; an FP64 sum around a
// density of 1 rounds by 1.1e-16 a term.  Populations are held as deviations
// from a rest state whose moments are exact integers, which keeps every
// intermediate small; mass and momentum are then conserved exactly by the MRT
// form (the relaxed moments' terms cancel in integers).  Against extended
// precision the populations' rms error is 4.3e-18 to 5.2e-18, 0.17 to 0.55 of
// the FP64 form's over relaxation times 0.503 to 2, with and without the eddy
// viscosity (tests/test_fixed64_cpu.py).  Measured: 60 steps of a 96x48x48
// sphere 7.87 -> 1.70 ms, chained 1.61 (131 -> 27 us a step, its bytes take 10).
//
// The range this holds for (fixed_load): f_0 < 1/2, the other |f_i| < 1/4,
// 1/2 <= rho < 2, |j_a| < 1/4: the densities and speeds at which the lattice
// model holds, with a margin.  Any other
// cell (also infinite, NaN) takes the FP64 form of lbm_core.cuh.
#pragma once

#include "lbm_core.cuh"

namespace lbm {

typedef long long fix;             // value * 2^58
constexpr int kFix = 58;
// rest state: edge weight kRestE, face weight 2 kRestE, rest weight 12 kRestE,
// so that its density is exactly 36 kRestE and its 2nd moments 12 kRestE
constexpr fix kRestE = 8006399486320277LL;   // round(2^58 / 36)
constexpr fix kRest = 36 * kRestE;
__host__ __device__ constexpr fix rest_of(int i) {
  return i == 0 ? 12 * kRestE : (i < 7 ? 2 * kRestE : kRestE);
}

// high 64 bits of the signed 128-bit product
__host__ __device__ __forceinline__ fix mulhi(fix a, fix b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return fix((__int128(a) * b) >> 64);
#endif
}
// a b for |a| < 1/2
__host__ __device__ __forceinline__ fix mulf(fix a, fix b) { return mulhi(a << 6, b); }
// double -> fix for |v| < 2, truncated towards zero (exact for |v| >= 2^-6).
__host__ __device__ __forceinline__ fix to_fix(double v) {
#ifdef __CUDA_ARCH__
  const unsigned hi = __double2hiint(v), lo = __double2loint(v);
#else
  unsigned long long b;
  memcpy(&b, &v, 8);
  const unsigned hi = unsigned(b >> 32), lo = unsigned(b);
#endif
  // mantissa with its leading bit at bit 63, then down by 1028 - exponent
  const unsigned mh = ((hi << 11) | (lo >> 21)) | 0x80000000u, ml = lo << 11;
  const unsigned s = 1028u - ((hi >> 20) & 0x7ffu);
  unsigned long long m = (unsigned long long)mh << 32 | ml;
#ifdef __CUDA_ARCH__
  asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(s));   // amounts above 63 give 0
#else
  m = s > 63 ? 0 : m >> s;
#endif
  const fix g = fix(int(hi) >> 31);
  return (fix(m) ^ g) - g;
}

// x 2^-BITS as a double, rounded to nearest even
template <int BITS = kFix>
__host__ __device__ __forceinline__ double from_fix(fix x) {
  const fix g = x >> 63;
  const unsigned long long a = (unsigned long long)((x ^ g) - g);
#ifdef __CUDA_ARCH__
  const int z = __clzll((long long)a);
#else
  const int z = a ? __builtin_clzll(a) : 64;
#endif
  // leading bit to bit 62; adding the mantissa with its leading bit onto the
  // exponent field below carries a round-up to the next power of two by itself
  unsigned long long m = a << ((z - 1) & 63);
  m = (m + 0x1ffull + ((m >> 10) & 1ull)) >> 10;
  const unsigned e = (unsigned(1022 + 63 - BITS - z) << 20) | (unsigned(int(g)) & 0x80000000u);
  unsigned hi = unsigned(m >> 32) + e, lo = unsigned(m);
  if (z == 64) hi = 0;
#ifdef __CUDA_ARCH__
  return __hiloint2double(int(hi), int(lo));
#else
  const unsigned long long r = (unsigned long long)hi << 32 | lo;
  double d;
  memcpy(&d, &r, 8);
  return d;
#endif
}

// Constants of a launch (host), times the power of two in the brackets: with
// the shifts of fixed_collide every relaxed moment comes out in units of 2^-61
// (the back transform multiplies some by up to 30).
struct FixConsts {
  fix m1, m2, m4, m10, m12, m16;       // fixed MRT rates over norms [67, m16: 65]
  fix s9, s11, s13;                    // omega / 36 [67], omega / 12 [65], omega / 4 [64]
  // transposed collision [65; t1a, t1b, t2a: 69; t2b: 68; t13, t16: 64]
  fix t1a, t1b, t2a, t2b, t4, t10, t12, t16, t9, t11, t13;
  fix tw[3];                           // w_0 [64], w_face [67], w_edge [68]
  fix om;                              // omega [62]
  fix b1, bw[3];                       // BGK: 1 - omega, omega w_0, w_face, w_edge [63]
  fix w[3];                            // w_0, w_face, w_edge [63]
  fix qa, qb, qc;                      // second moments of the weights less their exact values:
                                       // W2 - 1/3, 9 W22 - 1, 4.5 W22 - 1.5 W2 [64]
  double w2, w22;                      // second moments of the weights: sum w e_x^2, sum w e_x^2 e_y^2
  double tau, c18cs2;
  int ok;                              // omega, the rates and the eddy viscosity's constant in range
};
inline fix fix_scale(long double v, int bits) { return fix(llrintl(ldexpl(v, bits))); }
inline FixConsts make_fix_consts(const Consts<double>& K, double tau, double c18cs2) {
  FixConsts c;
  const double om0 = 1.0 / tau;
  c.ok = om0 > 0.0 && om0 < 2.0;
  // the roots of the eddy viscosity start from an FP32 seed; beyond these (a NaN
  // constant too) the FP64 form runs, whose result says so
  if (!(tau <= 1e6 && c18cs2 >= 0.0 && c18cs2 <= 1e3)) c.ok = 0;
  const long double om = c.ok ? om0 : 1.0;
  for (int k = 0; k < Q; ++k)
    if (!(K.rate[k] >= 0.0 && K.rate[k] <= (k < 3 ? 1.5 : 2.0))) c.ok = 0;
  auto rate = [&](int k) -> long double { return c.ok ? K.rate[k] : 0.0; };
  c.m1 = fix_scale(rate(1) / 126.0L, 67);
  c.m2 = fix_scale(rate(2) / 252.0L, 67);
  c.m4 = fix_scale(rate(4) / 24.0L, 66);
  c.m10 = fix_scale(rate(10) / 72.0L, 67);
  c.m12 = fix_scale(rate(12) / 24.0L, 66);
  c.m16 = fix_scale(rate(16) / 8.0L, 64);
  c.s9 = fix_scale(om / 36.0L, 67);
  c.s11 = fix_scale(om / 12.0L, 65);
  c.s13 = fix_scale(om / 4.0L, 64);
  c.t1a = fix_scale(rate(1) / 126.0L, 69);
  c.t1b = fix_scale(11.0L * rate(1) / 2394.0L, 69);
  c.t2a = fix_scale(rate(2) / 252.0L, 69);
  c.t2b = fix_scale(rate(2) / 63.0L, 68);
  c.t4 = fix_scale(rate(4) / 40.0L, 65);
  c.t10 = fix_scale(rate(10) / 72.0L, 65);
  c.t12 = fix_scale(rate(12) / 24.0L, 65);
  c.t16 = fix_scale(rate(16) / 8.0L, 64);
  c.t9 = fix_scale(om / 36.0L, 65);
  c.t11 = fix_scale(om / 12.0L, 65);
  c.t13 = fix_scale(om / 4.0L, 64);
  c.tw[0] = fix_scale(K.w[0], 64);
  c.tw[1] = fix_scale(K.w[1], 67);
  c.tw[2] = fix_scale(K.w[7], 68);
  c.om = fix_scale(om, 62);
  c.b1 = fix(0x8000000000000000ull - (unsigned long long)ldexpl(om, 63));
  const double w[3] = {K.w[0], K.w[1], K.w[7]};
  for (int k = 0; k < 3; ++k) {
    c.w[k] = fix_scale(w[k], 63);
    c.bw[k] = fix_scale(om * w[k], 63);
  }
  const long double W2 = 2.0L * w[1] + 8.0L * w[2], W22 = 4.0L * w[2];
  c.qa = fix_scale(W2 - 1.0L / 3.0L, 64);
  c.qb = fix_scale(9.0L * W22 - 1.0L, 64);
  c.qc = fix_scale(4.5L * W22 - 1.5L * W2, 64);
  c.w2 = 2.0 * w[1] + 8.0 * w[2];
  c.w22 = 4.0 * w[2];
  c.tau = tau;
  c.c18cs2 = c18cs2;
  return c;
}

// A cell in fixed point: deviations from the rest state and the macroscopic
// products.
struct FixCell {
  fix D[Q];
  fix dr, jx, jy, jz;                  // density deviation, momentum
  fix rxx, ryy, rzz;                   // rho u_a u_a
  fix ux, uy, uz, ir;                  // velocity, 1 / rho
};

__host__ __device__ __forceinline__ void fix_momentum(FixCell& c) {
  const fix* D = c.D;
  c.jx = (D[1] - D[2]) + (D[7] - D[8]) + (D[9] - D[10]) + (D[11] - D[12]) + (D[13] - D[14]);
  c.jy = (D[3] - D[4]) + (D[7] + D[8]) - (D[9] + D[10]) + (D[15] - D[16]) + (D[17] - D[18]);
  c.jz = (D[5] - D[6]) + (D[11] + D[12]) - (D[13] + D[14]) + (D[15] + D[16]) - (D[17] + D[18]);
}

// f -> c; false when the cell is out of the fixed-point range.
__host__ __device__ __forceinline__ bool fixed_load(const double f[Q], FixCell& c) {
  unsigned big = 0;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
#ifdef __CUDA_ARCH__
    const unsigned h = unsigned(__double2hiint(f[i])) & 0x7fffffffu;
#else
    unsigned long long b;
    memcpy(&b, &f[i], 8);
    const unsigned h = unsigned(b >> 32) & 0x7fffffffu;
#endif
    // exponents: |f_0| < 1/2, |f_i| < 1/4 (infinities and NaN have the largest)
    const unsigned v = i == 0 ? (h > 0x100000u ? h - 0x100000u : 0u) : h;
    big = big > v ? big : v;
    c.D[i] = to_fix(f[i]) - rest_of(i);
  }
  if (big >= 0x3fd00000u) return false;
  fix dr = c.D[0];
#pragma unroll
  for (int i = 1; i < Q; ++i) dr += c.D[i];
  c.dr = dr;
  fix_momentum(c);
  constexpr fix half = fix(1) << (kFix - 1);
  const fix rho = kRest + dr;
  if (!(rho >= half && rho < 4 * half)) return false;
  constexpr fix lim = fix(1) << (kFix - 2);
  if (!(c.jx > -lim && c.jx < lim && c.jy > -lim && c.jy < lim && c.jz > -lim && c.jz < lim))
    return false;
  // 1 / rho by Newton's method (as a power series) from an FP32 seed: with
  // e = 1 - rho r0, |e| < 2^-22, r0 (1 + e + e^2) is off by e^3 < 2^-66
  const float seed = 1.0f / float(unsigned(rho >> 28));             // 2^-30 / rho
  const fix r0 = fix(int(seed * 288230376151711744.0f)) << 30;      // (2^58)
  const fix e = (fix(1) << kFix) - mulhi(rho << 3, r0 << 3);
  c.ir = r0 + mulf(e + mulf(e, e), r0);
  c.ux = mulf(c.jx, c.ir);
  c.uy = mulf(c.jy, c.ir);
  c.uz = mulf(c.jz, c.ir);
  c.rxx = mulf(c.jx, c.ux);
  c.ryy = mulf(c.jy, c.uy);
  c.rzz = mulf(c.jz, c.uz);
  return true;
}

// |u| > 0.4 as the guard tests it (unstable_rj): |j|^2 > 0.16 rho^2; the
// density bounds lie outside or at the edge of the fixed-point range.
__host__ __device__ __forceinline__ bool fixed_fast(const FixCell& c) {
  constexpr fix k016 = 46116860184273879LL;                 // 0.16 * 2^58
  return c.rxx + c.ryy + c.rzz > mulf(k016, kRest + c.dr);
}

// sqrt(x) and 1 / x of normal FP32-range x > 0 by Newton's method from an FP32
// seed (coupled iteration for x^1/2 and x^-1/2 / 2, as Markstein gives it):
// 22 -> 44 -> 88 bits, the last step rounding once.
__host__ __device__ __forceinline__ double newton_sqrt(double x) {
#ifdef __CUDA_ARCH__
  const float y = rsqrtf(float(x));
#else
  const float y = 1.0f / sqrtf(float(x));
#endif
  double s = x * double(y), h = 0.5 * double(y);
  const double r = fma(-h, s, 0.5);
  s = fma(s, r, s);
  h = fma(h, r, h);
  return fma(h, fma(-s, s, x), s);
}
__host__ __device__ __forceinline__ double newton_rcp(double x) {
  const double r = double(1.0f / float(x));
  const double e = fma(-x, r, 1.0);
  return fma(fma(e, e, e), r, r);
}

// Eddy viscosity of a loaded cell (see smag_pi, smag_tau): the non-equilibrium
// stress in fixed point, the roots in FP64.
struct FixEddy {
  double s[6];             // stress xx, yy, zz, xy, xz, yz
  double pi, inv, R, omega;   // |stress|, 1 / (rho + 1e-10), root, 1 / tau_eff
};
__host__ __device__ __forceinline__ FixEddy fixed_eddy(const FixCell& c, const FixConsts& K) {
  const fix* D = c.D;
  const fix rxy = mulf(c.jx, c.uy), rxz = mulf(c.jx, c.uz), ryz = mulf(c.jy, c.uz);
  const fix a1 = D[1] + D[2], a3 = D[3] + D[4], a5 = D[5] + D[6];
  const fix pxy = D[7] + D[10], qxy = D[8] + D[9];
  const fix pxz = D[11] + D[14], qxz = D[12] + D[13];
  const fix pyz = D[15] + D[18], qyz = D[16] + D[17];
  const fix sxy = pxy + qxy, sxz = pxz + qxz, syz = pyz + qyz;
  const fix rho = kRest + c.dr;
  constexpr fix third = 6148914691236517205LL;              // 2^64 / 3
  const fix base = mulhi(c.dr, third) + mulhi(rho, K.qa);
  const fix xx = 3 * c.rxx, yy = 3 * c.ryy, zz = 3 * c.rzz;
  FixEddy e;
  e.s[0] = from_fix(a1 + sxy + sxz - base - c.rxx - mulhi(xx, K.qa) - mulhi(c.ryy + c.rzz, K.qc));
  e.s[1] = from_fix(a3 + sxy + syz - base - c.ryy - mulhi(yy, K.qa) - mulhi(c.rxx + c.rzz, K.qc));
  e.s[2] = from_fix(a5 + sxz + syz - base - c.rzz - mulhi(zz, K.qa) - mulhi(c.rxx + c.ryy, K.qc));
  e.s[3] = from_fix(pxy - qxy - rxy - mulhi(rxy, K.qb));
  e.s[4] = from_fix(pxz - qxz - rxz - mulhi(rxz, K.qb));
  e.s[5] = from_fix(pyz - qyz - ryz - mulhi(ryz, K.qb));
  const double* s = e.s;
  const double pi2 = fma(s[0], s[0], fma(s[1], s[1], s[2] * s[2])) +
                     2.0 * fma(s[3], s[3], fma(s[4], s[4], s[5] * s[5]));
  // (below 1e-16 the stress is rounding noise and changes tau by less than an ulp)
  e.pi = pi2 > 1e-32 ? newton_sqrt(pi2) : 0.0;
  const double ir = from_fix(c.ir);
  e.inv = fma(-1e-10 * ir, ir, ir);                         // 1 / (rho + 1e-10)
  e.R = newton_sqrt(fma(K.c18cs2 * e.pi, e.inv, K.tau * K.tau));
  e.omega = newton_rcp(0.5 * (K.tau + e.R));
  return e;
}

// Collision of a loaded cell (see collide_cell_rj): BGK or MRT, with the eddy
// viscosity when smag; emits each post-collision population in units of
// 2^-fix_out(MRT).
// MRT works on m - m_eq of the deviations; with the rest state's moments and
// the conserved ones eliminated,
//   m1 - m1eq = 19 (se - D0 - rho u^2)      m2 - m2eq = 9 D0 - 7 sf - 2 se + 5.5 rho u^2
//   m4 - m4eq = 5/3 (jx_edges - 2 (D1 - D2)), m6 and m8 alike,
// (sf, se: sums over faces and edges), and the factors go into the rates.
__host__ __device__ constexpr int fix_out(bool mrt) { return mrt ? 61 : 59; }
template <bool MRT, class Out>
__host__ __device__ __forceinline__ void fixed_collide(const FixCell& c, bool smag,
                                                       const FixConsts& K, Out out) {
  const fix* D = c.D;
  const fix rxy = mulf(c.jx, c.uy), rxz = mulf(c.jx, c.uz), ryz = mulf(c.jy, c.uz);
  const fix ru2 = c.rxx + c.ryy + c.rzz;
  const fix a1 = D[1] + D[2], a3 = D[3] + D[4], a5 = D[5] + D[6];
  const fix pxy = D[7] + D[10], qxy = D[8] + D[9];
  const fix pxz = D[11] + D[14], qxz = D[12] + D[13];
  const fix pyz = D[15] + D[18], qyz = D[16] + D[17];
  const fix sxy = pxy + qxy, sxz = pxz + qxz, syz = pyz + qyz;
  fix om = 0;                          // omega of the eddy viscosity (2^58)
  if (smag) om = to_fix(fixed_eddy(c, K).omega);
  if (MRT) {
    const fix dd1 = D[1] - D[2], dd3 = D[3] - D[4], dd5 = D[5] - D[6];
    const fix u1 = D[7] - D[10], u2 = D[9] - D[8];
    const fix v1 = D[11] - D[14], v2 = D[13] - D[12];
    const fix w1 = D[15] - D[18], w2 = D[17] - D[16];
    const fix jx_xy = u1 + u2, jy_xy = u1 - u2, jx_xz = v1 + v2, jz_xz = v1 - v2;
    const fix jy_yz = w1 + w2, jz_yz = w1 - w2;
    const fix se = sxy + sxz + syz;
    const fix t9 = sxy + sxz - 2 * syz, t11 = sxy - sxz;
    const fix pxx = 2 * c.rxx - c.ryy - c.rzz, pww = c.ryy - c.rzz;
    const fix d1 = mulhi(se - D[0] - ru2, K.m1);
    // 9 D0 - 7 sf - 2 se with sf = dr - D0 - se
    const fix d2 = mulhi(16 * D[0] - 7 * c.dr + 5 * se + 5 * ru2 + (ru2 >> 1), K.m2);
    const fix d4 = mulhi((jx_xy + jx_xz - 2 * dd1) << 1, K.m4);
    const fix d6 = mulhi((jy_xy + jy_yz - 2 * dd3) << 1, K.m4);
    const fix d8 = mulhi((jz_xz + jz_yz - 2 * dd5) << 1, K.m4);
    const fix n9 = 2 * a1 - a3 - a5 + t9 - pxx, n11 = a3 - a5 + t11 - pww;
    const fix n13 = pxy - qxy - rxy, n14 = pyz - qyz - ryz, n15 = pxz - qxz - rxz;
    fix d9, d11, d13, d14, d15;
    if (smag) {
      constexpr fix c36 = 512409557603043101LL, c12 = 1537228672809129301LL;  // 2^64 / 36, / 12
      const fix o = om << 4;
      d9 = mulhi(mulhi(n9 << 2, o), c36 << 3);
      d11 = mulhi(mulhi(n11 << 2, o), c12 << 1) << 2;
      d13 = mulhi(n13 << 3, o);        // (58 + 3 + 62 - 64 = 59: omega n13 / 4 in 2^-61)
      d14 = mulhi(n14 << 3, o);
      d15 = mulhi(n15 << 3, o);
    } else {
      d9 = mulhi(n9, K.s9);
      d11 = mulhi(n11 << 2, K.s11);
      d13 = mulhi(n13 << 3, K.s13);
      d14 = mulhi(n14 << 3, K.s13);
      d15 = mulhi(n15 << 3, K.s13);
    }
    const fix d10 = mulhi(2 * (a3 + a5) - 4 * a1 + t9 + (pxx >> 1), K.m10);
    const fix d12 = mulhi((t11 - 2 * (a3 - a5) + (pww >> 1)) << 1, K.m12);
    const fix d16 = mulhi((jx_xy - jx_xz) << 3, K.m16);
    const fix d17 = mulhi((jy_yz - jy_xy) << 3, K.m16);
    const fix d18 = mulhi((jz_xz - jz_yz) << 3, K.m16);
    // f - M^T d (mrt_back), the rest state added back
    auto put = [&](int i, fix t) { out(i, ((D[i] + rest_of(i)) << 3) - t); };
    const fix cf = -11 * d1 - 4 * d2, ce = 8 * d1 + d2;
    const fix x9 = d9 - 2 * d10, y11 = d11 - 2 * d12, e9 = d9 + d10, e11 = d11 + d12;
    const fix fx = cf + 2 * x9, fy = cf - x9 + y11, fz = cf - x9 - y11;
    put(0, 12 * d2 - 30 * d1);
    put(1, fx - 4 * d4);
    put(2, fx + 4 * d4);
    put(3, fy - 4 * d6);
    put(4, fy + 4 * d6);
    put(5, fz - 4 * d8);
    put(6, fz + 4 * d8);
    const fix exy = ce + e9 + e11, exz = ce + e9 - e11, eyz = ce - 2 * e9;
    {
      const fix p = exy + d13, m = exy - d13;
      const fix g = (d4 + d16), h = (d6 - d17);     // rows 4 + 16 along x, 6 - 17 along y
      put(7, p + g + h);
      put(8, m - g + h);
      put(9, m + g - h);
      put(10, p - g - h);
    }
    {
      const fix p = exz + d15, m = exz - d15;
      const fix g = (d4 - d16), h = (d8 + d18);
      put(11, p + g + h);
      put(12, m - g + h);
      put(13, m + g - h);
      put(14, p - g - h);
    }
    {
      const fix p = eyz + d14, m = eyz - d14;
      const fix g = (d6 + d17), h = (d8 - d18);
      put(15, p + g + h);
      put(16, m - g + h);
      put(17, m + g - h);
      put(18, p - g - h);
    }
  } else {
    // f - omega (f - feq), feq_i = w_i (rho + 3 e.j + 4.5 rho (e.u)^2 - 1.5 rho u^2)
    const fix base = kRest + c.dr - ru2 - (ru2 >> 1);
    fix b1 = 0, ow[3] = {0, 0, 0};
    if (smag) {
      b1 = (fix(1) << 62) - (om << 4);               // (1 - omega) 2^62, then 2^63
      b1 = fix((unsigned long long)b1 << 1);
      for (int k = 0; k < 3; ++k) ow[k] = mulhi(om << 4, K.w[k]) << 2;
    } else {
      b1 = K.b1;
      for (int k = 0; k < 3; ++k) ow[k] = K.bw[k];
    }
    auto put = [&](int i, fix t) {
      // two products rounded down, half a unit each
      out(i, mulhi((D[i] + rest_of(i)) << 2, b1) + mulhi(t << 2, ow[i == 0 ? 0 : (i < 7 ? 1 : 2)]) +
                 1);
    };
    auto pair = [&](int i, int io, fix j, fix r) {   // e.j, rho (e.u)^2
      const fix s = base + 4 * r + (r >> 1), t = 3 * j;
      put(i, s + t);
      put(io, s - t);
    };
    put(0, base);
    pair(1, 2, c.jx, c.rxx);
    pair(3, 4, c.jy, c.ryy);
    pair(5, 6, c.jz, c.rzz);
    pair(7, 10, c.jx + c.jy, c.rxx + c.ryy + 2 * rxy);
    pair(9, 8, c.jx - c.jy, c.rxx + c.ryy - 2 * rxy);
    pair(11, 14, c.jx + c.jz, c.rxx + c.rzz + 2 * rxz);
    pair(13, 12, c.jx - c.jz, c.rxx + c.rzz - 2 * rxz);
    pair(15, 18, c.jy + c.jz, c.ryy + c.rzz + 2 * ryz);
    pair(17, 16, c.jy - c.jz, c.ryy + c.rzz - 2 * ryz);
  }
}

// ---------------------------------------------------------------------------
// Transposed collision.  The cotangents of a cell are integers with one exponent
// for the cell: F_i = mu_i 2^sh, |F_i| < 2^56 (a cotangent field spans many
// orders of magnitude over the domain, a cell's 19 values do not; what a term
// loses is below 2^-57 of the cell's largest value, where an FP64 sum of them
// rounds by 2^-54 and more).  Products with the velocity take it from the fixed-point
// cell.  Every bound below is for the worst alignment of signs, so nothing can
// overflow.  The rms error against extended precision is 0.2 to 0.7 of the FP64
// form's (tests/test_fixed64_cpu.py, and at the limits tests/test_fixed64_limits.py).
// Measured, us a step of a run and its adjoint, both before and after in fixed point:
// 64x32x32 131 -> 45, 96x48x48 353 -> 83, 128x64x64 795 -> 146; with the eddy viscosity
// and a porosity blend 229 -> 78, 642 -> 166, 1494 -> 319.
// ---------------------------------------------------------------------------

// mu -> F and sh; false for infinite, NaN or extreme values, or all zero (whose
// transpose is zero, without any arithmetic).
__host__ __device__ __forceinline__ bool fixed_load_T(const double mu[Q], fix F[Q], int& sh) {
  unsigned hi[Q], lo[Q], top = 0;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
#ifdef __CUDA_ARCH__
    hi[i] = unsigned(__double2hiint(mu[i]));
    lo[i] = unsigned(__double2loint(mu[i]));
#else
    unsigned long long b;
    memcpy(&b, &mu[i], 8);
    hi[i] = unsigned(b >> 32);
    lo[i] = unsigned(b);
#endif
    const unsigned h = hi[i] & 0x7fffffffu;
    top = top > h ? top : h;
  }
  const unsigned E = top >> 20;                    // biased exponent of the largest
  if (E < 128 || E > 1980) return false;
  sh = 1078 - int(E);
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const unsigned mh = ((hi[i] << 11) | (lo[i] >> 21)) | 0x80000000u, ml = lo[i] << 11;
    const unsigned s = 7u + E - ((hi[i] >> 20) & 0x7ffu);   // one bit short, then rounded
    unsigned long long m = (unsigned long long)mh << 32 | ml;
#ifdef __CUDA_ARCH__
    asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(s));
#else
    m = s > 63 ? 0 : m >> s;
#endif
    m = (m + 1) >> 1;
    const fix g = fix(int(hi[i]) >> 31);
    F[i] = (fix(m) ^ g) - g;
  }
  return true;
}

// x 2^-bits as a double, rounded to nearest even (a normal result)
__host__ __device__ __forceinline__ double from_fix_at(fix x, int bits) {
  const fix g = x >> 63;
  const unsigned long long a = (unsigned long long)((x ^ g) - g);
#ifdef __CUDA_ARCH__
  const int z = __clzll((long long)a);
#else
  const int z = a ? __builtin_clzll(a) : 64;
#endif
  unsigned long long m = a << ((z - 1) & 63);
  m = (m + 0x1ffull + ((m >> 10) & 1ull)) >> 10;
  const unsigned e = (unsigned(1085 - bits - z) << 20) | (unsigned(int(g)) & 0x80000000u);
  unsigned hi = unsigned(m >> 32) + e, lo = unsigned(m);
  if (z == 64) hi = 0;
#ifdef __CUDA_ARCH__
  return __hiloint2double(int(hi), int(lo));
#else
  const unsigned long long r = (unsigned long long)hi << 32 | lo;
  double d;
  memcpy(&d, &r, 8);
  return d;
#endif
}

// mu <- C^T mu at a loaded cell, without the eddy viscosity (collide_vjp_s in
// closed form): with d the relaxed moments of mu and w = 19 d1 - 5.5 d2,
//   h   = (2 w + ...) u + ... - 2/3 d_q     (the momentum's cotangent over rho)
//   c_0 = 3 d2 - 11 d1 - w u^2 - a9 pxx - a11 pww - d13 ux uy - ...
//   g_i = mu_i - (M^T d)_i + c_0 + e_i . h,    a9 = d9 - d10 / 2, a11 = d11 - d12 / 2;
// for BGK, with A = sum w e mu, B = sum w e e mu, s = sum w mu:
//   h = 3 omega (A + 3 B u - s u), c_0 = omega (s + 1.5 u^2 s - 4.5 u.B u).
// Intermediate results in units of 2^-(sh + 1).
__host__ __device__ __forceinline__ bool all_zero(const double mu[Q]) {
  bool z = true;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
#ifdef __CUDA_ARCH__
    z = z && (__double2hiint(mu[i]) & 0x7fffffff) == 0 && __double2loint(mu[i]) == 0;
#else
    z = z && mu[i] == 0.0;
#endif
  }
  return z;
}

// Eddy viscosity (MRT): its terms (see collide_vjp_s) are formed in FP64 from the
// cotangent of omega and come in as c_0, h and e_a e_b q_ab parts (FixEddyT).
struct FixEddyT {
  fix om;                  // omega (2^58)
  fix c0, hx, hy, hz;      // units of 2^-(sh + 1)
  fix q[6];                // xx, yy, zz, xy, xz, yz (off-diagonal ones doubled)
};

// x 2^bits, rounded
__host__ __device__ __forceinline__ fix scaled_fix(double x, double scale) {
#ifdef __CUDA_ARCH__
  return __double2ll_rn(x * scale);
#else
  return llrint(x * scale);
#endif
}

// The eddy terms of a cell; false when they are too large for the cell's exponent.
__host__ __device__ __forceinline__ bool fixed_eddy_T(const FixCell& c, const FixConsts& K, int sh,
                                                      const fix F[Q], FixEddyT& t) {
  const FixEddy e = fixed_eddy(c, K);
  const fix* D = c.D;
  double go;
  {
    // cotangent of omega: - sum over the stress moments of mu_k / norm_k (m_k - meq_k)
    const fix p1 = F[1] + F[2], p3 = F[3] + F[4], p5 = F[5] + F[6];
    const fix p7 = F[7] + F[10], p9 = F[9] + F[8], p11 = F[11] + F[14], p13 = F[13] + F[12];
    const fix p15 = F[15] + F[18], p17 = F[17] + F[16];
    const fix sxy = p7 + p9, sxz = p11 + p13, syz = p15 + p17;
    const fix a1 = D[1] + D[2], a3 = D[3] + D[4], a5 = D[5] + D[6];
    const fix pxy = D[7] + D[10], qxy = D[8] + D[9], pxz = D[11] + D[14], qxz = D[12] + D[13];
    const fix pyz = D[15] + D[18], qyz = D[16] + D[17];
    const fix rxy = mulf(c.jx, c.uy), rxz = mulf(c.jx, c.uz), ryz = mulf(c.jy, c.uz);
    const fix dxy = pxy + qxy, dxz = pxz + qxz, dyz = pyz + qyz;
    const double n9 = from_fix(2 * a1 - a3 - a5 + dxy + dxz - 2 * dyz - (2 * c.rxx - c.ryy - c.rzz));
    const double n11 = from_fix(a3 - a5 + dxy - dxz - (c.ryy - c.rzz));
    const double n13 = from_fix(pxy - qxy - rxy), n14 = from_fix(pyz - qyz - ryz);
    const double n15 = from_fix(pxz - qxz - rxz);
    const double l9 = from_fix_at(2 * p1 - p3 - p5 + sxy + sxz - 2 * syz, sh);
    const double l11 = from_fix_at(p3 - p5 + sxy - sxz, sh);
    const double l13 = from_fix_at(p7 - p9, sh), l14 = from_fix_at(p15 - p17, sh);
    const double l15 = from_fix_at(p11 - p13, sh);
    go = -(l9 * n9 * (1.0 / 36.0) + l11 * n11 * (1.0 / 12.0) +
           0.25 * (l13 * n13 + l14 * n14 + l15 * n15));
  }
  const double gX = -0.25 * go * e.omega * e.omega * newton_rcp(e.R);   // gR / (2 R), gR = g_tau_eff / 2
  const double gp = gX * K.c18cs2 * e.inv;                             // of |stress|
  double c0 = -gp * e.pi * e.inv, hx = 0.0, hy = 0.0, hz = 0.0;
  double q[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (e.pi > 0.0) {
    const double ip = gp * newton_rcp(e.pi);
#pragma unroll
    for (int k = 0; k < 6; ++k) q[k] = (k < 3 ? ip : 2.0 * ip) * e.s[k];
    const double ux = from_fix(c.ux), uy = from_fix(c.uy), uz = from_fix(c.uz);
    const double xx = ux * ux, yy = uy * uy, zz = uz * uz, c9 = 9.0 * K.w22;
    const double base = K.w2 * (1.0 - 1.5 * (xx + yy + zz)), d = 4.5 * (K.w2 - K.w22);
    const double all = fma(4.5 * K.w22, xx + yy + zz, base);   // base + 4.5 (W2 aa + W22 rest) = all + d aa
    const double qd = q[0] + q[1] + q[2];
    const double ox = fma(q[3], uy, q[4] * uz), oy = fma(q[3], ux, q[5] * uz),
                 oz = fma(q[4], ux, q[5] * uy);
    // (the rho cotangent's cross terms are half of u . o)
    const double er = all * qd + d * (q[0] * xx + q[1] * yy + q[2] * zz) +
                      0.5 * c9 * (ux * ox + uy * oy + uz * oz);
    const double own = 6.0 * K.w2, oth = 9.0 * K.w22 - 3.0 * K.w2;
    hx = -(ux * (oth * qd + (own - oth) * q[0]) + c9 * ox);
    hy = -(uy * (oth * qd + (own - oth) * q[1]) + c9 * oy);
    hz = -(uz * (oth * qd + (own - oth) * q[2]) + c9 * oz);
    c0 -= er + (hx * ux + hy * uy + hz * uz);
  }
  const double scale = ldexp(1.0, sh + 1);
  double top = fabs(c0);
  top = fmax(top, fmax(fabs(hx), fmax(fabs(hy), fabs(hz))));
#pragma unroll
  for (int k = 0; k < 6; ++k) top = fmax(top, fabs(q[k]));
  if (!(top * scale < 144115188075855872.0)) return false;           // 2^57
  t.om = to_fix(e.omega);
  t.c0 = scaled_fix(c0, scale);
  t.hx = scaled_fix(hx, scale);
  t.hy = scaled_fix(hy, scale);
  t.hz = scaled_fix(hz, scale);
#pragma unroll
  for (int k = 0; k < 6; ++k) t.q[k] = scaled_fix(q[k], scale);
  return true;
}

template <bool MRT, bool EDDY = false>
__host__ __device__ __forceinline__ void fixed_collide_T(const FixCell& c, const FixConsts& K,
                                                         int sh, const fix F[Q], double mu[Q],
                                                         const FixEddyT* ed = nullptr) {
  // velocity times 2^63 and its products (|u_a| < 1/2)
  const fix ux = c.ux << 5, uy = c.uy << 5, uz = c.uz << 5;
  const fix xx = mulhi(ux, c.ux), yy = mulhi(uy, c.uy), zz = mulhi(uz, c.uz);   // 2^57
  const fix p1 = F[1] + F[2], m1 = F[1] - F[2], p3 = F[3] + F[4], m3 = F[3] - F[4];
  const fix p5 = F[5] + F[6], m5 = F[5] - F[6];
  const fix p7 = F[7] + F[10], m7 = F[7] - F[10], p9 = F[9] + F[8], m9 = F[9] - F[8];
  const fix p11 = F[11] + F[14], m11 = F[11] - F[14], p13 = F[13] + F[12], m13 = F[13] - F[12];
  const fix p15 = F[15] + F[18], m15 = F[15] - F[18], p17 = F[17] + F[16], m17 = F[17] - F[16];
  const int bits = sh + 1;
  if (MRT) {
    const fix u2 = (xx + yy + zz) << 6;                     // 2^63
    const fix uxy = mulhi(ux, c.uy) << 6, uxz = mulhi(ux, c.uz) << 6, uyz = mulhi(uy, c.uz) << 6;
    const fix pxx = (2 * xx - yy - zz) << 6, pww = (yy - zz) << 6;
    const fix sf = p1 + p3 + p5;
    const fix sxy = p7 + p9, sxz = p11 + p13, syz = p15 + p17, se = sxy + sxz + syz;
    const fix jx_xy = m7 + m9, jy_xy = m7 - m9, jx_xz = m11 + m13, jz_xz = m11 - m13;
    const fix jy_yz = m15 + m17, jz_yz = m15 - m17;
    const fix m0 = F[0] + sf + se;
    const fix t9 = sxy + sxz - 2 * syz, t11 = sxy - sxz;
    // relaxed moments, in units of 2^-(sh + 1); d1 and d2, which the transform
    // multiplies by up to 30, in units of 2^-(sh + 5)
    const fix d1h = mulhi(se - F[0], K.t1a) - mulhi(m0, K.t1b);
    const fix d2h = mulhi(16 * F[0] + 5 * se, K.t2a) - mulhi(m0 << 1, K.t2b);
    const fix d4 = mulhi(jx_xy + jx_xz - 4 * m1, K.t4);
    const fix d6 = mulhi(jy_xy + jy_yz - 4 * m3, K.t4);
    const fix d8 = mulhi(jz_xz + jz_yz - 4 * m5, K.t4);
    const fix l9 = 2 * p1 - p3 - p5 + t9, l11 = p3 - p5 + t11;
    fix d9, d11, d13, d14, d15;
    if (EDDY) {
      // omega 2^62; 2^65 / 36, 2^65 / 12
      constexpr fix c36 = 1024819115206086201LL, c12 = 3074457345618258603LL;
      const fix o = ed->om << 4;
      d9 = mulhi(mulhi(l9 << 2, o), c36);
      d11 = mulhi(mulhi(l11 << 2, o), c12);
      d13 = mulhi((p7 - p9) << 1, o);
      d14 = mulhi((p15 - p17) << 1, o);
      d15 = mulhi((p11 - p13) << 1, o);
    } else {
      d9 = mulhi(l9, K.t9);
      d11 = mulhi(l11, K.t11);
      d13 = mulhi((p7 - p9) << 1, K.t13);
      d14 = mulhi((p15 - p17) << 1, K.t13);
      d15 = mulhi((p11 - p13) << 1, K.t13);
    }
    const fix d10 = mulhi(2 * (p3 + p5) - 4 * p1 + t9, K.t10);
    const fix d12 = mulhi(t11 - 2 * (p3 - p5), K.t12);
    const fix d16 = mulhi((jx_xy - jx_xz) << 1, K.t16);
    const fix d17 = mulhi((jy_yz - jy_xy) << 1, K.t16);
    const fix d18 = mulhi((jz_xz - jz_yz) << 1, K.t16);
    const fix a9 = d9 - (d10 >> 1), a11 = d11 - (d12 >> 1);
    const fix d1x11 = (11 * d1h + 8) >> 4, d2x4 = (d2h + 2) >> 2;
    const fix q12 = (19 * (d1h >> 2) >> 1) - (11 * (d2h >> 2) >> 2);
    constexpr fix third = 6148914691236517205LL;            // 2^64 / 3
    // (a product with a velocity comes out halved)
    fix hx = (mulhi(q12 + 4 * a9, ux) + mulhi(d13, uy) + mulhi(d15, uz) - mulhi(d4, third)) * 2 + 2;
    fix hy = (mulhi(q12 - 2 * (a9 - a11), uy) + mulhi(d13, ux) + mulhi(d14, uz) -
                    mulhi(d6, third)) * 2 + 2;
    fix hz = (mulhi(q12 - 2 * (a9 + a11), uz) + mulhi(d14, uy) + mulhi(d15, ux) -
                    mulhi(d8, third)) * 2 + 2;
    fix c0 = ((3 * d2h + 8) >> 4) - d1x11 - mulhi(q12, u2) -
                   ((mulhi(a9, pxx) + mulhi(a11, pww) + mulhi(d13, uxy) + mulhi(d14, uyz) +
                     mulhi(d15, uxz)) * 2 + 5);
    fix q0 = 0, q1 = 0, q2 = 0, q3 = -d13, q4 = -d15, q5 = -d14;   // e_a e_b terms
    if (EDDY) {
      c0 += ed->c0;
      hx += ed->hx;
      hy += ed->hy;
      hz += ed->hz;
      q0 = ed->q[0];
      q1 = ed->q[1];
      q2 = ed->q[2];
      q3 += ed->q[3];
      q4 += ed->q[4];
      q5 += ed->q[5];
    }
    auto put = [&](int i, fix t) { mu[i] = from_fix_at(2 * F[i] + t, bits); };
    // c_0 + e.h - M^T d (mrt_back)
    const fix cf = c0 + d1x11 + d2x4, ce = c0 - ((d1h + 1) >> 1) - ((d2h + 8) >> 4);
    const fix x9 = d9 - 2 * d10, y11 = d11 - 2 * d12, e9 = d9 + d10 + 1, e11 = d11 + d12 + 1;
    const fix fx = cf - 2 * x9 + q0, fy = cf + x9 - y11 + q1, fz = cf + x9 + y11 + q2;
    const fix gx = hx + 4 * d4 + 2, gy = hy + 4 * d6 + 2, gz = hz + 4 * d8 + 2;
    put(0, c0 + ((15 * d1h + 4) >> 3) - ((3 * d2h + 2) >> 2));
    put(1, fx + gx);
    put(2, fx - gx);
    put(3, fy + gy);
    put(4, fy - gy);
    put(5, fz + gz);
    put(6, fz - gz);
    const fix exy = ce - e9 - e11 + q0 + q1, exz = ce - e9 + e11 + q0 + q2;
    const fix eyz = ce + 2 * e9 + q1 + q2;
    {
      const fix p = exy + q3, m = exy - q3;
      const fix g = hx - d4 - d16, h = hy - d6 + d17;
      put(7, p + g + h);
      put(8, m - g + h);
      put(9, m + g - h);
      put(10, p - g - h);
    }
    {
      const fix p = exz + q4, m = exz - q4;
      const fix g = hx - d4 + d16, h = hz - d8 - d18;
      put(11, p + g + h);
      put(12, m - g + h);
      put(13, m + g - h);
      put(14, p - g - h);
    }
    {
      const fix p = eyz + q5, m = eyz - q5;
      const fix g = hy - d6 - d17, h = hz - d8 + d18;
      put(15, p + g + h);
      put(16, m - g + h);
      put(17, m + g - h);
      put(18, p - g - h);
    }
  } else {
    // sums over the weights in units of 2^-(sh + 4), the rest scaled back at the end
    // (a floor is half a unit low: sums of products that are multiplied on are put right)
    auto wf = [&](fix x) { return mulhi(x << 1, K.tw[1]); };
    auto we = [&](fix x) { return mulhi(x, K.tw[2]); };
    const fix s = mulhi(F[0] << 4, K.tw[0]) + wf(p1 + p3 + p5) +
                  we(p7 + p9 + p11 + p13 + p15 + p17);
    const fix ax = wf(m1) + we(m7 + m9 + m11 + m13) + 1;
    const fix ay = wf(m3) + we(m7 - m9 + m15 + m17) + 1;
    const fix az = wf(m5) + we(m11 - m13 + m15 - m17) + 1;
    const fix bxx = wf(p1) + we(p7 + p9 + p11 + p13);
    const fix byy = wf(p3) + we(p7 + p9 + p15 + p17);
    const fix bzz = wf(p5) + we(p11 + p13 + p15 + p17);
    const fix bxy = we(p7 - p9), bxz = we(p11 - p13), byz = we(p15 - p17);
    const fix vx = (mulhi(bxx, ux) + mulhi(bxy, uy) + mulhi(bxz, uz)) * 2 + 3;
    const fix vy = (mulhi(bxy, ux) + mulhi(byy, uy) + mulhi(byz, uz)) * 2 + 3;
    const fix vz = (mulhi(bxz, ux) + mulhi(byz, uy) + mulhi(bzz, uz)) * 2 + 3;
    const fix ubu = (mulhi(vx, ux) + mulhi(vy, uy) + mulhi(vz, uz)) * 2 + 3;
    const fix su2 = mulhi(s, (xx + yy + zz) << 6) << 1;
    auto om = [&](fix x) { return mulhi(x << 1, K.om); };    // units of 2^-(sh + 3)
    auto back = [&](fix x) { return (x + 2) >> 2; };         // to 2^-(sh + 1), rounded
    const fix hx = back(3 * om(ax + 3 * vx - (mulhi(s, ux) << 1)));
    const fix hy = back(3 * om(ay + 3 * vy - (mulhi(s, uy) << 1)));
    const fix hz = back(3 * om(az + 3 * vz - (mulhi(s, uz) << 1)));
    const fix c0 = back(om(s + su2 + (su2 >> 1) - 4 * ubu - (ubu >> 1)));
    auto put = [&](int i, fix t) { mu[i] = from_fix_at(mulhi(F[i] << 2, K.b1) + t, bits); };
    put(0, c0);
    put(1, c0 + hx);
    put(2, c0 - hx);
    put(3, c0 + hy);
    put(4, c0 - hy);
    put(5, c0 + hz);
    put(6, c0 - hz);
    put(7, c0 + hx + hy);
    put(10, c0 - hx - hy);
    put(9, c0 + hx - hy);
    put(8, c0 - hx + hy);
    put(11, c0 + hx + hz);
    put(14, c0 - hx - hz);
    put(13, c0 + hx - hz);
    put(12, c0 - hx + hz);
    put(15, c0 + hy + hz);
    put(18, c0 - hy - hz);
    put(17, c0 + hy - hz);
    put(16, c0 - hy + hz);
  }
}

}  // namespace lbm
