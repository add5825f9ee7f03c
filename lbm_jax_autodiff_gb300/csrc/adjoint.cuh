// Adjoint (reverse-mode) time step of the fused solver: the hand-derived
// transpose of one forward step, giving dCd/dr and dCd/dq without storing
// any per-step intermediate beyond the populations S_k.
//
// Forward (one step k):  f_k = Z(T_q(S_{k-1})),  S_k = B_p(C(f_k))
//   T_q : pull streaming + Bouzidi with wall distances q   streaming.py:40-185
//   Z   : Zou-He inlet / outlet (affine in f)              boundary.py:35-200
//   C   : BGK / MRT collision (+ Smagorinsky)               collision.py:46-270
//   B_p : hard bounce-back or sigmoid-porosity blend        smooth.py:118-155
// Objective: Cd(F(S_{N-1}, f_N)) with the momentum-exchange force F
// (forces.py:37-120, 237-276) -- the reference drivers' simulate_cd
// (examples/11:139-165) whose gradient jax.grad derives.
//
// Adjoint state stored between launches: nu_k = Z^T lambda_k, the cotangent
// of the streamed (pre-boundary) populations of step k.  One launch of
// k_adjoint for step k does, per cell y:
//   mu_k(y)  = (T_q^T nu_{k+1})(y)      gather form of the transposed stream
//   f_k(y)   = recomputed from the stashed S_{k-1}
//   dJ/dp   += mu_k . dB/dp  (sigmoid porosity, dp/dr = alpha p (1-p))
//   dJ/dq   += nu_{k+1} . dT/dq (S_k), per wall link, times dq/dr
//   lambda_k = C^T B^T mu_k;  nu_k = Z^T lambda_k on the inlet/outlet faces
#pragma once

#include "batch.cuh"
#include "capi_util.cuh"
#include "sim.cuh"
#include "vec2.cuh"

namespace lbm {

template <class Re> struct AdjArgs {
  StepArgs<Re> s;          // forward description; s.src = S_{k-1} (or f_0 when first)
  const void* S_k;         // stashed S_k (storage type), for q < 0.5 neighbour reads
  const Re* nu_in;         // nu_{k+1}
  Re* nu_out;              // nu_k (lambda_0 when first)
  int first;               // k == 0
  int last;                // k == N-1: add dJ/dS_{N-1} of the momentum exchange
  const double* dj_dfx;    // device scalar dJ/dFx
  double* gr_partials;     // [gridDim.x] running dJ/dr per block
  double* gq;              // [nrec][19] running dJ/dq per link
};

// Zou-He transposes (affine maps; see boundary.py:95-122 and :176-198).
template <class Re>
__device__ __forceinline__ void zou_he_inlet_T(Re l[Q], Re ux, Re uy, Re uz) {
  const Re c3 = Re(1.0 / 3.0), c6 = Re(1.0 / 6.0);
  const Re grho = c3 * ux * l[1] + c6 * (ux + uy) * l[7] + c6 * (ux - uy) * l[9] +
                  c6 * (ux + uz) * l[11] + c6 * (ux - uz) * l[13];
  const Re d = grho / (Re(1) - ux);
  Re o[Q];
#pragma unroll
  for (int j = 0; j < Q; ++j) o[j] = l[j];
  o[1] = o[7] = o[9] = o[11] = o[13] = Re(0);
  o[2] += l[1];
  o[10] += l[7];
  o[8] += l[9];
  o[14] += l[11];
  o[12] += l[13];
  o[0] += d; o[3] += d; o[4] += d; o[5] += d; o[6] += d;
  o[15] += d; o[16] += d; o[17] += d; o[18] += d;
  o[2] += Re(2) * d; o[8] += Re(2) * d; o[10] += Re(2) * d; o[12] += Re(2) * d;
  o[14] += Re(2) * d;
#pragma unroll
  for (int j = 0; j < Q; ++j) l[j] = o[j];
}

template <class Re>
__device__ __forceinline__ void zou_he_outlet_T(Re l[Q], Re rho_out) {
  const Re c3 = Re(1.0 / 3.0), c6 = Re(1.0 / 6.0);
  const Re gu = -rho_out * (c3 * l[2] + c6 * (l[10] + l[8] + l[14] + l[12]));
  const Re d = gu / rho_out;
  Re o[Q];
#pragma unroll
  for (int j = 0; j < Q; ++j) o[j] = l[j];
  o[2] = o[10] = o[8] = o[14] = o[12] = Re(0);
  o[1] += l[2];
  o[7] += l[10];
  o[9] += l[8];
  o[11] += l[14];
  o[13] += l[12];
  o[0] += d; o[3] += d; o[4] += d; o[5] += d; o[6] += d;
  o[15] += d; o[16] += d; o[17] += d; o[18] += d;
  o[1] += Re(2) * d; o[7] += Re(2) * d; o[9] += Re(2) * d; o[11] += Re(2) * d;
  o[13] += Re(2) * d;
#pragma unroll
  for (int j = 0; j < Q; ++j) l[j] = o[j];
}

// dJ/dq of the wall links owned by a cell at this step, d T(S_k)/dq with
// S_k = B(c) (c = C(f_k)); accumulates per link.  (dJ/dr = sum dJ/dq dq/dr is summed
// once at the end, k_link_gr: dq/dr does not change over the steps, and the FP64
// operations of a sum per step were 3 of the list's 16 us on small grids.)
// With q = q[opp i] of the link that direction i reads:
//   q >= 0.5: T_i = a S_io + (1 - a) S_i, a = 1 / (2 clip(q, 0.5, 1))
//   q <  0.5: T_i = b S_io + (1 - b) S_io(x + e_i), b = 2 clip(q, 0, 0.5)
// so dT_i/dq = gc (S_io - other) with the record's gc = da/dq or db/dq.
// The loads of a group of three pairs of directions are issued together
// (see bouzidi).  LATE: all stores at the end, since a group's coherent loads do not pass
// the stores of the group before (the split list, whose launch lasts as long as
// this chain: 200 steps and their adjoint at 96x48x48 4.70 -> 4.59 ms; where
// many cells fill the chip the 18 sums' registers cost more, 60 steps of 256x128x128
// FP16 18.44 -> 18.57 ms, twelve domains 119.5 -> 120.3).
template <class St, bool LATE = false>
__device__ __forceinline__ void link_q_grad(const AdjArgs<typename Storage<St>::Re>& A,
                                            const typename Storage<St>::Re c[Q],
                                            typename Storage<St>::Re p, bool soft, bool hard,
                                            uint32_t ri, int idx, int x, int y, int z) {
  using Re = typename Storage<St>::Re;
  using S = Storage<St>;
  const StepArgs<Re>& a = A.s;
  const Grid& g = a.g;
  const size_t N = size_t(g.n);
  const LinkRec<Re>& r = a.rec[ri - 1];
  const uint32_t lm = r.linkmask, low = r.low;
  const St* Sk = static_cast<const St*>(A.S_k);
  const NearMask M(g, a.near, x, y, z, 1);
  double* gq = A.gq + size_t(ri - 1) * Q;
  double sum[Q];
#pragma unroll
  for (int k0 = 0; k0 < 9; k0 += 3) {
    Re nv[6], sn[6], gc[6];
    double old[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int i = (k & 1) ? opp(pair_dir(k0 + (k >> 1))) : pair_dir(k0 + (k >> 1));
      const int io = opp(i);
      nv[k] = ld_c(A.nu_in + i * N + idx);
      gc[k] = __ldg(&r.gc[io]);
      old[k] = gq[io];
      // (the cell's own value in the place of one that is not needed)
      const int nb = ((low >> io) & 1u) ? ahead_wrap(g, x, y, z, ex(i), ey(i), ez(i)) : idx;
      sn[k] = S::ld(Sk + io * N + nb, M.nbr_in(i) ? a.soff_near[io] : a.soff[io]);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int i = (k & 1) ? opp(pair_dir(k0 + (k >> 1))) : pair_dir(k0 + (k >> 1));
      const int io = opp(i);
      const Re s_io = soft ? (Re(1) - p) * c[io] + p * c[i] : (hard ? c[i] : c[io]);
      const Re s_i = soft ? (Re(1) - p) * c[i] + p * c[io] : (hard ? c[io] : c[i]);
      const Re dout = gc[k] * (s_io - (((low >> io) & 1u) ? sn[k] : s_i));
      sum[io] = old[k] + double(nv[k]) * double(dout);
      if (!LATE && ((lm >> io) & 1u)) gq[io] = sum[io];
    }
  }
  if (LATE) {
#pragma unroll
    for (int j = 1; j < Q; ++j)
      if ((lm >> j) & 1u) gq[j] = sum[j];
  }
}

// A cell's part of dJ/dr = sum over links of dJ/dq dq/dr.
template <class Re>
__device__ __forceinline__ double link_gr(uint32_t tag, const LinkRec<Re>* rec, const double* gq) {
  const uint32_t ri = tag & TAG_INDEX;
  if (!ri) return 0.0;
  const LinkRec<Re>& r = rec[ri - 1];
  double v = 0.0;
#pragma unroll
  for (int j = 1; j < Q; ++j)
    if ((r.linkmask >> j) & 1u) v += gq[size_t(ri - 1) * Q + j] * double(r.dqdr[j]);
  return v;
}

// The record cells' corrections of the plain gather in mu: the transposed
// Bouzidi terms and, at the last step, the seed dJ/dS_{N-1} of the momentum
// exchange.
template <class Re>
__device__ __forceinline__ void gather_record(const AdjArgs<Re>& A, uint32_t ri, int idx, int x,
                                              int y, int z, Re mu[Q]) {
  const StepArgs<Re>& a = A.s;
  const Grid& g = a.g;
  const size_t N = size_t(g.n);
  const Re* nu = A.nu_in;
  // the loads of a group of three pairs of directions are issued together
  // (see bouzidi)
  const PullIdx P(g, x, y, z);
  const LinkRec<Re>& r = a.rec[ri - 1];
  const uint32_t lm = r.linkmask, nbw = r.nb_wall, nbl = r.nb_low, low = r.low;
  const Re gfx = A.last ? Re(*A.dj_dfx) : Re(0);
#pragma unroll
  for (int k0 = 0; k0 < 9; k0 += 3) {
    Re own[6], far[6], w[6], fw[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int j = (k & 1) ? opp(pair_dir(k0 + (k >> 1))) : pair_dir(k0 + (k >> 1));
      own[k] = ld_c(nu + j * N + idx);
      w[k] = __ldg(&r.w[j]);
      fw[k] = __ldg(&r.nbw[j]);
      const int nb = ((nbl >> j) & 1u) ? ahead_wrap(g, x, y, z, ex(j), ey(j), ez(j)) : idx;
      far[k] = ld_c(nu + opp(j) * N + nb);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int j = (k & 1) ? opp(pair_dir(k0 + (k >> 1))) : pair_dir(k0 + (k >> 1));
      // mu[j] holds the plain gather: nu_j(x + e_j), plus own nu_j when its
      // source is out of range
      const bool a_ok = !((nbw >> j) & 1u);
      const bool wall_out = (lm >> opp(j)) & 1u;
      Re v = mu[j];
      if (P.valid(j)) {
        if (!a_ok) v = Re(0);
      } else {
        // an edge cell: the two terms of the plain gather, each kept or dropped
        v = P.valid(opp(j)) && a_ok ? ld_c(nu + j * N + P.raw(opp(j))) : Re(0);
        if (!wall_out) v += own[k];
      }
      if ((nbl >> j) & 1u) v += fw[k] * far[k];
      mu[j] = v;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int i = (k & 1) ? opp(pair_dir(k0 + (k >> 1))) : pair_dir(k0 + (k >> 1));
      const int io = opp(i);
      const Re wi = w[k ^ 1];               // weight of the link in direction io
      if ((lm >> io) & 1u) {
        mu[io] += wi * own[k];
        if (!((low >> io) & 1u)) mu[i] += (Re(1) - wi) * own[k];
      }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int j = (k & 1) ? opp(pair_dir(k0 + (k >> 1))) : pair_dir(k0 + (k >> 1));
      if (A.last && ex(j) != 0 && ((lm >> j) & 1u)) mu[j] += Re(ex(j)) * gfx;
    }
  }
}

// mu_k(y) = (T_q^T nu_{k+1})(y) for one cell: the gather form of the
// transposed pull (x + e_j pulled S_j(y)), the fallback terms of out-of-range
// sources, and on boundary cells the transposed Bouzidi terms and, at the
// last step, the seed dJ/dS_{N-1} of the momentum exchange.
template <class Re>
__device__ __forceinline__ void gather_mu(const AdjArgs<Re>& A, int idx, int x, int y, int z,
                                          uint32_t tag, Re mu[Q]) {
  const StepArgs<Re>& a = A.s;
  const Grid& g = a.g;
  const size_t N = size_t(g.n);
  const uint32_t ri = tag & TAG_INDEX;
  const Re* nu = A.nu_in;
  // ---- mu_k = T^T nu_{k+1}: normal-stream part (gather from x + e_j) ---
  mu[0] = ld_c(nu + idx);
  {
    const NbrOff O(g, x, y, z);
    if (!O.face) {
#pragma unroll
      for (int j = 1; j < Q; ++j) mu[j] = ld_c(nu + j * N + O.push(j, idx));
    } else {
      const PullIdx P(g, x, y, z);
#pragma unroll
      for (int j = 1; j < Q; ++j) {
        // (a) output (y + e_j, j) pulls S_j(y) when that neighbour is in range
        Re v = P.valid(opp(j)) ? ld_c(nu + j * N + P.raw(opp(j))) : Re(0);
        // (b) output (y, j) keeps S_j(y) when its own source is out of range
        if (!P.valid(j)) v += ld_c(nu + j * N + idx);
        mu[j] = v;
      }
    }
  }

  // ---- boundary-cell corrections of T^T, force seed --------------------
  if (ri) gather_record<Re>(A, ri, idx, x, y, z, mu);
}

// f_k of a cell: f_0 at the first step, else the pull of S_{k-1} with its boundary
// rules (CALL as in pull_post_bc).
template <class St, bool CALL>
__device__ __forceinline__ void recompute_f(const AdjArgs<typename Storage<St>::Re>& A, int idx,
                                            int x, int y, int z, uint32_t tag,
                                            typename Storage<St>::Re f[Q]) {
  using Re = typename Storage<St>::Re;
  const StepArgs<Re>& a = A.s;
  if (A.first) {
    const Re* f0 = static_cast<const Re*>(a.src);
    const size_t N = size_t(a.g.n);
#pragma unroll
    for (int i = 0; i < Q; ++i) f[i] = ld_c(f0 + i * N + idx);
  } else {
    pull_post_bc<St, CALL>(a, static_cast<const St*>(a.src), idx, x, y, z, tag, f);
  }
}

// The FP64 form of the collision (c = C(f_k)) and of its transpose (mu <- C^T mu) as
// calls, for the cells that the fixed-point forms do not take: they pull f_k
// again, so that neither it nor their registers weigh on the others.
template <bool MRT>
__device__ __noinline__ void collide_call(const AdjArgs<double>* A, int idx, int x, int y, int z,
                                          uint32_t tag, double* c) {
  const StepArgs<double>& a = A->s;
  double f[Q], o[Q];
  recompute_f<double, true>(*A, idx, x, y, z, tag, f);
  collide_cell<double>(f, a.tau, MRT, (a.flags & SF_SMAG) != 0, a.c18cs2, a.K, o);
#pragma unroll
  for (int i = 0; i < Q; ++i) c[i] = o[i];
}
template <bool MRT>
__device__ __noinline__ void collide_T_call(const AdjArgs<double>* A, int idx, int x, int y, int z,
                                            uint32_t tag, double* mu) {
  const StepArgs<double>& a = A->s;
  double f[Q], m[Q];
  recompute_f<double, true>(*A, idx, x, y, z, tag, f);
#pragma unroll
  for (int i = 0; i < Q; ++i) m[i] = mu[i];
  CellScalars<double> cs;
  cell_scalars<double>(f, cs);
  collide_vjp_s<double>(cs, f, m, a.tau, MRT, (a.flags & SF_SMAG) != 0, a.c18cs2, a.K,
                        static_cast<double*>(nullptr));
#pragma unroll
  for (int i = 0; i < Q; ++i) mu[i] = m[i];
}

// resident 256-thread blocks per SM the register allocation is sized for
#ifndef LBM_ADJ_MINB
#define LBM_ADJ_MINB 3
#endif

// mu <- B^T mu: transposed porosity blend (soft) or bounce-back of a solid cell.
template <class Re>
__device__ __forceinline__ void blend_T(Re mu[Q], bool soft, Re p, bool hard) {
  Re m2[Q];
  if (soft) {
    if (sizeof(Re) == 8 && p == Re(0)) return;   // (FP64 operations are slow: not for a zero blend)
#pragma unroll
    for (int i = 0; i < Q; ++i) m2[i] = (Re(1) - p) * mu[i] + p * mu[opp(i)];
  } else if (hard) {
#pragma unroll
    for (int i = 0; i < Q; ++i) m2[i] = mu[opp(i)];
  } else {
    return;
  }
#pragma unroll
  for (int i = 0; i < Q; ++i) mu[i] = m2[i];
}

// nu_k = Z^T lambda_k on the faces, stored.
template <class Re>
__device__ __forceinline__ void store_nu(const AdjArgs<Re>& A, int idx, int x, int y, int z,
                                         Re mu[Q]) {
  const StepArgs<Re>& a = A.s;
  const Grid& g = a.g;
  const int fl = a.flags;
  const size_t N = size_t(g.n);
  if (!A.first) {
    if (x == g.nx - 1 && !(fl & SF_NO_OUTLET)) zou_he_outlet_T<Re>(mu, a.rho_out);
    if (x == 0 && !(fl & SF_NO_INLET)) {
      Re ux = a.u_in[0], uy = a.u_in[1], uz = a.u_in[2];
      if (fl & SF_INLET_FACE) {
        const int fi = y * g.nz + z, fn = g.ny * g.nz;
        ux = a.u_face[fi];
        uy = a.u_face[fn + fi];
        uz = a.u_face[2 * fn + fi];
      }
      zou_he_inlet_T<Re>(mu, ux, uy, uz);
    }
  }
#pragma unroll
  for (int i = 0; i < Q; ++i) A.nu_out[i * N + idx] = mu[i];
}

// The adjoint step of one cell; returns its dJ/dr contribution.  EDDY: FP64 with the
// eddy viscosity (apart, so that its registers stay out of the other form).  With
// BGK its transpose is the FP64 form of every cell, on the f_k at hand (through the
// call, which pulls f_k again, us a step of a run and its adjoint, 64x32x32 99.8 -> 89.9,
// 128x64x64 279 -> 268; at a density of 3, out of the fixed-point range, 154.4 -> 145.9).
template <class St, bool MRT, bool EDDY = false>
__device__ __forceinline__ double adjoint_cell(const AdjArgs<typename Storage<St>::Re>& A,
                                               int idx) {
  using Re = typename Storage<St>::Re;
  using S = Storage<St>;
  const StepArgs<Re>& a = A.s;
  const Grid& g = a.g;
  const int n = g.n;
  const int fl = a.flags;
  double gr = 0.0;

  if (idx < n) {
    int x, y, z;
    decode(g, idx, x, y, z);
    const uint32_t tag = a.tag ? __ldg(a.tag + idx) : 0u;
    const uint32_t ri = tag & TAG_INDEX;
    const size_t N = size_t(n);
    const Re* nu = A.nu_in;

    Re mu[Q];
    gather_mu<Re>(A, idx, x, y, z, tag, mu);

    // ---- f_k (recompute) --------------------------------------------------
    Re f[Q];
    recompute_f<St, false>(A, idx, x, y, z, tag, f);

    // FP64: the collision and its transpose in fixed point (fixed64.cuh)
    bool fast = false;
    FixCell cell;
    if constexpr (sizeof(Re) == 8) fast = a.fix.ok && fixed_load(f, cell);
    auto collide = [&](Re c[Q]) {
      if constexpr (sizeof(Re) == 8) {
        if (fast) {
          fixed_collide<MRT>(cell, (fl & SF_SMAG) != 0, a.fix,
                             [&](int i, fix v) { c[i] = from_fix<fix_out(MRT)>(v); });
        } else {
          Re o[Q];
          collide_call<MRT>(&A, idx, x, y, z, tag, o);
#pragma unroll
          for (int i = 0; i < Q; ++i) c[i] = o[i];
        }
      } else {
        collide_cell<Re>(f, a.tau, MRT, (fl & SF_SMAG) != 0, a.c18cs2, a.K, c);
      }
    };

    const bool soft = (fl & (SF_SOLID_SPHERE | SF_SOLID_FIELD)) != 0;
    const bool hard = (fl & SF_SOLID_HARD) && (tag & TAG_SOLID);
    Re p = Re(0);
    if (soft) {
      // porosity field, or the sigmoid sphere's precomputed p and dp/dr
      p = a.porosity[idx];
      const Re dpdr = (fl & SF_SOLID_SPHERE) ? a.dpdr[idx] : Re(0);
      // dJ/dr gets mu . dB/dp dp/dr; dp/dr = alpha p (1 - p) is below
      // alpha 2^-40 (2^-70 in FP64) outside a shell a few cells thick around
      // the surface, 4e-12 of its peak alpha / 4, so the collision recompute
      // is skipped there
      const Re tiny = sizeof(Re) == 8 ? Re(8.470329472543003e-22) : Re(9.094947017729282e-13);
      if (ri || ((fl & SF_SOLID_SPHERE) && dpdr > a.sph.alpha * tiny)) {
        // dJ/dp = mu . (c[opp] - c) with c = C(f_k)
        Re c[Q];
        collide(c);
        if (fl & SF_SOLID_SPHERE) {
          Re gp = Re(0);
#pragma unroll
          for (int i = 0; i < Q; ++i) gp += mu[i] * (c[opp(i)] - c[i]);
          gr += double(gp) * double(dpdr);
        }
        if (ri) link_q_grad<St>(A, c, p, true, false, ri, idx, x, y, z);
      }
    } else if (ri) {
      Re c[Q];
      collide(c);
      link_q_grad<St>(A, c, p, false, hard, ri, idx, x, y, z);
    }

    blend_T<Re>(mu, soft, p, hard);

    // ---- lambda_k = C^T mu (in place) --------------------------------------
    auto transposed = [&](Re m[Q]) {
      CellScalars<Re> cs;
      cell_scalars<Re>(f, cs);
      collide_vjp_s<Re>(cs, f, m, a.tau, MRT, (fl & SF_SMAG) != 0, a.c18cs2, a.K,
                        static_cast<Re*>(nullptr));
    };
    if constexpr (sizeof(Re) == 8 && EDDY && !MRT) {
      // BGK with the eddy viscosity: no fixed-point form, so f_k stays at hand
      if (!(fast && all_zero(mu))) transposed(mu);
    } else if constexpr (sizeof(Re) == 8) {
      fix F[Q];
      int sh;
      bool done = false;
      if (fast && fixed_load_T(mu, F, sh)) {
        if constexpr (EDDY) {
          FixEddyT t;
          done = fixed_eddy_T(cell, a.fix, sh, F, t);
          if (done) fixed_collide_T<MRT, true>(cell, a.fix, sh, F, mu, &t);
        } else {
          fixed_collide_T<MRT>(cell, a.fix, sh, F, mu);
          done = true;
        }
      } else {
        done = fast && all_zero(mu);      // beyond the reach of the objective so far
      }
      if (!done) {
        Re m2[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) m2[i] = mu[i];
        collide_T_call<MRT>(&A, idx, x, y, z, tag, m2);
#pragma unroll
        for (int i = 0; i < Q; ++i) mu[i] = m2[i];
      }
    } else {
      transposed(mu);
    }

    store_nu<Re>(A, idx, x, y, z, mu);
  }
  return gr;
}

// One block of the adjoint step: cells [block * blockDim.x, +blockDim.x);
// the block's dJ/dr goes to gr_partials[block * 8 + warp].
template <class St, bool MRT, bool EDDY = false>
__device__ __forceinline__ void adjoint_body(const AdjArgs<typename Storage<St>::Re>& A,
                                             int block) {
  double gr = adjoint_cell<St, MRT, EDDY>(A, block * blockDim.x + threadIdx.x);
  // deterministic per-warp accumulation across steps of the porosity's part of dJ/dr
  if (!(A.s.flags & SF_SOLID_SPHERE)) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) gr += __shfl_down_sync(0xffffffffu, gr, o);
  if ((threadIdx.x & 31) == 0) A.gr_partials[block * 8 + (threadIdx.x >> 5)] += gr;
}

// ---------------------------------------------------------------------------
// k_adjoint_pair: the same adjoint step for two z-adjacent cells per thread
// (FP32 arithmetic): the interior gather of nu_{k+1}, the recomputed
// f_k, the bounce-back or porosity-blend transpose and the collision transpose
// run on packed float2 values (FP32x2 pipe).  Pairs with a boundary record, on
// an x face, on a non-periodic y/z edge or (16-bit storage) straddling the
// storage-offset box are listed and take the per-cell path of k_adjoint.  ODD
// (nz odd): rows start at either parity, so every access is one cell's, and
// the pairs that straddle two rows are listed too.
// ---------------------------------------------------------------------------
template <class St> struct AdjPairArgs {
  AdjArgs<float> A;
  const St* pull[Q];      // S_{k-1} + i N - (e_x nyz + e_y nz + e_z): pull source of cell 0
  const float* push[Q];   // nu_{k+1} + j N + (e_x nyz + e_y nz + e_z): cell 0 + e_j
  float* out[Q];          // nu_k + i N
  float2 soff2[2][Q];     // storage offsets outside / inside the body box (as PairArgs)
};

constexpr int kAdjPairBlock = 128;   // 256 cells per block, as k_adjoint

// Per-direction base pointers of a pair launch (as pair_pull / pair_out of
// the forward step): from the argument block's pointer tables, or with
// LBM_PAIR_PTR_ARITH 1 from the state pointers and grid sizes.
#ifndef LBM_PAIR_PTR_ARITH
#define LBM_PAIR_PTR_ARITH 0
#endif
template <class St>
__device__ __forceinline__ long long dir_off(const AdjPairArgs<St>& P, int i) {
  const Grid& g = P.A.s.g;
  return (long long)(ex(i) * g.ny * g.nz + ey(i) * g.nz + ez(i));
}
// ARITH (a template argument): formed from the state pointers and grid sizes
// regardless of LBM_PAIR_PTR_ARITH -- the batched kernel's argument block
// sits in shared memory, where a table entry costs a shared load per use.
template <bool ARITH, class St>
__device__ __forceinline__ const St* adj_pull(const AdjPairArgs<St>& P, int i) {
  if (ARITH || LBM_PAIR_PTR_ARITH)
    return static_cast<const St*>(P.A.s.src) + (long long)i * P.A.s.g.n - dir_off(P, i);
  return P.pull[i];
}
template <bool ARITH, class St>
__device__ __forceinline__ const float* adj_push(const AdjPairArgs<St>& P, int j) {
  if (ARITH || LBM_PAIR_PTR_ARITH) return P.A.nu_in + (long long)j * P.A.s.g.n + dir_off(P, j);
  return P.push[j];
}
template <bool ARITH, class St>
__device__ __forceinline__ float* adj_out(const AdjPairArgs<St>& P, int i) {
  if (ARITH || LBM_PAIR_PTR_ARITH) return P.A.nu_out + (long long)i * P.A.s.g.n;
  return P.out[i];
}

#ifndef LBM_ADJ_PAIR_MINB
#define LBM_ADJ_PAIR_MINB 4
#endif

// FP32 values of cells idx, idx + 1; aligned to the pair unless ODD.
template <bool ODD> __device__ __forceinline__ float2 ld_pair(const float* p) {
  if constexpr (ODD) return make_float2(ld_c(p), ld_c(p + 1));
  else return ld_c(reinterpret_cast<const float2*>(p));
}

// The part of an interior pair's adjoint step after mu and f_k: the
// transpose B^T of the hard bounce-back or (SOFT) of the porosity blend, with
// dJ/dp for a sigmoid sphere; lambda_k = C^T mu on the packed values; store
// of nu_k.  Returns the pair's dJ/dr contribution
// (nonzero only for a sigmoid sphere).
template <class St, bool MRT, bool SOFT, bool ARITH = false, bool ODD = false>
__device__ __forceinline__ double adj_pair_finish(const AdjPairArgs<St>& P, int idx, int x, int y,
                                                  int z, uint32_t t0, uint32_t t1, V2 mu[Q],
                                                  V2 f[Q]) {
  const AdjArgs<float>& A = P.A;
  const StepArgs<float>& a = A.s;
  const Grid& g = a.g;
  constexpr FixedConstsF K{};
  const int fl = a.flags;
  double gr = 0.0;
  if constexpr (SOFT) {
    // S = (1 - p) c + p c_opp per lane (smooth.py:118-155).  A sigmoid
    // sphere adds dJ/dr += mu . (c_opp - c) dp/dr, skipped where dp/dr <
    // alpha 2^-40 as in adjoint_cell
    // porosity field, or the sigmoid sphere's precomputed p and dp/dr
    const V2 p(ld_pair<ODD>(a.porosity + idx));
    if (fl & SF_SOLID_SPHERE) {
      const float2 dd = ld_pair<ODD>(a.dpdr + idx);
      const float d0 = dd.x, d1 = dd.y;
      const float thr = a.sph.alpha * 9.094947017729282e-13f;
      const bool n0 = d0 > thr, n1 = d1 > thr;
      if (n0 || n1) {
        // mu . (c_opp - c) = sum_i c_i (mu_opp(i) - mu_i), summed as C emits c_i
        V2 gp(0.0f);
        auto acc = [&](int i, V2 c) { gp = gp + c * (mu[opp(i)] - mu[i]); };
        collide_cell<V2>(f, V2(a.tau), MRT, (fl & SF_SMAG) != 0, V2(a.c18cs2), K, acc);
        if (n0) gr += double(gp.x()) * double(d0);
        if (n1) gr += double(gp.y()) * double(d1);
      }
    }
    const V2 omp = V2(1.0f) - p;
    V2 m2[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) m2[i] = omp * mu[i] + p * mu[opp(i)];
#pragma unroll
    for (int i = 0; i < Q; ++i) mu[i] = m2[i];
  } else if (fl & SF_SOLID_HARD) {
    // B^T of the hard bounce-back: S_i = c_opp(i) on solid cells
    const bool s0 = (t0 & TAG_SOLID) != 0, s1 = (t1 & TAG_SOLID) != 0;
    if (s0 || s1) {
      V2 m2[Q];
#pragma unroll
      for (int i = 0; i < Q; ++i)
        m2[i] = V2(s0 ? mu[opp(i)].x() : mu[i].x(), s1 ? mu[opp(i)].y() : mu[i].y());
#pragma unroll
      for (int i = 0; i < Q; ++i) mu[i] = m2[i];
    }
  }
  // lambda_k = C^T mu
  CellScalars<V2> cs;
  cell_scalars<V2>(f, cs);
  collide_vjp_s<V2>(cs, f, mu, V2(a.tau), MRT, (fl & SF_SMAG) != 0, V2(a.c18cs2), K,
                    static_cast<V2*>(nullptr));
  // (x faces are listed pairs: no Zou-He transpose here)
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    float* o = adj_out<ARITH>(P, i) + idx;
    if constexpr (ODD) {
      o[0] = mu[i].v.x;
      o[1] = mu[i].v.y;
    } else {
      *reinterpret_cast<float2*>(o) = mu[i].v;
    }
  }
  return gr;
}


// k_adjoint_pair is one launch in two parts.  Blocks [0, nlist): the boundary pairs
// (pair_special, listed in spec_pairs) on the per-cell adjoint, dJ/dr partials
// after the per-cell slots.  Blocks [nlist, ...): the interior pairs on packed
// values.  The list blocks come first so their longer per-thread latency
// overlaps the interior blocks.

// dJ/dr partials of the listed cells, one per 32 of them (at most n / 32, since
// at most every pair is listed), after the nblocks * 8 per-cell ones.
__device__ __forceinline__ void add_list_gr(const AdjArgs<float>& A, int slot, double gr) {
  if (!(A.s.flags & SF_SOLID_SPHERE)) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) gr += __shfl_down_sync(0xffffffffu, gr, o);
  if ((threadIdx.x & 31) == 0)
    A.gr_partials[size_t((A.s.g.n + 255) / 256) * 8 + size_t(slot)] += gr;
}

// The listed cells, one thread per cell (large grids and batches, which fill the
// chip: twelve 128x64x64 domains 120.4 ms, with two threads per cell 123.5).
template <class St, bool MRT>
__device__ __forceinline__ void adjoint_pair_list_part(const AdjPairArgs<St>& P, int nlist_block) {
  const AdjArgs<float>& A = P.A;
  const int t = nlist_block * kAdjPairBlock + int(threadIdx.x);
  const int idx =
      t < 2 * A.s.spec_count ? (__ldg(A.s.spec_pairs + (t >> 1)) << 1) + (t & 1) : A.s.g.n;
  add_list_gr(A, t >> 5, adjoint_cell<St, MRT, false>(A, idx));
}

// The listed cells, two threads per cell: on small grids the launch lasts as
// long as one listed cell's chain of loads and ~2500 instructions (15 us, the
// interiors 5 to 9).  One warp pulls f_k of its 32 cells, then does the
// collision, dJ/dq and dJ/dp; another gathers mu_k, then does the transposes and the
// store; in between they exchange f_k and mu_k through shared memory
// (sh[2][Q][kListCells]).
constexpr int kListCells = kAdjPairBlock / 2;   // cells per list block
constexpr int kListShared = 2 * Q * kListCells * int(sizeof(float));

template <class St, bool MRT>
__device__ __forceinline__ void adjoint_pair_list_split(const AdjPairArgs<St>& P, int nlist_block) {
  extern __shared__ float sh_list[];
  auto sh = reinterpret_cast<float(*)[Q][kListCells]>(sh_list);
  const AdjArgs<float>& A = P.A;
  const StepArgs<float>& a = A.s;
  const Grid& g = a.g;
  const int fl = a.flags;
  const int c = threadIdx.x % kListCells;
  const bool fwd = int(threadIdx.x) >= kListCells;
  const int t = nlist_block * kListCells + c;
  int idx = 0, x = 0, y = 0, z = 0;
  uint32_t tag = 0u;
  bool in = t < 2 * a.spec_count;
  if (in) {
    idx = (__ldg(a.spec_pairs + (t >> 1)) << 1) + (t & 1);
    in = idx < g.n;                             // (the partner of an odd grid's last cell)
  }
  if (in) {
    decode(g, idx, x, y, z);
    tag = a.tag ? __ldg(a.tag + idx) : 0u;
  }
  float v[Q];                                   // f_k or mu_k
  if (in) {
    if (fwd)
      recompute_f<St, false>(A, idx, x, y, z, tag, v);
    else
      gather_mu<float>(A, idx, x, y, z, tag, v);
#pragma unroll
    for (int i = 0; i < Q; ++i) sh[fwd][i][c] = v[i];
  }
  __syncthreads();
  const bool soft = (fl & (SF_SOLID_SPHERE | SF_SOLID_FIELD)) != 0;
  const bool hard = (fl & SF_SOLID_HARD) && (tag & TAG_SOLID);
  float w[Q];
  if (!fwd) {
    if (!in) return;
#pragma unroll
    for (int i = 0; i < Q; ++i) w[i] = sh[1][i][c];
    blend_T<float>(v, soft, soft ? a.porosity[idx] : 0.0f, hard);
    CellScalars<float> cs;
    cell_scalars<float>(w, cs);
    collide_vjp_s<float>(cs, w, v, a.tau, MRT, (fl & SF_SMAG) != 0, a.c18cs2, a.K,
                         static_cast<float*>(nullptr));
    store_nu<float>(A, idx, x, y, z, v);
    return;
  }
  double gr = 0.0;
  if (in) {
    const uint32_t ri = tag & TAG_INDEX;
    const float p = soft ? a.porosity[idx] : 0.0f;
    const float dpdr = (fl & SF_SOLID_SPHERE) ? a.dpdr[idx] : 0.0f;
    // (dp/dr below alpha 2^-40 as in adjoint_cell)
    const bool shell = (fl & SF_SOLID_SPHERE) && dpdr > a.sph.alpha * 9.094947017729282e-13f;
    if (ri || shell) {
      collide_cell<float>(v, a.tau, MRT, (fl & SF_SMAG) != 0, a.c18cs2, a.K, w);
      if (fl & SF_SOLID_SPHERE) {
        float gp = 0.0f;
#pragma unroll
        for (int i = 0; i < Q; ++i) gp += sh[0][i][c] * (w[opp(i)] - w[i]);
        gr = double(gp) * double(dpdr);
      }
      if (ri) link_q_grad<St, true>(A, w, p, soft, hard, ri, idx, x, y, z);
    }
  }
  add_list_gr(A, t >> 5, gr);
}

// One interior pair of interior block `iblock`: mu_k gathered from
// nu_{k+1}, f_k pulled from S_{k-1}, then adj_pair_finish.  Returns the
// pair's dJ/dr contribution.
template <class St, bool MRT, bool SOFT, bool ARITH = false, bool ODD = false>
__device__ __forceinline__ double adjoint_pair_interior(const AdjPairArgs<St>& P, int iblock) {
  using Pr = Pair<St>;
  const AdjArgs<float>& A = P.A;
  const StepArgs<float>& a = A.s;
  const Grid& g = a.g;
  const int pidx = iblock * blockDim.x + threadIdx.x;
  if (pidx >= (g.n >> 1)) return 0.0;     // (a last cell without a partner is listed)
  const int idx = pidx << 1;
  int x, y, z;
  decode(g, idx, x, y, z);
  const uint32_t t0 = a.tag ? __ldg(a.tag + idx) : 0u;
  const uint32_t t1 = a.tag ? __ldg(a.tag + idx + 1) : 0u;
  if (pair_special(g, a.near, sizeof(St) == 2, x, y, z, t0, t1)) return 0.0;
  const int cls = sizeof(St) == 2 ? near_class(g, a.near, x, y, z, 2) : 0;
  V2 mu[Q], f[Q];
  const int nyz = g.ny * g.nz;
  // mu_k(y) = nu_{k+1}(y + e_j): y wrap shared, z wrap per lane (x faces are
  // in the list launch)
  {
    const int iyp = idx - (y == g.ny - 1 ? nyz : 0);   // e_y = +1 reads y + 1
    const int iym = idx + (y == 0 ? nyz : 0);          // e_y = -1 reads y - 1
    const int zw1 = z + 2 == g.nz ? -g.nz : 0;         // lane 1, e_z = +1 reads z + 2
    const int zw0 = z == 0 ? g.nz : 0;                 // lane 0, e_z = -1 reads z - 1
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      const int b = ey(j) == 1 ? iyp : (ey(j) == -1 ? iym : idx);
      const float* p = adj_push<ARITH>(P, j) + b;
      if (ez(j) == 0)
        mu[j] = ODD ? V2(ld_s(p), ld_s(p + 1)) : V2(ld_s(reinterpret_cast<const float2*>(p)));
      else if (ez(j) == 1) mu[j] = V2(ld_s(p), ld_s(p + 1 + zw1));
      else mu[j] = V2(ld_s(p + zw0), ld_s(p + 1));
    }
  }
  // f_k
  if (A.first) {
    const float* f0 = static_cast<const float*>(a.src);
    const size_t N = size_t(g.n);
#pragma unroll
    for (int i = 0; i < Q; ++i)
      f[i] = V2(ld_pair<ODD>(f0 + i * N + idx));
  } else {
    const int iym = idx + (y == 0 ? nyz : 0);          // e_y = +1 pulls y - 1
    const int iyp = idx - (y == g.ny - 1 ? nyz : 0);   // e_y = -1 pulls y + 1
    const int zw0 = z == 0 ? g.nz : 0;                 // lane 0, e_z = +1 pulls z - 1
    const int zw1 = z + 2 == g.nz ? -g.nz : 0;         // lane 1, e_z = -1 pulls z + 2
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int b = ey(i) == 1 ? iym : (ey(i) == -1 ? iyp : idx);
      const St* p = adj_pull<ARITH>(P, i) + b;
      const V2 so(P.soff2[cls][i]);
      if (ez(i) == 0) f[i] = ODD ? Pr::ld2s(p, p + 1, so) : Pr::ld2(p, so);
      else if (ez(i) == 1) f[i] = Pr::ld2s(p + zw0, p + 1, so);
      else f[i] = Pr::ld2s(p, p + 1 + zw1, so);
    }
  }
  return adj_pair_finish<St, MRT, SOFT, ARITH, ODD>(P, idx, x, y, z, t0, t1, mu, f);
}


// Interior block `iblock`; a sigmoid sphere's dJ/dr partials go to one of the
// per-cell slots per warp (at most n / 64 of the n / 32).
template <class St, bool MRT, bool SOFT, bool ARITH = false, bool ODD = false>
__device__ __forceinline__ void adjoint_pair_interior_part(const AdjPairArgs<St>& P, int iblock) {
  double gr = adjoint_pair_interior<St, MRT, SOFT, ARITH, ODD>(P, iblock);
  if (SOFT && (P.A.s.flags & SF_SOLID_SPHERE)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gr += __shfl_down_sync(0xffffffffu, gr, o);
    if ((threadIdx.x & 31) == 0)
      P.A.gr_partials[size_t(iblock) * (kAdjPairBlock / 32) + (threadIdx.x >> 5)] += gr;
  }
}

// nu_N = Z^T lambda_N with lambda_N = dJ/df_N from the momentum exchange:
// lambda_N[opp j](x) = dJ/dFx * e_jx on every link (x, j).
template <class Re>
__device__ __forceinline__ void adjoint_seed_cell(const StepArgs<Re>& a,
                                                  const double* __restrict__ dj_dfx,
                                                  Re* __restrict__ nu, int idx) {
  const Grid& g = a.g;
  if (idx >= g.n) return;
  const size_t N = size_t(g.n);
  Re l[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) l[i] = Re(0);
  const uint32_t tag = a.tag ? a.tag[idx] : 0u;
  const uint32_t ri = tag & TAG_INDEX;
  if (ri) {
    const uint32_t lm = a.rec[ri - 1].linkmask;
    const Re gfx = Re(*dj_dfx);
#pragma unroll
    for (int j = 1; j < Q; ++j)
      if (ex(j) != 0 && ((lm >> j) & 1u)) l[opp(j)] += Re(ex(j)) * gfx;
    const int z = idx % g.nz, t = idx / g.nz, y = t % g.ny, x = t / g.ny;
    if (x == g.nx - 1 && !(a.flags & SF_NO_OUTLET)) zou_he_outlet_T<Re>(l, a.rho_out);
    if (x == 0 && !(a.flags & SF_NO_INLET)) {
      Re ux = a.u_in[0], uy = a.u_in[1], uz = a.u_in[2];
      if (a.flags & SF_INLET_FACE) {
        const int fi = y * g.nz + z, fn = g.ny * g.nz;
        ux = a.u_face[fi];
        uy = a.u_face[fn + fi];
        uz = a.u_face[2 * fn + fi];
      }
      zou_he_inlet_T<Re>(l, ux, uy, uz);
    }
  }
#pragma unroll
  for (int i = 0; i < Q; ++i) nu[i * N + idx] = l[i];
}

// Defined in adjoint_pair.cuh, instantiated per storage type.
template <class St>
cudaError_t launch_adjoint_pair(const AdjArgs<float>& A, bool mrt, cudaStream_t st);

}  // namespace lbm
