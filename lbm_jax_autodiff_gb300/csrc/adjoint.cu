// Adjoint time step, one cell per thread (device code in adjoint.cuh), the
// seeds of the adjoint state and the reductions of a gradient evaluation.
#include <type_traits>

#include <algorithm>

#include "adjoint.cuh"

namespace lbm {

// MINB: resident blocks per SM that the registers are sized for.
template <class St, bool MRT, bool EDDY, int MINB>
__global__ void __launch_bounds__(256, MINB)
    k_adjoint(const __grid_constant__ AdjArgs<typename Storage<St>::Re> A) {
  chain_begin();
  adjoint_body<St, MRT, EDDY>(A, blockIdx.x);
}

template <class Re>
__global__ void k_adjoint_seed(StepArgs<Re> a, const double* __restrict__ dj_dfx,
                               Re* __restrict__ nu) {
  adjoint_seed_cell<Re>(a, dj_dfx, nu, blockIdx.x * blockDim.x + threadIdx.x);
}

// nu_N = Z^T g for a given cotangent g on the final post-boundary f_N (the
// reference's state after N steps, state.py:129-171): the Zou-He
// transposes on the inlet / outlet faces, g itself elsewhere.
template <class Re>
__global__ void k_adjoint_seed_dense(StepArgs<Re> a, const Re* __restrict__ gin,
                                     Re* __restrict__ nu) {
  const Grid& g = a.g;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= g.n) return;
  const size_t N = size_t(g.n);
  Re l[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) l[i] = gin[i * N + idx];
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
#pragma unroll
  for (int i = 0; i < Q; ++i) nu[i * N + idx] = l[i];
}

// dJ/dFx = sign(Fx) / (0.5 rho U^2 A + 1e-10) from the finalized force record
// out = (Fx, Fy, Fz, Cd).
__global__ void k_dj_dfx(const double* __restrict__ fcd, double dyn_area, double* __restrict__ g) {
  const double fx = fcd[0];
  const double s = fx > 0.0 ? 1.0 : (fx < 0.0 ? -1.0 : 0.0);
  *g = s / (dyn_area + 1e-10);
}

// Sum of n partials in a fixed order: one value per block, then one launch
// more over those (a single block took 469 us for the 262,144 slots of a
// 256x128x128 gradient).
constexpr int kReduceBlocks = 256;
__global__ void __launch_bounds__(256)
    k_reduce_sum(const double* __restrict__ part, int n, double* __restrict__ out) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    s += part[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = sh[0];
}

// dJ/dr of the links, dJ/dq dq/dr summed over each block's cells in a fixed order,
// added to the block's first slot of the dJ/dr partials.
template <class Re>
__global__ void __launch_bounds__(256)
    k_link_gr(int n, const uint32_t* __restrict__ tag, const LinkRec<Re>* __restrict__ rec,
              const double* __restrict__ gq, double* __restrict__ gr_partials) {
  __shared__ double sh[8];
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  double v = idx < n ? link_gr<Re>(tag[idx], rec, gq) : 0.0;
  if (!__syncthreads_or(v != 0.0)) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = sh[0];
    for (int k = 1; k < 8; ++k) s += sh[k];
    gr_partials[size_t(blockIdx.x) * 8] += s;
  }
}

// per-link dJ/dq -> dense [19][n] (zero where there is no link)
template <class Re>
__global__ void k_scatter_gq(Grid g, const uint32_t* __restrict__ tag,
                             const LinkRec<Re>* __restrict__ rec, const double* __restrict__ gq,
                             Re* __restrict__ out) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= g.n) return;
  const size_t N = size_t(g.n);
  const uint32_t ri = tag[idx] & TAG_INDEX;
  if (!ri) {
    // (apart: an FP64 conversion per direction in every cell took 98 of 145 us)
#pragma unroll
    for (int j = 0; j < Q; ++j) out[j * N + idx] = Re(0);
    return;
  }
  const uint32_t lm = rec[ri - 1].linkmask;
#pragma unroll
  for (int j = 0; j < Q; ++j)
    out[j * N + idx] = ((lm >> j) & 1u) ? Re(gq[size_t(ri - 1) * Q + j]) : Re(0);
}

static inline int nblk(int n) { return (n + 255) / 256; }

template <class St>
cudaError_t launch_adjoint(const AdjArgs<typename Storage<St>::Re>& A, bool mrt,
                           cudaStream_t st) {
  // FP32 arithmetic (FP32 / FP16 / BF16 storage): k_adjoint_pair, one launch of
  // list blocks + interior blocks (166 us per 256x128x128 step against 280 / 265
  // us for k_adjoint); SOFT for a porosity blend.  Short odd rows are mostly
  // listed pairs (one in nz straddles two rows): those stay with k_adjoint.
  if constexpr (sizeof(typename Storage<St>::Re) == 4) {
    if (A.s.spec_pairs && (A.s.g.nz % 2 == 0 || A.s.g.nz >= 5))
      return launch_adjoint_pair<St>(A, mrt, st);
  }
  constexpr bool f64 = sizeof(St) == 8;
  constexpr int many = f64 ? 2 : LBM_ADJ_MINB, few = f64 ? 1 : many;
  const int nb = nblk(A.s.g.n);
  const bool soft = (A.s.flags & (SF_SOLID_SPHERE | SF_SOLID_FIELD)) != 0;
  const bool small =
      f64 && one_block_per_sm(nb, sm_count(), soft, (A.s.flags & SF_SMAG) != 0, mrt);
  auto pick = [&](auto mrt_c, auto eddy_c) {
    constexpr bool M = decltype(mrt_c)::value, E = decltype(eddy_c)::value;
    return small ? k_adjoint<St, M, E, few> : k_adjoint<St, M, E, many>;
  };
  using Yes = std::true_type;
  using No = std::false_type;
  auto* k = mrt ? pick(Yes{}, No{}) : pick(No{}, No{});
  if constexpr (f64)
    if (A.s.flags & SF_SMAG) k = mrt ? pick(Yes{}, Yes{}) : pick(No{}, Yes{});
  return launch_chained(k, nb, 256, st, A);
}

template <class Re>
cudaError_t launch_adjoint_seed(const StepArgs<Re>& a, const double* dj, Re* nu, cudaStream_t st) {
  k_adjoint_seed<Re><<<nblk(a.g.n), 256, 0, st>>>(a, dj, nu);
  return cudaGetLastError();
}

template <class Re>
cudaError_t launch_adjoint_seed_dense(const StepArgs<Re>& a, const Re* g, Re* nu,
                                      cudaStream_t st) {
  k_adjoint_seed_dense<Re><<<nblk(a.g.n), 256, 0, st>>>(a, g, nu);
  return cudaGetLastError();
}

cudaError_t launch_dj_dfx(const double* fcd, double dyn_area, double* g, cudaStream_t st) {
  k_dj_dfx<<<1, 1, 0, st>>>(fcd, dyn_area, g);
  return cudaGetLastError();
}

cudaError_t launch_reduce_sum(const double* part, int n, double* out, double* scratch,
                              cudaStream_t st) {
  const int nb = std::min(kReduceBlocks, (n + 255) / 256);
  k_reduce_sum<<<nb, 256, 0, st>>>(part, n, scratch);
  k_reduce_sum<<<1, 256, 0, st>>>(scratch, nb, out);
  return cudaGetLastError();
}

template <class Re>
cudaError_t launch_link_gr(const Grid& g, const uint32_t* tag, const LinkRec<Re>* rec,
                           const double* gq, double* gr_partials, cudaStream_t st) {
  k_link_gr<Re><<<nblk(g.n), 256, 0, st>>>(g.n, tag, rec, gq, gr_partials);
  return cudaGetLastError();
}

template <class Re>
cudaError_t launch_scatter_gq(const Grid& g, const uint32_t* tag, const LinkRec<Re>* rec,
                              const double* gq, Re* out, cudaStream_t st) {
  k_scatter_gq<Re><<<nblk(g.n), 256, 0, st>>>(g, tag, rec, gq, out);
  return cudaGetLastError();
}

template cudaError_t launch_adjoint<float>(const AdjArgs<float>&, bool, cudaStream_t);
template cudaError_t launch_adjoint<double>(const AdjArgs<double>&, bool, cudaStream_t);
template cudaError_t launch_adjoint<__half>(const AdjArgs<float>&, bool, cudaStream_t);
template cudaError_t launch_adjoint<__nv_bfloat16>(const AdjArgs<float>&, bool, cudaStream_t);
template cudaError_t launch_adjoint_seed<float>(const StepArgs<float>&, const double*, float*,
                                                cudaStream_t);
template cudaError_t launch_adjoint_seed<double>(const StepArgs<double>&, const double*, double*,
                                                 cudaStream_t);
template cudaError_t launch_adjoint_seed_dense<float>(const StepArgs<float>&, const float*,
                                                      float*, cudaStream_t);
template cudaError_t launch_adjoint_seed_dense<double>(const StepArgs<double>&, const double*,
                                                       double*, cudaStream_t);
template cudaError_t launch_link_gr<float>(const Grid&, const uint32_t*, const LinkRec<float>*,
                                           const double*, double*, cudaStream_t);
template cudaError_t launch_link_gr<double>(const Grid&, const uint32_t*, const LinkRec<double>*,
                                            const double*, double*, cudaStream_t);
template cudaError_t launch_scatter_gq<float>(const Grid&, const uint32_t*, const LinkRec<float>*,
                                              const double*, float*, cudaStream_t);
template cudaError_t launch_scatter_gq<double>(const Grid&, const uint32_t*, const LinkRec<double>*,
                                               const double*, double*, cudaStream_t);

}  // namespace lbm
