// k_adjoint_pair and its launch (device code in adjoint.cuh); one translation
// unit per storage type, so that they compile side by side.
#pragma once

#include <type_traits>

#include "adjoint.cuh"

namespace lbm {

// Grids up to this many cells take two threads per listed cell: there the list
// is the launch's longest chain.  One against two threads per cell, us a step
// (FP32, Smagorinsky): 64x32x32 19.2 / 10.4, 96x48x48 21.7 / 13.6, 128x64x64
// 42.8 / 24.5, 192x96x96 73.9 / 71.7.  Beyond, the blocks' idle half costs as much
// (256x128x128 177.8 / 176.6 alone, but 60 steps with 16-bit storage 19.0 / 19.6 ms).
#ifndef LBM_ADJ_SPLIT_MAX
#define LBM_ADJ_SPLIT_MAX (1 << 21)
#endif

template <class St, bool MRT, bool SOFT, bool ODD>
__global__ void __launch_bounds__(kAdjPairBlock, LBM_ADJ_PAIR_MINB)
    k_adjoint_pair(const AdjPairArgs<St> P, int nlist, int split) {
  chain_begin();
  if (int(blockIdx.x) < nlist)
    if (split)
      adjoint_pair_list_split<St, MRT>(P, blockIdx.x);
    else
      adjoint_pair_list_part<St, MRT>(P, blockIdx.x);
  else
    adjoint_pair_interior_part<St, MRT, SOFT, false, ODD>(P, blockIdx.x - nlist);
}

template <class St>
cudaError_t launch_adjoint_pair(const AdjArgs<float>& A, bool mrt, cudaStream_t st) {
  AdjPairArgs<St> P;
  P.A = A;
  const Grid& g = A.s.g;
  const long long N = g.n, nyz = (long long)g.ny * g.nz;
  for (int i = 0; i < Q; ++i) {
    const long long off = ex(i) * nyz + ey(i) * g.nz + ez(i);
    P.pull[i] = static_cast<const St*>(A.s.src) + i * N - off;
    P.push[i] = A.nu_in + i * N + off;
    P.out[i] = A.nu_out + i * N;
    P.soff2[0][i] = make_float2(A.s.soff[i], A.s.soff[i]);
    P.soff2[1][i] = make_float2(A.s.soff_near[i], A.s.soff_near[i]);
  }
  const int nb = (g.n / 2 + kAdjPairBlock - 1) / kAdjPairBlock;
  const int split = g.n <= LBM_ADJ_SPLIT_MAX;
  const int per = split ? kListCells : kAdjPairBlock;
  const int nlist = (2 * A.s.spec_count + per - 1) / per;
  const bool soft = (A.s.flags & (SF_SOLID_SPHERE | SF_SOLID_FIELD)) != 0;
  auto pick = [&](auto odd) {
    constexpr bool O = decltype(odd)::value;
    return mrt ? (soft ? k_adjoint_pair<St, true, true, O> : k_adjoint_pair<St, true, false, O>)
               : (soft ? k_adjoint_pair<St, false, true, O> : k_adjoint_pair<St, false, false, O>);
  };
  auto* k = g.nz % 2 ? pick(std::true_type{}) : pick(std::false_type{});
  return launch_chained_shared(k, nlist + nb, kAdjPairBlock, split ? kListShared : 0, st, P, nlist,
                               split);
}

}  // namespace lbm
