// Batched adjoint (device code in adjoint.cuh): one launch covers every
// instance of a batch.
#include "adjoint.cuh"

namespace lbm {

#ifndef LBM_ADJ_BATCH_MINB
#define LBM_ADJ_BATCH_MINB 2
#endif

template <class St, bool MRT>
__global__ void __launch_bounds__(256, LBM_ADJ_BATCH_MINB)
    k_adjoint_batch(const AdjArgs<float>* __restrict__ args, const BatchInst* __restrict__ inst,
                    const int2* __restrict__ map, int sprev_slot, int sk_slot, int nu_in_slot,
                    int nu_out_slot, int first, int last) {
  __shared__ AdjArgs<float> A;
  chain_begin();
  const int2 m = map[blockIdx.x];
  copy_to_shared(&A, args + m.x);
  __syncthreads();
  const BatchInst& b = inst[m.x];
  if (threadIdx.x == 0) {
    A.s.src = batch_slot(b, sprev_slot);
    A.S_k = batch_slot(b, sk_slot);
    A.nu_in = static_cast<const float*>(batch_slot(b, nu_in_slot));
    A.nu_out = static_cast<float*>(batch_slot(b, nu_out_slot));
    A.first = first;
    A.last = last;
    A.dj_dfx = b.out + 4;
    A.gr_partials = b.gr_part;
    A.gq = b.gq;
  }
  __syncthreads();
  const int end = m.y + kBatchChunk < b.nblk ? m.y + kBatchChunk : b.nblk;
  for (int sb = m.y; sb < end; ++sb) adjoint_body<St, MRT>(A, sb);
}

// Batched k_adjoint_pair (FP32 storage, nz even): map[b] = (instance, sub-block),
// a sub-block y >= 0 being interior block y and y < 0 list block ~y; entries
// with instance -1 pad the map to the grid the launch (and a captured graph)
// was sized for.  Two launches a step: the list blocks of all instances and the
// interiors without a porosity blend, then (SOFT) the interiors with one.
#ifndef LBM_ADJ_PAIR_BATCH_MINB
#define LBM_ADJ_PAIR_BATCH_MINB 4
#endif
// LBM_BATCH_PTR_ARITH 1: the batched pair adjoint forms its per-direction
// pointers from the instance's state pointers (adj_pull<true>), 0: it
// builds the tables in shared memory.
#ifndef LBM_BATCH_PTR_ARITH
#define LBM_BATCH_PTR_ARITH 1
#endif

template <bool MRT, bool SOFT>
__global__ void __launch_bounds__(kAdjPairBlock, LBM_ADJ_PAIR_BATCH_MINB)
    k_adjoint_pair_batch(const AdjArgs<float>* __restrict__ args,
                         const BatchInst* __restrict__ inst, const int2* __restrict__ map,
                         int sprev_slot, int sk_slot, int nu_in_slot, int nu_out_slot, int first,
                         int last) {
  __shared__ AdjPairArgs<float> P;
  chain_begin();
  const int2 m = map[blockIdx.x];
  if (m.x < 0) return;
  copy_to_shared(&P.A, args + m.x);
  __syncthreads();
  const BatchInst& b = inst[m.x];
  const float* src = static_cast<const float*>(batch_slot(b, sprev_slot));
  const float* nu_in = static_cast<const float*>(batch_slot(b, nu_in_slot));
  float* nu_out = static_cast<float*>(batch_slot(b, nu_out_slot));
  if (threadIdx.x == 0) {
    AdjArgs<float>& A = P.A;
    A.s.src = src;
    A.S_k = batch_slot(b, sk_slot);
    A.nu_in = nu_in;
    A.nu_out = nu_out;
    A.first = first;
    A.last = last;
    A.dj_dfx = b.out + 4;
    A.gr_partials = b.gr_part;
    A.gq = b.gq;
  } else if (!LBM_BATCH_PTR_ARITH && threadIdx.x <= Q) {
    // the per-direction tables, one direction per thread
    const int i = threadIdx.x - 1;
    const Grid& g = P.A.s.g;
    const long long N = g.n, nyz = (long long)g.ny * g.nz;
    const long long off = ex(i) * nyz + ey(i) * g.nz + ez(i);
    P.pull[i] = src + i * N - off;
    P.push[i] = nu_in + i * N + off;
    P.out[i] = nu_out + i * N;
    P.soff2[0][i] = make_float2(0.0f, 0.0f);
    P.soff2[1][i] = make_float2(0.0f, 0.0f);
  }
  __syncthreads();
  if (!SOFT && m.y < 0)
    adjoint_pair_list_part<float, MRT>(P, ~m.y);
  else
    adjoint_pair_interior_part<float, MRT, SOFT, LBM_BATCH_PTR_ARITH != 0>(P, m.y);
}

__global__ void __launch_bounds__(256)
    k_adjoint_seed_batch(const StepArgs<float>* __restrict__ args,
                         const BatchInst* __restrict__ inst, const int2* __restrict__ map,
                         int nu_slot) {
  __shared__ StepArgs<float> sa;
  const int2 m = map[blockIdx.x];
  copy_to_shared(&sa, args + m.x);
  __syncthreads();
  const BatchInst& b = inst[m.x];
  float* nu = static_cast<float*>(batch_slot(b, nu_slot));
  const int end = m.y + kBatchChunk < b.nblk ? m.y + kBatchChunk : b.nblk;
  for (int sb = m.y; sb < end; ++sb)
    adjoint_seed_cell<float>(sa, b.out + 4, nu, sb * blockDim.x + threadIdx.x);
}

// Per instance (one block each): clear the dJ/dr partials and the per-link dJ/dq.
__global__ void __launch_bounds__(256) k_zero_grad_batch(const BatchInst* __restrict__ inst) {
  const BatchInst& b = inst[blockIdx.x];
  for (int i = threadIdx.x; i < b.ngr; i += blockDim.x) b.gr_part[i] = 0.0;
  for (int i = threadIdx.x; i < b.ngq; i += blockDim.x) b.gq[i] = 0.0;
}

// Per instance (one block each): dCd/dr = fixed-order sum of the partials and of
// dJ/dq dq/dr over the links; where the domain has a pair list, its cells only
// (every cell with links is listed).
__global__ void __launch_bounds__(256)
    k_reduce_gr_batch(const StepArgs<float>* __restrict__ args,
                      const BatchInst* __restrict__ inst) {
  __shared__ double sh[256];
  const BatchInst& b = inst[blockIdx.x];
  const StepArgs<float>& a = args[blockIdx.x];
  double v = 0.0;
  for (int i = threadIdx.x; i < b.ngr; i += blockDim.x) v += b.gr_part[i];
  const int cells = a.spec_pairs ? 2 * a.spec_count : a.g.n;
  for (int t = threadIdx.x; t < cells; t += blockDim.x) {
    const int idx = a.spec_pairs ? (a.spec_pairs[t >> 1] << 1) + (t & 1) : t;
    if (idx < a.g.n) v += link_gr<float>(a.tag[idx], a.rec, b.gq);
  }
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) b.out[5] = sh[0];
}

// One Adam step on each instance's radius (optax.adam, examples/11:182-194):
// loss = Cd (minimize_cd_loss) or (Cd - target)^2 (target_cd_loss,
// optim/losses.py:34-99); m, v bias-corrected; r clipped to [r_min, r_max]
// afterwards.  opt[i] = (r, m, v, t).
__global__ void k_adam_batch(const BatchInst* __restrict__ inst, int count, AdamP p,
                             double* __restrict__ opt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const BatchInst& b = inst[i];
  const double cd = b.out[3], dcd = b.out[5];
  const double loss = p.target ? (cd - p.target_cd) * (cd - p.target_cd) : cd;
  const double g = p.target ? 2.0 * (cd - p.target_cd) * dcd : dcd;
  b.out[6] = loss;
  b.out[7] = g;
  double* o = opt + 4 * i;
  const double t = o[3] + 1.0;
  const double m = p.b1 * o[1] + (1.0 - p.b1) * g;
  const double v = p.b2 * o[2] + (1.0 - p.b2) * g * g;
  const double mh = m / (1.0 - pow(p.b1, t));
  const double vh = v / (1.0 - pow(p.b2, t));
  double r = o[0] - p.lr * mh / (sqrt(vh) + p.eps);
  r = fmin(fmax(r, p.r_min), p.r_max);
  o[0] = r;
  o[1] = m;
  o[2] = v;
  o[3] = t;
}

template <class St>
cudaError_t launch_adjoint_batch(const AdjArgs<float>* args, const BatchInst* inst,
                                 const int2* map, int nblocks, int block, bool mrt,
                                 int sprev_slot, int sk_slot, int nu_in_slot, int nu_out_slot,
                                 int first, int last, cudaStream_t st) {
  return launch_chained(mrt ? k_adjoint_batch<St, true> : k_adjoint_batch<St, false>, nblocks, block,
                        st, args, inst, map, sprev_slot, sk_slot, nu_in_slot, nu_out_slot, first,
                        last);
}

cudaError_t launch_adjoint_pair_batch(const AdjArgs<float>* args, const BatchInst* inst,
                                      const int2* map, int nblocks, bool mrt, bool soft,
                                      int sprev_slot, int sk_slot, int nu_in_slot,
                                      int nu_out_slot, int first, int last, cudaStream_t st) {
  auto* k = mrt ? (soft ? k_adjoint_pair_batch<true, true> : k_adjoint_pair_batch<true, false>)
                : (soft ? k_adjoint_pair_batch<false, true> : k_adjoint_pair_batch<false, false>);
  return launch_chained(k, nblocks, kAdjPairBlock, st, args, inst, map, sprev_slot, sk_slot,
                        nu_in_slot, nu_out_slot, first, last);
}

cudaError_t launch_adjoint_seed_batch(const StepArgs<float>* args, const BatchInst* inst,
                                      const int2* map, int nblocks, int block, int nu_slot,
                                      cudaStream_t st) {
  k_adjoint_seed_batch<<<nblocks, block, 0, st>>>(args, inst, map, nu_slot);
  return cudaGetLastError();
}

cudaError_t launch_zero_grad_batch(const BatchInst* inst, int count, cudaStream_t st) {
  k_zero_grad_batch<<<count, 256, 0, st>>>(inst);
  return cudaGetLastError();
}

cudaError_t launch_reduce_gr_batch(const StepArgs<float>* args, const BatchInst* inst, int count,
                                   cudaStream_t st) {
  k_reduce_gr_batch<<<count, 256, 0, st>>>(args, inst);
  return cudaGetLastError();
}

cudaError_t launch_adam_batch(const BatchInst* inst, int count, const AdamP& p, double* opt,
                              cudaStream_t st) {
  k_adam_batch<<<(count + 127) / 128, 128, 0, st>>>(inst, count, p, opt);
  return cudaGetLastError();
}

template cudaError_t launch_adjoint_batch<float>(const AdjArgs<float>*, const BatchInst*,
                                                 const int2*, int, int, bool, int, int, int, int,
                                                 int, int, cudaStream_t);

}  // namespace lbm
