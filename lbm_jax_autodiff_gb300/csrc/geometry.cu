// Geometry builder: solid mask, Bouzidi q (and dq/dr) per link, per-cell tags
// and the compacted boundary-cell records used by the fused kernels.
//
// Reference semantics:
//   world frame            geometry/primitives.py:26-53
//   hard sphere + q        geometry/primitives.py:56-174 (ray-sphere :145-172)
//   sigmoid sphere + q     geometry/smooth.py:158-248, examples/11:56-119
//   q from a mask          geometry/bouzidi.py:32-106
//   projected area         core/forces.py:199-234
#include <climits>

#include "sim_handle.cuh"

namespace lbm {

// A sphere's parameters in the kernels' arithmetic type, formed on the host:
// the builders run no FP64 operation in FP32 (each one costs an SM 64 times an
// FP32 one; converted per thread they took 108 of k_sphere_solid's us at
// 256x128x128).
template <class Re> struct SphereK {
  Re sx, sy, sz;          // cells per world unit
  Re c[3], r, r2, alpha, disc_floor, denom_eps;
  int sigmoid_mask;       // 0: dist^2 <= r^2 ; 1: sigmoid(alpha (r - dist)) > 0.5
  int bouzidi;            // 0: q = 0.5 ; 1: ray-sphere q(r)
};

template <class Re> static SphereK<Re> sphere_k(const Grid& g, const SphereSpec& s) {
  SphereK<Re> k;
  k.sx = Re(g.nx / 8.0);
  k.sy = Re(g.ny / 4.0);
  k.sz = Re(g.nz / 4.0);
  for (int i = 0; i < 3; ++i) k.c[i] = Re(s.c[i]);
  k.r = Re(s.r);
  k.r2 = Re(s.r * s.r);
  k.alpha = Re(s.alpha);
  k.disc_floor = Re(s.disc_floor);
  k.denom_eps = Re(s.denom_eps);
  k.sigmoid_mask = s.sigmoid_mask;
  k.bouzidi = s.bouzidi;
  return k;
}

// cell centre relative to the sphere's centre, world units
template <class Re>
__device__ __forceinline__ void offset_of(const SphereK<Re>& s, int x, int y, int z, Re& dx, Re& dy,
                                          Re& dz) {
  dx = ((Re(x) + Re(0.5)) / s.sx - Re(4)) - s.c[0];
  dy = ((Re(y) + Re(0.5)) / s.sy - Re(2)) - s.c[1];
  dz = ((Re(z) + Re(0.5)) / s.sz - Re(2)) - s.c[2];
}

// a b + c in one rounding, a b in one.  The builders say which products are
// fused instead of leaving it to the compiler, which chooses by context: a
// link's q is then the same number in every kernel that forms it.
__device__ __forceinline__ float mad(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double mad(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float prod(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double prod(double a, double b) { return __dmul_rn(a, b); }
template <class Re> __device__ __forceinline__ Re norm2(Re x, Re y, Re z) {
  return mad(z, z, mad(y, y, prod(x, x)));
}

template <class Re> __device__ __forceinline__ Re sigmoid_of(const SphereK<Re>& s, Re dx, Re dy, Re dz) {
  const Re d = sqrt(norm2(dx, dy, dz));
  return Re(1) / (Re(1) + exp(-s.alpha * (s.r - d)));
}

// Solid codes per cell: 0 fluid, 1 body, 2 ground.
template <class Re> struct SphereSolid {
  SphereK<Re> s;
  __device__ __forceinline__ int operator()(int, int x, int y, int z) const {
    Re dx, dy, dz;
    offset_of<Re>(s, x, y, z, dx, dy, dz);
    if (s.sigmoid_mask) return sigmoid_of<Re>(s, dx, dy, dz) > Re(0.5) ? 1 : 0;
    return norm2(dx, dy, dz) <= s.r2 ? 1 : 0;
  }
};
struct MaskSolid {
  const int32_t* m;
  __device__ __forceinline__ int operator()(int idx, int, int, int) const {
    const int v = m[idx];
    return v < 0 ? 0 : (v > 2 ? 2 : v);
  }
};

__device__ __forceinline__ bool link_at(const Grid& g, const uint8_t* solid, int idx, int x,
                                        int y, int z, int j) {
  const int nx = x + ex(j), ny = y + ey(j), nz = z + ez(j);
  if (nx < 0 || nx >= g.nx || ny < 0 || ny >= g.ny || nz < 0 || nz >= g.nz) return false;
  return solid[idx] == 0 && solid[(nx * g.ny + ny) * g.nz + nz] == 1;
}

// q[j] of a link of the sphere (clipped ray-sphere distance, 0.5 without a
// hit), and dq/dr.
template <class Re>
__device__ __forceinline__ Re sphere_link_q(const SphereK<Re>& s, int x, int y, int z, int j,
                                            Re& dq) {
  dq = Re(0);
  if (!s.bouzidi) return Re(0.5);
  Re ox, oy, oz;
  offset_of<Re>(s, x, y, z, ox, oy, oz);
  const Re rdx = Re(ex(j)) / s.sx, rdy = Re(ey(j)) / s.sy, rdz = Re(ez(j)) / s.sz;
  const Re a = mad(rdz, rdz, mad(rdx, rdx, prod(rdy, rdy)));
  const Re b = Re(2) * mad(oz, rdz, mad(ox, rdx, prod(oy, rdy)));
  const Re c = mad(-s.r, s.r, norm2(ox, oy, oz));
  const Re disc = mad(b, b, -prod(prod(Re(4), a), c));
  const Re dfl = fmax(disc, s.disc_floor);
  const Re sq = sqrt(dfl);
  const Re den = Re(2) * a + s.denom_eps;
  const Re tt = (-b - sq) / den;
  const bool valid = (disc >= Re(0)) && (tt > Re(0)) && (tt <= Re(1));
  if (valid) {
    // d t / d r through sqrt(max(disc, floor)) and clip(t, 0.01, 0.99), with
    // jax's half-cotangent rule at ties
    const Re wmax = disc > s.disc_floor ? Re(1) : (disc == s.disc_floor ? Re(0.5) : Re(0));
    dq = wmax * clip_weight<Re>(tt, Re(0.01), Re(0.99)) * (-(Re(4) * a * s.r) / (sq * den));
  }
  return fmin(fmax(valid ? tt : Re(0.5), Re(0.01)), Re(0.99));
}

// Sources of the wall distance q[j] (x): q < 0 where direction j meets no wall.
// LOCAL: links exist only next to a solid cell.
template <class Re> struct SphereQ {
  static constexpr bool LOCAL = true;
  SphereK<Re> s;
  __device__ __forceinline__ Re q(const Grid& g, const uint8_t* solid, int idx, int x, int y,
                                  int z, int j, Re& dq) const {
    dq = Re(0);
    return link_at(g, solid, idx, x, y, z, j) ? sphere_link_q<Re>(s, x, y, z, j, dq) : Re(-1);
  }
  __device__ __forceinline__ bool has(const Grid& g, const uint8_t* solid, int idx, int x, int y,
                                      int z, int j) const {
    return link_at(g, solid, idx, x, y, z, j);   // (a sphere's q is at least 0.01)
  }
};
template <class Re> struct DefaultQ {
  static constexpr bool LOCAL = true;
  Re v;
  __device__ __forceinline__ Re q(const Grid& g, const uint8_t* solid, int idx, int x, int y,
                                  int z, int j, Re& dq) const {
    dq = Re(0);
    return link_at(g, solid, idx, x, y, z, j) ? v : Re(-1);
  }
  __device__ __forceinline__ bool has(const Grid& g, const uint8_t* solid, int idx, int x, int y,
                                      int z, int j) const {
    return v >= Re(0) && link_at(g, solid, idx, x, y, z, j);
  }
};
template <class Re> struct DenseQ {
  static constexpr bool LOCAL = false;
  const Re* d;
  __device__ __forceinline__ Re q(const Grid& g, const uint8_t*, int idx, int, int, int, int j,
                                  Re& dq) const {
    dq = Re(0);
    return __ldg(d + size_t(j) * g.n + idx);
  }
  __device__ __forceinline__ bool has(const Grid& g, const uint8_t*, int idx, int, int, int,
                                      int j) const {
    return __ldg(d + size_t(j) * g.n + idx) >= Re(0);
  }
};

__global__ void k_geo_init(GeoInfo* info) {
  const int k = threadIdx.x;
  if (k < 6) info->bb[k] = (k & 1) ? -1 : INT_MAX;
  if (k == 6) info->nrec = info->nlinks = info->area = info->nspec = 0;
}

// Solid codes, their bounding box (any nonzero code) and the number of columns
// along x that hold a body cell (code 1): one pass over the cells.  The grids
// of this file stream n bytes, so a warp reduces its extrema and only warps
// with a solid cell touch the shared counters.
template <class Src>
__global__ void __launch_bounds__(256)
    k_mark(Grid g, Src src, uint8_t* __restrict__ solid, int* __restrict__ cols,
           GeoInfo* __restrict__ info) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  int v = 0, x = 0, y = 0, z = 0;
  if (idx < g.n) {
    decode(g, idx, x, y, z);
    v = src(idx, x, y, z);
    solid[idx] = uint8_t(v);
    if (v == 1 && atomicExch(cols + (y * g.nz + z), 1) == 0) atomicAdd(&info->area, 1);
  }
  if (__ballot_sync(0xffffffffu, v != 0) == 0u) return;
  const int c[3] = {x, y, z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int lo = __reduce_min_sync(0xffffffffu, v ? c[k] : INT_MAX);
    const int hi = __reduce_max_sync(0xffffffffu, v ? c[k] : -1);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(info->bb + 2 * k, lo);
      atomicMax(info->bb + 2 * k + 1, hi);
    }
  }
}

// v within [lo - 2, hi + 2], also across a wrap of [0, n)
__device__ __forceinline__ bool near_axis(int v, int lo, int hi, int n) {
  return (v >= lo - 2 && v <= hi + 2) || v + n <= hi + 2 || v - n >= lo - 2;
}

// Tags and records of the boundary cells, straight from the wall-distance
// source: no dense q or dq/dr array is written or read (at 256x128x128 these
// took 2 x 319 MB, a 136 us pass to write and two 411 us passes to read).  A
// cell needs a record if it owns a link, is the target of one, or is the
// second fluid cell of a q < 0.5 link; for a LOCAL source all of those lie
// within two cells of a solid one (wrapped, as the ahead cell wraps).  Records
// beyond `cap` are counted but not written.
template <class Re, class QS>
__global__ void __launch_bounds__(256)
    k_links(Grid g, QS qs, const uint8_t* __restrict__ solid, uint32_t* __restrict__ tag,
            LinkRec<Re>* __restrict__ rec, int cap, GeoInfo* __restrict__ info) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= g.n) return;
  int x, y, z;
  decode(g, idx, x, y, z);
  const uint32_t sb = solid[idx] >= 1 ? TAG_SOLID : 0u;
  if (QS::LOCAL) {
    const int* bb = info->bb;
    if (bb[1] < 0 || !near_axis(x, bb[0], bb[1], g.nx) || !near_axis(y, bb[2], bb[3], g.ny) ||
        !near_axis(z, bb[4], bb[5], g.nz)) {
      tag[idx] = sb;
      return;
    }
  }
  uint32_t lm = 0, nbw = 0, nbl = 0;
  Re qo[Q], qn[Q], dq[Q];
  qo[0] = qn[0] = Re(-1);
  dq[0] = Re(0);
#pragma unroll
  for (int j = 1; j < Q; ++j) {
    qo[j] = qs.q(g, solid, idx, x, y, z, j, dq[j]);
    if (qo[j] >= Re(0)) lm |= 1u << j;
    // pull neighbour x+e_j under the streaming rules
    int px = x + ex(j), py = y + ey(j), pz = z + ez(j);
    bool ok = px >= 0 && px < g.nx;
    if (g.periodic_yz) {
      py = wrapi(py, g.ny);
      pz = wrapi(pz, g.nz);
    } else {
      ok = ok && py >= 0 && py < g.ny && pz >= 0 && pz < g.nz;
    }
    if (ok && qs.has(g, solid, (px * g.ny + py) * g.nz + pz, px, py, pz, opp(j))) nbw |= 1u << j;
    const int wx = wrapi(x + ex(j), g.nx), wy = wrapi(y + ey(j), g.ny), wz = wrapi(z + ez(j), g.nz);
    Re unused;
    qn[j] = qs.q(g, solid, (wx * g.ny + wy) * g.nz + wz, wx, wy, wz, j, unused);
    if (qn[j] >= Re(0) && qn[j] < Re(0.5)) nbl |= 1u << j;
  }
  if ((lm | nbw | nbl) == 0) {
    tag[idx] = sb;
    return;
  }
  const int ri = atomicAdd(&info->nrec, 1);
  if (lm) atomicAdd(&info->nlinks, __popc(lm));
  if (ri >= cap) {
    tag[idx] = sb;
    return;
  }
  fill_rec<Re>(rec[ri], lm, nbw, nbl, qo, qn, dq);
  tag[idx] = sb | uint32_t(ri + 1);
}

// The list of the pairs that pair_special marks, in ascending order: counts
// per block of kPairScan pairs, their prefix sums, then each block writes its
// pairs at its offset.
constexpr int kPairScan = 2048;

__device__ __forceinline__ bool pair_flag(const Grid& g, const uint32_t* tag, const int near[6],
                                          int use_class, int p) {
  const int idx = p << 1;
  if (idx >= g.n) return false;
  int x, y, z;
  decode(g, idx, x, y, z);
  const uint32_t t1 = idx + 1 < g.n ? __ldg(tag + idx + 1) : 0u;
  return pair_special(g, near, use_class != 0, x, y, z, __ldg(tag + idx), t1);
}

__global__ void __launch_bounds__(256)
    k_pair_count(Grid g, const uint32_t* __restrict__ tag, int use_class,
                 const GeoInfo* __restrict__ info, int* __restrict__ blk) {
  int near[6];
  near_box(g, info->bb, near);
  int c = 0;
  for (int it = 0; it < kPairScan; it += 256)
    c += __syncthreads_count(
        pair_flag(g, tag, near, use_class, blockIdx.x * kPairScan + it + threadIdx.x));
  if (threadIdx.x == 0) blk[blockIdx.x] = c;
}

__global__ void __launch_bounds__(1024) k_pair_scan(int* __restrict__ blk, int nb, GeoInfo* info) {
  __shared__ int warp_sum[32];
  __shared__ int base;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int b0 = 0; b0 < nb; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    const int c = b < nb ? blk[b] : 0;
    int s = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    if (lane == 31) warp_sum[wid] = s;
    __syncthreads();
    if (wid == 0) {
      int w = warp_sum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
      }
      warp_sum[lane] = w;
    }
    __syncthreads();
    const int before = base + (wid ? warp_sum[wid - 1] : 0) + s - c;
    if (b < nb) blk[b] = before;
    __syncthreads();
    if (threadIdx.x == 0) base += warp_sum[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) info->nspec = base;
}

__global__ void __launch_bounds__(256)
    k_pair_write(Grid g, const uint32_t* __restrict__ tag, int use_class,
                 const GeoInfo* __restrict__ info, const int* __restrict__ blk,
                 int* __restrict__ list, int cap) {
  __shared__ int warp_cnt[8];
  int near[6];
  near_box(g, info->bb, near);
  int base = blk[blockIdx.x];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int it = 0; it < kPairScan; it += 256) {
    const int p = blockIdx.x * kPairScan + it + threadIdx.x;
    const bool f = pair_flag(g, tag, near, use_class, p);
    const unsigned m = __ballot_sync(0xffffffffu, f);
    if (lane == 0) warp_cnt[wid] = __popc(m);
    __syncthreads();
    int before = base, all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      if (w < wid) before += warp_cnt[w];
      all += warp_cnt[w];
    }
    const int at = before + __popc(m & ((1u << lane) - 1u));
    if (f && at < cap) list[at] = p;
    base += all;
    __syncthreads();
  }
}

// Dense q[j][cell] (-1 where no link) and dq/dr (may be null), for the per-op
// geometry functions.
template <class Re, class QS>
__global__ void k_dense_q(Grid g, QS qs, const uint8_t* __restrict__ solid, Re* __restrict__ q,
                          Re* __restrict__ dqdr) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= g.n) return;
  int x, y, z;
  decode(g, idx, x, y, z);
  const size_t N = size_t(g.n);
  q[idx] = Re(-1);
  if (dqdr) dqdr[idx] = Re(0);
#pragma unroll
  for (int j = 1; j < Q; ++j) {
    Re dq;
    q[j * N + idx] = qs.q(g, solid, idx, x, y, z, j, dq);
    if (dqdr) dqdr[j * N + idx] = dq;
  }
}

template <class Src>
__global__ void k_solid(Grid g, Src src, uint8_t* __restrict__ solid) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= g.n) return;
  int x, y, z;
  decode(g, idx, x, y, z);
  solid[idx] = uint8_t(src(idx, x, y, z));
}

// axis-aligned box, world corners (primitives.py:177-255): solid = inside
template <class Re> struct BoxSolid {
  Re sx, sy, sz, lo[3], hi[3];
  __device__ __forceinline__ int operator()(int, int x, int y, int z) const {
    const Re wx = (Re(x) + Re(0.5)) / sx - Re(4);
    const Re wy = (Re(y) + Re(0.5)) / sy - Re(2);
    const Re wz = (Re(z) + Re(0.5)) / sz - Re(2);
    return wx >= lo[0] && wx <= hi[0] && wy >= lo[1] && wy <= hi[1] && wz >= lo[2] && wz <= hi[2];
  }
};

// dense outputs of the builders for the per-op geometry functions
template <class Re>
__global__ void k_export_fields(Grid g, SphereK<Re> s, int with_porosity,
                                const uint8_t* __restrict__ solid, int32_t* __restrict__ solid_out,
                                Re* __restrict__ porosity) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= g.n) return;
  if (solid_out) solid_out[idx] = solid[idx];
  if (porosity && with_porosity) {
    int x, y, z;
    decode(g, idx, x, y, z);
    Re dx, dy, dz;
    offset_of<Re>(s, x, y, z, dx, dy, dz);
    porosity[idx] = sigmoid_of<Re>(s, dx, dy, dz);
  } else if (porosity) {
    porosity[idx] = Re(solid[idx] >= 1 ? 1 : 0);
  }
}

static inline int nblk(int n) { return (n + 255) / 256; }

template <class Re>
cudaError_t launch_sphere_fields(const Grid& g, const SphereSpec& s, uint8_t* solid, Re* q,
                                 Re* dqdr, cudaStream_t st) {
  const SphereK<Re> k = sphere_k<Re>(g, s);
  k_solid<<<nblk(g.n), 256, 0, st>>>(g, SphereSolid<Re>{k}, solid);
  k_dense_q<Re><<<nblk(g.n), 256, 0, st>>>(g, SphereQ<Re>{k}, solid, q, dqdr);
  return cudaGetLastError();
}

template <class Re>
cudaError_t launch_q_from_solid(const Grid& g, const uint8_t* solid, double dq, Re* q,
                                cudaStream_t st) {
  k_dense_q<Re><<<nblk(g.n), 256, 0, st>>>(g, DefaultQ<Re>{Re(dq)}, solid, q, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_solid_from_i32(const Grid& g, const int32_t* m, uint8_t* s, cudaStream_t st) {
  k_solid<<<nblk(g.n), 256, 0, st>>>(g, MaskSolid{m}, s);
  return cudaGetLastError();
}

template <class Re>
cudaError_t launch_box_fields(const Grid& g, const double lo[3], const double hi[3],
                              uint8_t* solid, Re* q, cudaStream_t st) {
  BoxSolid<Re> b;
  b.sx = Re(g.nx / 8.0);
  b.sy = Re(g.ny / 4.0);
  b.sz = Re(g.nz / 4.0);
  for (int k = 0; k < 3; ++k) {
    b.lo[k] = Re(lo[k]);
    b.hi[k] = Re(hi[k]);
  }
  k_solid<<<nblk(g.n), 256, 0, st>>>(g, b, solid);
  return launch_q_from_solid<Re>(g, solid, 0.5, q, st);
}

template <class Re>
cudaError_t launch_export_fields(const Grid& g, const SphereSpec& s, int with_porosity,
                                 const uint8_t* solid, int32_t* solid_out, Re* porosity,
                                 cudaStream_t st) {
  k_export_fields<Re><<<nblk(g.n), 256, 0, st>>>(g, sphere_k<Re>(g, s), with_porosity, solid,
                                                 solid_out, porosity);
  return cudaGetLastError();
}

int pair_scan_blocks(const Grid& g) { return ((g.n + 1) / 2 + kPairScan - 1) / kPairScan; }

// The geometry of a handle into its scratch, tag, record and pair-list buffers
// (GeoBuffers): one pass marks the solid cells, one writes tags and records,
// and three small ones build the pair list; the counts come back in `info`.
template <class Re>
cudaError_t launch_geometry(const Grid& g, const GeoSource& src, const GeoBuffers& b,
                            cudaStream_t st) {
  k_geo_init<<<1, 32, 0, st>>>(b.info);
  cudaError_t e = cudaMemsetAsync(b.cols, 0, size_t(g.ny) * g.nz * sizeof(int), st);
  if (e != cudaSuccess) return e;
  LinkRec<Re>* rec = static_cast<LinkRec<Re>*>(b.rec);
  const int nb = nblk(g.n);
  if (src.sphere) {
    const SphereK<Re> k = sphere_k<Re>(g, *src.sphere);
    k_mark<<<nb, 256, 0, st>>>(g, SphereSolid<Re>{k}, b.solid, b.cols, b.info);
    k_links<Re><<<nb, 256, 0, st>>>(g, SphereQ<Re>{k}, b.solid, b.tag, rec, b.rec_cap, b.info);
  } else {
    k_mark<<<nb, 256, 0, st>>>(g, MaskSolid{src.mask}, b.solid, b.cols, b.info);
    if (src.q)
      k_links<Re><<<nb, 256, 0, st>>>(g, DenseQ<Re>{static_cast<const Re*>(src.q)}, b.solid, b.tag,
                                      rec, b.rec_cap, b.info);
    else
      k_links<Re><<<nb, 256, 0, st>>>(g, DefaultQ<Re>{Re(src.default_q)}, b.solid, b.tag, rec,
                                      b.rec_cap, b.info);
  }
  if (b.pair_blk) {
    const int pb = pair_scan_blocks(g);
    k_pair_count<<<pb, 256, 0, st>>>(g, b.tag, b.use_class, b.info, b.pair_blk);
    k_pair_scan<<<1, 1024, 0, st>>>(b.pair_blk, pb, b.info);
    if (b.spec_cap > 0)
      k_pair_write<<<pb, 256, 0, st>>>(g, b.tag, b.use_class, b.info, b.pair_blk, b.spec_pairs,
                                       b.spec_cap);
  }
  return cudaGetLastError();
}

// Per-cell porosity and dp/dr of a sigmoid sphere (sphere_porosity), once per
// geometry: the step and adjoint kernels read them instead of evaluating the
// sigmoid (three divisions, a square root and an exponential) every step.
template <class Re>
__global__ void k_sphere_porosity(Grid g, SphereP<Re> sp, Re* __restrict__ p,
                                  Re* __restrict__ dpdr) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= g.n) return;
  int x, y, z;
  decode(g, idx, x, y, z);
  Re d;
  p[idx] = sphere_porosity<Re>(sp, x, y, z, &d);
  dpdr[idx] = d;
}

template <class Re>
cudaError_t launch_sphere_porosity(const Grid& g, const SphereP<Re>& sp, Re* p, Re* dpdr,
                                   cudaStream_t st) {
  k_sphere_porosity<Re><<<(g.n + 255) / 256, 256, 0, st>>>(g, sp, p, dpdr);
  return cudaGetLastError();
}

template cudaError_t launch_sphere_porosity<float>(const Grid&, const SphereP<float>&, float*,
                                                   float*, cudaStream_t);
template cudaError_t launch_sphere_porosity<double>(const Grid&, const SphereP<double>&, double*,
                                                    double*, cudaStream_t);
template cudaError_t launch_sphere_fields<float>(const Grid&, const SphereSpec&, uint8_t*, float*,
                                                 float*, cudaStream_t);
template cudaError_t launch_sphere_fields<double>(const Grid&, const SphereSpec&, uint8_t*,
                                                  double*, double*, cudaStream_t);
template cudaError_t launch_q_from_solid<float>(const Grid&, const uint8_t*, double, float*,
                                                cudaStream_t);
template cudaError_t launch_q_from_solid<double>(const Grid&, const uint8_t*, double, double*,
                                                 cudaStream_t);
template cudaError_t launch_box_fields<float>(const Grid&, const double*, const double*,
                                              uint8_t*, float*, cudaStream_t);
template cudaError_t launch_box_fields<double>(const Grid&, const double*, const double*,
                                               uint8_t*, double*, cudaStream_t);
template cudaError_t launch_export_fields<float>(const Grid&, const SphereSpec&, int,
                                                 const uint8_t*, int32_t*, float*, cudaStream_t);
template cudaError_t launch_export_fields<double>(const Grid&, const SphereSpec&, int,
                                                  const uint8_t*, int32_t*, double*, cudaStream_t);
template cudaError_t launch_geometry<float>(const Grid&, const GeoSource&, const GeoBuffers&,
                                            cudaStream_t);
template cudaError_t launch_geometry<double>(const Grid&, const GeoSource&, const GeoBuffers&,
                                             cudaStream_t);

}  // namespace lbm
