// Shared device-side structures of the fused solver: grid, boundary-cell
// records, kernel argument blocks and the pull / Bouzidi / Zou-He helpers.
//
// Data layout in HBM (identical to jax_lbm's arrays, state.py:41-44):
//   populations  [19][nx][ny][nz]  z fastest (structure of arrays)
//   tag          [nx][ny][nz] uint32: bit 31 = hard-solid cell, bits 0..30 =
//                1 + index of the cell's LinkRec (0 = plain cell)
//   LinkRec[]    one record per "special" cell: a cell that owns a Bouzidi
//                link, is the target of one, or is the second fluid cell of a
//                q < 0.5 link.  Only these cells read anything beyond the pull.
#pragma once

#include <atomic>
#include <utility>

#include "fixed64.cuh"
#include "lbm_core.cuh"

namespace lbm {

constexpr uint32_t TAG_SOLID = 0x80000000u;
constexpr uint32_t TAG_INDEX = 0x7FFFFFFFu;

// A boundary cell's record: what the pull and its transpose need per direction,
// in the compute type.  The per-direction tables are padded to 20 entries and
// 16-byte aligned, so a cell's table is a few wide loads issued together.
// Weights are formed once per geometry (fill_rec), not per step.
template <class Re> struct alignas(16) LinkRec {
  uint32_t linkmask;  // bit j: q[j](x) >= 0  (direction j from x hits a wall)
  uint32_t nb_wall;   // bit j: pull neighbour x+e_j has q[opp j] >= 0
  uint32_t nb_low;    // bit j: 0 <= q[j](wrap(x+e_j)) < 0.5
  uint32_t low;       // bit j: 0 <= q[j](x) < 0.5
  Re w[Q + 1];        // Bouzidi weight of link j: 1 / (2 min(q, 1)), low: 2 max(q, 0)
  Re nbw[Q + 1];      // 1 - 2 q[j](wrap(x+e_j)) for nb_low bits, else 0
  Re gc[Q + 1];       // dT/dq of link j is gc (S_j(x) - other), see link_q_grad
  Re dqdr[Q + 1];     // d q[j](x) / d r
};

// Record of a cell from its wall distances q[j], the ahead neighbours'
// distances qnb[j] (read where nb_low is set) and dq/dr.
template <class Re>
__device__ __forceinline__ void fill_rec(LinkRec<Re>& R, uint32_t lm, uint32_t nbw, uint32_t nbl,
                                         const Re q[Q], const Re qnb[Q], const Re* dqdr) {
  uint32_t low = 0;
#pragma unroll
  for (int j = 0; j <= Q; ++j) {
    Re w = Re(0), gc = Re(0);
    if (j < Q && ((lm >> j) & 1u)) {
      const Re qv = q[j];
      if (qv >= Re(0.5)) {
        // a = 1 / (2 clip(q, 0.5, 1)); clip passes half the cotangent at a tie
        const Re qc = fmin(qv, Re(1));
        w = Re(1) / (Re(2) * qc);
        gc = -(clip_weight<Re>(qv, Re(0.5), Re(1)) / (Re(2) * qc * qc));
      } else {
        // b = 2 clip(q, 0, 0.5)
        w = Re(2) * fmax(qv, Re(0));
        gc = Re(2) * clip_weight<Re>(qv, Re(0), Re(0.5));
        low |= 1u << j;
      }
    }
    R.w[j] = w;
    R.gc[j] = gc;
    R.nbw[j] = j < Q && ((nbl >> j) & 1u) ? Re(1) - Re(2) * qnb[j] : Re(0);
    R.dqdr[j] = j < Q ? dqdr[j] : Re(0);
  }
  R.linkmask = lm;
  R.nb_wall = nbw;
  R.nb_low = nbl;
  R.low = low;
}

// One representative i < opp(i) of each pair of opposite directions, in
// ascending order (the order in which the two directions' terms are added).
__host__ __device__ constexpr int pair_dir(int k) {
  constexpr int t[9] = {1, 3, 5, 7, 8, 11, 12, 15, 16};
  return t[k];
}

// Unsigned division by a runtime constant with a multiply-high
// (Granlund-Montgomery): q = (umulhi(n, mul) + n) >> shift, exact for n < 2^31.
struct FastDiv {
  uint32_t d, mul, shift;
  __host__ __device__ __forceinline__ uint32_t div(uint32_t n) const {
#ifdef __CUDA_ARCH__
    return (__umulhi(n, mul) + n) >> shift;
#else
    return uint32_t(((uint64_t(n) * mul >> 32) + n) >> shift);
#endif
  }
};
inline FastDiv make_fastdiv(uint32_t d) {
  FastDiv f;
  f.d = d;
  uint32_t l = 0;
  while ((1ull << l) < d) ++l;
  f.shift = l;
  f.mul = uint32_t(((1ull << 32) * ((1ull << l) - d)) / d + 1);
  return f;
}

// Chained launches.  A time step is one launch, and a run is a chain of them in
// one stream.  launch_chained lets the next launch of the chain start while the
// last blocks of this one still run (programmatic dependent launch); chain_begin,
// first thing in such a kernel, lets its own successor start in turn and then
// waits until the predecessor's writes are all visible.  What a launch of the chain
// writes is read with ld_s / ld_c or plain loads only; tags, records and pair lists
// may be read with __ldg, since a geometry is finished, with a wait on the host,
// before the first launch that reads it.  What overlaps is the
// launch latency and the block start-up: 100 steps of a 64x21x8 channel 623 ->
// 464 us, of a 64x32x32 sphere 690 -> 643 us, of 256x128x128 11.70 -> 11.47 ms
// (16-bit storage 92.1 -> 90.2 us a step), 60 FP64 steps of 96x48x48 1.70 ->
// 1.60 ms, the 96x48x48 gradient 5.93 -> 5.43 ms.
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
inline cudaError_t launch_chained_shared(void (*kernel)(P...), int grid, int block, int shared,
                                         cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(unsigned(grid));
  c.blockDim = dim3(unsigned(block));
  c.dynamicSmemBytes = size_t(shared);
  c.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), int grid, int block, cudaStream_t st,
                                  A&&... args) {
  return launch_chained_shared(kernel, grid, block, 0, st, std::forward<A>(args)...);
}

// SMs of the current device, which the size rules of the kernels' forms count in
// (asked once per device).
inline int sm_count() {
  static std::atomic<int> known[64] = {};
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1)
    n = 152;
  if (dev >= 0 && dev < 64) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

// Whether a step of n cells runs k_step_roomy (see launch_step): up to one wave of
// k_step's 64-register threads.
inline bool roomy_cells(long long n, int sms) { return n <= 1024LL * sms; }

// Whether an FP64 adjoint step of nb blocks runs with one block per SM, which keeps
// every value in registers, rather than two, which hide more latency but spill.  The
// longer a launch, the more the latency counts; a porosity blend has more loads
// to hide, BGK with the eddy viscosity spills most (860 bytes).  us a step of a run and
// its adjoint, one / two blocks per SM, at 256, 500, 864, 1099, 1372 and 2048 blocks:
//   hard MRT        45 / 50    56 / 58    83 / 85   100 / 97   120 / 109  163 / 142
//   with the eddy   63 / 74    85 / 97   119 / 129  141 / 147  167 / 165  226 / 209
//   soft MRT        56 / 62    86 / 78   136 / 114  167 / 136  202 / 163  285 / 222
//   hard BGK eddy   90 / 115  126 / 149  166 / 187  190 / 212  219 / 239  296 / 304
//   soft BGK eddy  108 / 138  156 / 175  228 / 228  275 / 263  331 / 304  464 / 412
inline bool one_block_per_sm(int nb, int sms, bool soft, bool eddy, bool mrt) {
  const int rounds = eddy && !mrt ? (soft ? 6 : 14) : soft ? 2 : eddy ? 8 : 6;
  return nb <= rounds * sms;
}

struct Grid {
  int nx, ny, nz;
  int n;              // nx*ny*nz
  int periodic_yz;
  FastDiv dz, dy;     // divide by nz, by ny
};

inline Grid make_grid(int nx, int ny, int nz, int periodic) {
  Grid g;
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.n = nx * ny * nz;
  g.periodic_yz = periodic ? 1 : 0;
  g.dz = make_fastdiv(uint32_t(nz));
  g.dy = make_fastdiv(uint32_t(ny));
  return g;
}

__device__ __forceinline__ void decode(const Grid& g, int idx, int& x, int& y, int& z) {
  const uint32_t t = g.dz.div(uint32_t(idx));
  z = idx - int(t) * g.nz;
  const uint32_t xx = g.dy.div(t);
  y = int(t) - int(xx) * g.ny;
  x = int(xx);
}

// flags of StepArgs::flags
enum : int {
  SF_SMAG = 1 << 0,
  SF_SOLID_HARD = 1 << 1,
  SF_SOLID_SPHERE = 1 << 2,   // analytic sigmoid porosity
  SF_SOLID_FIELD = 1 << 3,    // porosity array
  SF_GUARD_PRE = 1 << 4,
  SF_GUARD_POST = 1 << 5,
  SF_FORCE = 1 << 6,
  SF_COLLIDE_ONLY = 1 << 7,   // input is the reference-layout f (no pull)
  SF_STREAM_ONLY = 1 << 8,    // output is the reference-layout post-BC f
  SF_INLET_FACE = 1 << 9,     // per-(y,z) inlet velocity
  SF_NO_INLET = 1 << 10,
  SF_NO_OUTLET = 1 << 11,
  SF_EMIT_F = 1 << 12,        // also write the post-BC f (after the post guard) to f_emit
};

template <class Re> struct SphereP {
  Re c[3];
  Re r;
  Re alpha;
  Re sx, sy, sz;   // cells per world unit: nx/8, ny/4, nz/4
};

// FP64 storage: the collision's fixed-point constants.
template <class Re> struct FixArgs {};
template <> struct FixArgs<double> { FixConsts fix; };

template <class Re> struct StepArgs : FixArgs<Re> {
  const void* src;        // populations S_{k-1} (storage type) or f_0 (Re)
  void* dst;              // populations S_k (storage type) or post-BC f (Re)
  const uint32_t* tag;
  const LinkRec<Re>* rec;
  Grid g;
  Consts<Re> K;
  Re tau;
  Re c18cs2;              // 18 Cs^2
  int flags;
  Re u_in[3];
  const Re* u_face;       // [3][ny][nz]
  Re rho_out;
  SphereP<Re> sph;
  const Re* porosity;     // [n] porosity field (also filled for a sigmoid sphere)
  const Re* dpdr;         // [n] dp/dr of a sigmoid sphere, else null
  Re guard_reset[Q];
  // 16-bit storage holds f_i minus an offset: the rest equilibrium w_i inside
  // the box `near` around the body (where u ~ 0), the free-stream equilibrium
  // f_eq(1, (u_in, 0, 0)) elsewhere -- so every cell stores a small deviation
  Re soff[Q];             // outside the box
  Re soff_near[Q];        // inside the box
  int near[6];            // [x0, x1) x [y0, y1) x [z0, z1); empty when x0 >= x1
  const int* spec_pairs;  // pairs the pair kernels run on their per-cell path
  int spec_count;
  double* force_partials; // [gridDim.x][3]
  unsigned long long* guard_count;
  void* f_emit;           // SF_EMIT_F: the post-BC f of the pull (Re), [19][n]
};

__device__ __forceinline__ int wrapi(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

// ---- storage offsets of 16-bit populations ----------------------------------
__device__ __forceinline__ bool in_near(const int b[6], int x, int y, int z) {
  return x >= b[0] && x < b[1] && y >= b[2] && y < b[3] && z >= b[4] && z < b[5];
}

// In-box masks of a cell's neighbourhood, one bit per offset along each
// axis: bit k of mx is "x + k - 1 inside the box" (x never wraps), of my
// likewise with y wrapped, and of mz for z - 1 .. z + zc (wrapped), zc = 1
// (one cell) or 2 (a z-pair).  The source x - e_i of direction i is inside
// iff bit 1 - e_x of mx, 1 - e_y of my and 1 - e_z of mz are all set.
struct NearMask {
  unsigned mx, my, mz;
  __device__ __forceinline__ NearMask(const Grid& g, const int b[6], int x, int y, int z, int zc) {
    auto in = [](int v, int lo, int hi) { return unsigned(v >= lo && v < hi); };
    mx = in(x - 1, b[0], b[1]) | (in(x, b[0], b[1]) << 1) | (in(x + 1, b[0], b[1]) << 2);
    my = in(wrapi(y - 1, g.ny), b[2], b[3]) | (in(y, b[2], b[3]) << 1) |
         (in(wrapi(y + 1, g.ny), b[2], b[3]) << 2);
    mz = in(wrapi(z - 1, g.nz), b[4], b[5]) | (in(z, b[4], b[5]) << 1) |
         (in(wrapi(z + 1, g.nz), b[4], b[5]) << 2);
    if (zc == 2) mz |= in(wrapi(z + 2, g.nz), b[4], b[5]) << 3;
  }
  // 0: the whole neighbourhood outside, 1: inside, 2: mixed
  __device__ __forceinline__ int cls(int zc) const {
    const unsigned full_z = zc == 2 ? 15u : 7u;
    if (mx == 0u || my == 0u || mz == 0u) return 0;
    if (mx == 7u && my == 7u && mz == full_z) return 1;
    return 2;
  }
  // class of the pull source x - e_i of the cell at z (lane 0)
  __device__ __forceinline__ bool src_in(int i) const {
    return ((mx >> (1 - ex(i))) & (my >> (1 - ey(i))) & (mz >> (1 - ez(i))) & 1u) != 0u;
  }
  // class of the neighbour x + e_i of the cell at z (lane 0)
  __device__ __forceinline__ bool nbr_in(int i) const {
    return ((mx >> (1 + ex(i))) & (my >> (1 + ey(i))) & (mz >> (1 + ez(i))) & 1u) != 0u;
  }
  __device__ __forceinline__ bool self_in() const { return ((mx & my & mz) >> 1) & 1u; }
};

__device__ __forceinline__ int near_class(const Grid& g, const int b[6], int x, int y, int z,
                                          int zc) {
  // x never wraps: most cells are decided by x alone
  if (x + 1 < b[0] || x - 1 >= b[1]) return 0;
  return NearMask(g, b, x, y, z, zc).cls(zc);
}

// A pair of cells (2p, 2p + 1) that the packed pair kernels run on their per-cell
// path: two cells of different rows (odd nz), a boundary record on either cell, an
// x face (fallback pull and Zou-He), a non-periodic y/z edge, or (when the storage
// offsets matter, use_class) a neighbourhood that straddles the body box.  The pair
// kernels' interior blocks skip these pairs; their list blocks compute them from
// the list built with this same predicate.  (Listing the x faces rather than
// testing for them in the interior measured 94 us against 100 us per 16-bit step
// at 256x128x128.)
__device__ __forceinline__ bool pair_special(const Grid& g, const int near[6], bool use_class,
                                             int x, int y, int z, uint32_t t0, uint32_t t1) {
  const bool xface = x == 0 || x == g.nx - 1;
  bool sp = ((t0 | t1) & TAG_INDEX) || xface || z + 1 == g.nz;
  if (!g.periodic_yz) sp = sp || y == 0 || y == g.ny - 1 || z == 0 || z + 2 == g.nz;
  if (use_class && !sp) sp = near_class(g, near, x, y, z, 2) == 2;
  return sp;
}

// Cell x + e_i wrapped in all three axes (jnp.roll semantics, streaming.py:166-172).
__device__ __forceinline__ int ahead_wrap(const Grid& g, int x, int y, int z, int dx, int dy,
                                          int dz) {
  return (wrapi(x + dx, g.nx) * g.ny + wrapi(y + dy, g.ny)) * g.nz + wrapi(z + dz, g.nz);
}

// Zou-He velocity inlet at x = 0 (boundary.py:35-124).
template <class Re>
__device__ __forceinline__ void zou_he_inlet(Re f[Q], Re ux, Re uy, Re uz) {
  const Re k0 = f[0] + f[3] + f[4] + f[5] + f[6] + f[15] + f[16] + f[17] + f[18];
  const Re kn = f[2] + f[8] + f[10] + f[12] + f[14];
  const Re rho = (k0 + Re(2) * kn) / (Re(1) - ux);
  const Re c3 = Re(1.0 / 3.0) * rho, c6 = Re(1.0 / 6.0) * rho;
  f[1] = f[2] + c3 * ux;
  f[7] = f[10] + c6 * (ux + uy);
  f[9] = f[8] + c6 * (ux - uy);
  f[11] = f[14] + c6 * (ux + uz);
  f[13] = f[12] + c6 * (ux - uz);
}

// Zou-He pressure outlet at x = nx-1 with u_y = u_z = 0 (boundary.py:127-200).
template <class Re>
__device__ __forceinline__ void zou_he_outlet(Re f[Q], Re rho_out) {
  const Re k0 = f[0] + f[3] + f[4] + f[5] + f[6] + f[15] + f[16] + f[17] + f[18];
  const Re kp = f[1] + f[7] + f[9] + f[11] + f[13];
  const Re ux = Re(-1) + (k0 + Re(2) * kp) / rho_out;
  const Re c3 = Re(1.0 / 3.0) * rho_out * ux, c6 = Re(1.0 / 6.0) * rho_out * ux;
  f[2] = f[1] - c3;
  f[10] = f[7] - c6;
  f[8] = f[9] - c6;
  f[14] = f[11] - c6;
  f[12] = f[13] - c6;
}

// Sigmoid porosity of the analytic sphere at cell (x,y,z), smooth.py:34-115:
// p = sigmoid(alpha (r - |x_world - c|)).
template <class Re>
__device__ __forceinline__ Re sphere_porosity(const SphereP<Re>& s, int x, int y, int z,
                                              Re* dpdr) {
  const Re wx = (Re(x) + Re(0.5)) / s.sx - Re(4);
  const Re wy = (Re(y) + Re(0.5)) / s.sy - Re(2);
  const Re wz = (Re(z) + Re(0.5)) / s.sz - Re(2);
  const Re dx = wx - s.c[0], dy = wy - s.c[1], dz = wz - s.c[2];
  const Re d = sqrt(dx * dx + dy * dy + dz * dz);
  const Re p = Re(1) / (Re(1) + exp(-s.alpha * (s.r - d)));
  if (dpdr) *dpdr = s.alpha * p * (Re(1) - p);
  return p;
}

// Guard test of state.py:161-166 / examples/10:164-167 on (rho, j):
// rho < 0.3, rho > 2, |u| > 0.4 (tested as |j|^2 > 0.16 rho^2, rho being in
// [0.3, 2] by then), or rho NaN (the first comparison fails for NaN).
template <class Re>
__device__ __forceinline__ bool unstable_rj(Re rho, Re jx, Re jy, Re jz) {
  const Re j2 = jx * jx + jy * jy + jz * jz;
  return !(rho >= Re(0.3) && rho <= Re(2.0)) || (j2 > Re(0.16) * rho * rho);
}

// Pull offsets of one cell, hoisted out of the 19-direction loop: source
// coordinate s = x - e along each axis, with validity (x never periodic;
// y/z periodic or clamped, streaming.py:109-142).
struct PullIdx {
  int xo[3], yo[3], zo[3];   // index 0: e = -1, 1: e = 0, 2: e = +1
  bool xv[3], yv[3], zv[3];
  __device__ __forceinline__ PullIdx(const Grid& g, int x, int y, int z) {
    const int nyz = g.ny * g.nz;
    xo[0] = (x + 1) * nyz; xo[1] = x * nyz; xo[2] = (x - 1) * nyz;
    xv[0] = x < g.nx - 1; xv[1] = true; xv[2] = x > 0;
    int yp = y + 1, ym = y - 1, zp = z + 1, zm = z - 1;
    if (g.periodic_yz) {
      yp = yp >= g.ny ? yp - g.ny : yp;
      ym = ym < 0 ? ym + g.ny : ym;
      zp = zp >= g.nz ? zp - g.nz : zp;
      zm = zm < 0 ? zm + g.nz : zm;
      yv[0] = yv[2] = zv[0] = zv[2] = true;
    } else {
      yv[0] = y < g.ny - 1; yv[2] = y > 0;
      zv[0] = z < g.nz - 1; zv[2] = z > 0;
    }
    yv[1] = zv[1] = true;
    yo[0] = yp * g.nz; yo[1] = y * g.nz; yo[2] = ym * g.nz;
    zo[0] = zp; zo[1] = z; zo[2] = zm;
  }
  __device__ __forceinline__ int src(int i, int idx) const {
    const int a = 1 + ex(i), b = 1 + ey(i), c = 1 + ez(i);
    const bool ok = xv[a] && yv[b] && zv[c];
    return ok ? xo[a] + yo[b] + zo[c] : idx;
  }
  // forward pull of direction i reads (x - e_i) (no fallback)
  __device__ __forceinline__ bool valid(int i) const {
    return xv[1 + ex(i)] && yv[1 + ey(i)] && zv[1 + ez(i)];
  }
  __device__ __forceinline__ int raw(int i) const {
    return xo[1 + ex(i)] + yo[1 + ey(i)] + zo[1 + ez(i)];
  }
};

// Neighbour offsets of a cell away from the domain faces: cell x + d (each
// component d in {-1,0,1}) is idx + ox[d+1] + oy[d+1] + oz[d+1], with the
// periodic y/z wrap folded in.  `face` marks cells where some neighbour is
// out of range (x = 0 / nx-1 always; y/z edges when not periodic); those use
// PullIdx and its fallback rule.
struct NbrOff {
  int ox[3], oy[3], oz[3];
  bool face;
  __device__ __forceinline__ NbrOff(const Grid& g, int x, int y, int z) {
    const int nyz = g.ny * g.nz;
    ox[0] = -nyz; ox[1] = 0; ox[2] = nyz;
    oy[0] = -g.nz + (y == 0 ? nyz : 0);
    oy[1] = 0;
    oy[2] = g.nz - (y == g.ny - 1 ? nyz : 0);
    oz[0] = -1 + (z == 0 ? g.nz : 0);
    oz[1] = 0;
    oz[2] = 1 - (z == g.nz - 1 ? g.nz : 0);
    face = (x == 0) || (x == g.nx - 1);
    if (!g.periodic_yz) face = face || y == 0 || y == g.ny - 1 || z == 0 || z == g.nz - 1;
  }
  // source of the pull of direction i: x - e_i
  __device__ __forceinline__ int pull(int i, int idx) const {
    return idx + ox[1 - ex(i)] + oy[1 - ey(i)] + oz[1 - ez(i)];
  }
  // x + e_j
  __device__ __forceinline__ int push(int j, int idx) const {
    return idx + ox[1 + ex(j)] + oy[1 + ey(j)] + oz[1 + ez(j)];
  }
};

// Bouzidi bounce-back on the wall links of a boundary cell
// (streaming.py:148-183).  In: f, the plain pull.  own(i) loads S_i(x);
// the second fluid cell's S_io(x + e_i) of a q < 0.5 link is the value the
// plain pull of direction io fetched, except next to a domain edge, where
// ahead(i, v) corrects it.
//
// What bounds it is the latency of dependent loads: the boundary cells are few
// and a launch on a small grid lasts as long as they do.  So the record's
// weights and the cell's own populations are loaded for all directions of a
// group at once, without a branch per link (one exposed latency per group of
// three pairs where a branch per link had one or two for each).  Measured,
// with the same form of the transposed terms (gather_mu, link_q_grad): 100
// steps of a 64x21x8 channel 827 -> 623 us, of a 64x32x32 sphere 894 -> 689
// us; 200 steps and their adjoint at 96x48x48 9.64 -> 6.40 ms.
template <class Re, class Own, class Ahead>
__device__ __forceinline__ void bouzidi(const LinkRec<Re>& r, bool edge, Re f[Q], Own own,
                                        Ahead ahead) {
  const uint32_t lm = r.linkmask, low = r.low;
#pragma unroll
  for (int k0 = 0; k0 < 9; k0 += 3) {
    Re s[3][2], w[3][2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int i = pair_dir(k0 + k), io = opp(i);
      s[k][0] = own(i);
      s[k][1] = own(io);
      w[k][0] = __ldg(&r.w[i]);
      w[k][1] = __ldg(&r.w[io]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int i = pair_dir(k0 + k), io = opp(i);
      Re nb_i = f[io], nb_o = f[i];          // S_io(x + e_i), S_i(x + e_io)
      if (edge) {
        if ((low >> io) & 1u) ahead(i, nb_i);
        if ((low >> i) & 1u) ahead(io, nb_o);
      }
      const Re oi = ((low >> io) & 1u) ? nb_i : s[k][0];
      const Re oo = ((low >> i) & 1u) ? nb_o : s[k][1];
      if ((lm >> io) & 1u) f[i] = w[k][1] * s[k][1] + (Re(1) - w[k][1]) * oi;
      if ((lm >> i) & 1u) f[io] = w[k][0] * s[k][0] + (Re(1) - w[k][0]) * oo;
    }
  }
}

// bouzidi for FP32 / FP64 storage as a call: the boundary cells' registers then
// stay out of the allocation of the cells that have no record (inlined, the
// 64-register k_step<float> spilled and took 123 against 112 us per step at
// 256x128x128).
template <class Re>
__device__ __noinline__ void bouzidi_call(const LinkRec<Re>* r, const Re* src, Grid g,
                                          int idx, int x, int y, int z, bool edge, Re* fio) {
  const size_t N = size_t(g.n);
  Re f[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) f[i] = fio[i];
  bouzidi<Re>(
      *r, edge, f, [&](int i) { return Storage<Re>::ld(src + i * N + idx, Re(0)); },
      [&](int i, Re& v) {
        const int io = opp(i);
        if (!PullIdx(g, x, y, z).valid(io))
          v = Storage<Re>::ld(src + io * N + ahead_wrap(g, x, y, z, ex(i), ey(i), ez(i)), Re(0));
      });
#pragma unroll
  for (int i = 0; i < Q; ++i) fio[i] = f[i];
}

// The same for 16-bit storage, whose storage offsets come from the launch's arguments.
template <class St>
__device__ __noinline__ void bouzidi_call16(const StepArgs<float>* a, const St* src, uint32_t ri,
                                            int idx, int x, int y, int z, bool edge, float* fio) {
  const Grid& g = a->g;
  const size_t N = size_t(g.n);
  const NearMask M(g, a->near, x, y, z, 1);
  const float* own_off = M.self_in() ? a->soff_near : a->soff;
  float f[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) f[i] = fio[i];
  bouzidi<float>(
      a->rec[ri - 1], edge, f,
      [&](int i) { return Storage<St>::ld(src + i * N + idx, own_off[i]); },
      [&](int i, float& v) {
        const int io = opp(i);
        if (!PullIdx(g, x, y, z).valid(io))
          v = Storage<St>::ld(src + io * N + ahead_wrap(g, x, y, z, ex(i), ey(i), ez(i)),
                              M.nbr_in(i) ? a->soff_near[io] : a->soff[io]);
      });
#pragma unroll
  for (int i = 0; i < Q; ++i) fio[i] = f[i];
}

// Post-stream, post-boundary populations f_k of cell (x,y,z) from the stored
// post-collision populations S_{k-1}: pull (streaming.py:109-142), Bouzidi on
// the cell's wall links (streaming.py:148-183), Zou-He inlet/outlet
// (boundary.py:35-200).
// `tab` (optional): per-direction pull bases src + i N - (e_x nyz + e_y nz +
// e_z) from the launch's argument block, so an interior pull address is one
// table entry plus the cell index and its y / z wrap corrections.
// CALL: boundary cells through bouzidi_call / bouzidi_call16 (the forward kernels
// that launch_step picks; `a` is then the kernel's argument block itself, since
// the call takes its address; the adjoint's list blocks are faster with it
// inlined, 6.40 against 6.82 ms for the 96x48x48 gradient above).
template <class St, bool CALL = false>
__device__ __forceinline__ void pull_post_bc(const StepArgs<typename Storage<St>::Re>& a,
                                             const St* src, int idx, int x, int y,
                                             int z, uint32_t tag,
                                             typename Storage<St>::Re f[Q],
                                             const St* const* tab = nullptr) {
  using Re = typename Storage<St>::Re;
  using S = Storage<St>;
  const Grid& g = a.g;
  const size_t N = size_t(g.n);
  const NbrOff O(g, x, y, z);
  // offset classes matter only for 16-bit storage (FP32/FP64 store f itself)
  constexpr bool offs = sizeof(St) == 2;
  const NearMask M(g, a.near, x, y, z, 1);
  const int cls = offs ? M.cls(1) : 0;
  if (!O.face && cls != 2 && tab) {
    const int nyz = g.ny * g.nz;
    const int wym = y == 0 ? nyz : 0;             // e_y = +1 pulls y - 1
    const int wyp = y == g.ny - 1 ? -nyz : 0;     // e_y = -1 pulls y + 1
    const int wzm = z == 0 ? g.nz : 0;            // e_z = +1 pulls z - 1
    const int wzp = z == g.nz - 1 ? -g.nz : 0;    // e_z = -1 pulls z + 1
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int b = idx + (ey(i) == 1 ? wym : (ey(i) == -1 ? wyp : 0)) +
                    (ez(i) == 1 ? wzm : (ez(i) == -1 ? wzp : 0));
      f[i] = S::ld(tab[i] + b, cls ? a.soff_near[i] : a.soff[i]);
    }
  } else if (!O.face && cls != 2) {
#pragma unroll
    for (int i = 0; i < Q; ++i)
      f[i] = S::ld(src + i * N + O.pull(i, idx), cls ? a.soff_near[i] : a.soff[i]);
  } else {
    const PullIdx P(g, x, y, z);
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      // offset class of the source cell (the cell itself on the fallback)
      const bool in = P.valid(i) ? M.src_in(i) : M.self_in();
      f[i] = S::ld(src + i * N + P.src(i, idx), in ? a.soff_near[i] : a.soff[i]);
    }
  }
  const uint32_t ri = tag & TAG_INDEX;
  if (ri) {
    if constexpr (CALL) {
      Re t[Q];
#pragma unroll
      for (int i = 0; i < Q; ++i) t[i] = f[i];
      if constexpr (offs)
        bouzidi_call16<St>(&a, src, ri, idx, x, y, z, O.face, t);
      else
        bouzidi_call<Re>(a.rec + (ri - 1), src, g, idx, x, y, z, O.face, t);
#pragma unroll
      for (int i = 0; i < Q; ++i) f[i] = t[i];
    } else {
      const bool own_near = M.self_in();
      bouzidi<Re>(
          a.rec[ri - 1], O.face, f,
          [&](int i) { return S::ld(src + i * N + idx, own_near ? a.soff_near[i] : a.soff[i]); },
          [&](int i, Re& v) {
            // the ahead cell's S_io wraps in every axis; the pull of io read it
            // unless its source was out of range
            const int io = opp(i);
            if (!PullIdx(g, x, y, z).valid(io))
              v = S::ld(src + io * N + ahead_wrap(g, x, y, z, ex(i), ey(i), ez(i)),
                        M.nbr_in(i) ? a.soff_near[io] : a.soff[io]);
          });
    }
  }
  if (x == 0 && !(a.flags & SF_NO_INLET)) {
    Re ux = a.u_in[0], uy = a.u_in[1], uz = a.u_in[2];
    if (a.flags & SF_INLET_FACE) {
      const int fi = y * g.nz + z, fn = g.ny * g.nz;
      ux = a.u_face[fi];
      uy = a.u_face[fn + fi];
      uz = a.u_face[2 * fn + fi];
    }
    zou_he_inlet<Re>(f, ux, uy, uz);
  }
  if (x == g.nx - 1 && !(a.flags & SF_NO_OUTLET)) zou_he_outlet<Re>(f, a.rho_out);
}

// The FP64-storage cell in fixed point: loads f and says whether the step may
// use it (in range, and not a cell that an enabled guard resets); `p` is the
// porosity of a blend.
__device__ __forceinline__ bool fixed_cell(const StepArgs<double>& a, const double f[Q], double p,
                                           FixCell& c) {
  if (!a.fix.ok || !(p >= 0.0 && p <= 1.0) || !fixed_load(f, c)) return false;
  return !((a.flags & (SF_GUARD_PRE | SF_GUARD_POST)) && fixed_fast(c));
}

// Post-collision, post-solid populations S of a fixed-point cell (hard
// bounce-back of a solid cell, or the blend (1 - p) c + p c_opp).
template <bool MRT>
__device__ __forceinline__ void fixed_step(const StepArgs<double>& a, const FixCell& c, bool hard,
                                           double p, double s[Q]) {
  constexpr int B = fix_out(MRT);
  fix v[Q];
  fixed_collide<MRT>(c, (a.flags & SF_SMAG) != 0, a.fix, [&](int i, fix x) { v[i] = x; });
  if (hard) {
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int i = pair_dir(k), io = opp(i);
      const fix t = v[i];
      v[i] = v[io];
      v[io] = t;
    }
  } else if (p != 0.0) {
    const fix pf = to_fix(p) << 4;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int i = pair_dir(k), io = opp(i);
      const fix m = mulhi((v[io] - v[i]) << (61 - B), pf);   // units of 2^-59
      const fix t = B > 59 ? m << (B - 59) : m;
      v[i] += t;
      v[io] -= t;
    }
  }
#pragma unroll
  for (int i = 0; i < Q; ++i) s[i] = from_fix<B>(v[i]);
}

// Block-wide sum of three doubles; thread 0 writes them to out[slot*3].
__device__ __forceinline__ void block_sum3_store_at(double a, double b, double c, double* out,
                                                    int slot) {
  __shared__ double sh[3][32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
    c += __shfl_down_sync(0xffffffffu, c, o);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { sh[0][wid] = a; sh[1][wid] = b; sh[2][wid] = c; }
  __syncthreads();
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    a = lane < nw ? sh[0][lane] : 0.0;
    b = lane < nw ? sh[1][lane] : 0.0;
    c = lane < nw ? sh[2][lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      b += __shfl_down_sync(0xffffffffu, b, o);
      c += __shfl_down_sync(0xffffffffu, c, o);
    }
    if (lane == 0) {
      out[3 * slot + 0] = a;
      out[3 * slot + 1] = b;
      out[3 * slot + 2] = c;
    }
  }
}

__device__ __forceinline__ void block_sum3_store(double a, double b, double c, double* out) {
  block_sum3_store_at(a, b, c, out, blockIdx.x);
}

}  // namespace lbm
