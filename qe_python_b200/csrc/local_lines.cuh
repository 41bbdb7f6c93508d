// The three passes of the local H|psi> (and the density accumulation) as
// two-factor line transforms, one line per lane (sm_100a).
//
// Same operator and HBM layout as the generic kernels of local_hpsi.cu
// (qepy_pw/_native_fft.pyx qepy_apply_serial_spatial :58-135):
//   z_inverse : inverse z transforms of the occupied sticks
//   plane     : per (z, band) plane the inverse 2-D transform, times V (or
//               |psi|^2 into the density), the forward 2-D transform
//   z_forward : forward z transforms, gather, 1/N and the kinetic term
//
// A line of length n = n1 n2 (both factors <= 16) is transformed in two
// steps: n2 small DFTs of length n1 over the values j + n2 i, a twiddle
// multiplication, and n1 small DFTs of length n2; the forward transform runs
// the same steps backwards.  One thread does one small DFT in registers, and
// consecutive threads take the same small DFT (role) of consecutive lines, so
//   * every lane of a warp works, whatever the factors (lines spread over the
//     lanes of a warp instead left up to 14 of 32 lanes idle in the DFT15 step
//     of 9 x 15 lines and transformed padding rows),
//   * shared-memory accesses of a warp fall on distinct banks: rows of the
//     plane and z lines lie an odd number of values apart, columns are
//     contiguous,
//   * twiddle reads are broadcasts from tables laid out [role][k].
// The steps of one transform are separated by block barriers; several blocks
// per SM fill them.  The plane pass is bound by the shared-memory data path
// (share of its wavefronts: 64 x 64 FP32 84 %, FP64 91 %, 135 x 135 FP32 72 %) with
// issue next (70, 41 and 66 %); FP64 planes of 135 points by neither (60 and
// 34 %): one block of 16 warps fits an SM and waits at its barriers.  The z passes
// wait for their gathered entries and barriers (52 to 67 % of the wavefronts).
// Measured against
// lines spread over the lanes of a warp, plane pass: 135^3 of 96 bands FP32
// 1.313 -> 0.887 ms, FP64 2.627 -> 1.866; 90^3 of 200 bands FP32 0.697 ->
// 0.520; 64^3 of 256 bands FP32 0.209 -> 0.197, FP64 0.383 -> 0.352; z passes
// of 64^3 0.055 + 0.053 -> 0.034 + 0.041, of 135^3 FP32 0.143 + 0.171 -> 0.105
// + 0.125; and against the generic Stockham kernels 80^3 of 60 bands FP32 0.992
// -> 0.114 ms, 45 x 50 x 90 of 37 bands FP64 0.559 -> 0.074.
//
// Plane pass, per block one z plane of one band; rows are the occupied x, the
// contiguous axis is y (sticks are ordered by (y, x), so the lanes of a warp
// read consecutive sticks):
//   rows 1   sticks -> DFT y1 -> twiddle -> plane      (x lanes)
//   rows 2   plane -> DFT y2 -> plane, in place, natural y order
//   per batch of columns (y values):
//     cols 1 plane -> DFT x1 -> twiddle -> buffer      (y lanes)
//     cols 2 buffer -> DFT x2 -> times V -> forward DFT x2 -> twiddle -> buffer
//     cols 3 buffer -> DFT x1 -> plane
//   rows 3   plane -> forward DFT y2 -> twiddle -> plane, in place
//   rows 4   plane -> DFT y1 -> sticks
// The plane holds whole blocks of x2 rows that contain an occupied x (bit i of
// xmask: x in [x2 i, x2 (i + 1))), so that a column's values sit at offsets
// that are uniform over the block; the rows among them without sticks stay
// zero on input and are not transformed.  Blocks of y (z) without sticks
// (entries) are neither read nor written.
#pragma once

#include "line_dft.cuh"
#include "local_plan.cuh"

namespace qeb {
namespace lines {

constexpr int kSticks = 32;  // sticks of one z block: one lane each
constexpr int kZThreads = 256;
constexpr int kAhead = 4;    // entries per thread that a z pass fetches ahead of a barrier

template <typename T>
struct KDesc {
  const C2<T>* psi;
  C2<T>* out;
  const T* kinetic;
  C2<T>* sticks;
  const int32_t* entry_g;
  const int32_t* entry_pos;
  const int32_t* stick_off;
  const int32_t* stick_map;
  int64_t ld, ldo;
  int nst, rows, nb;
  uint32_t xmask, ymask, zmask;
};

template <typename T>
struct KBatch {
  KDesc<T> k[QEB_MAX_KBATCH];
};

// Factors and sizes of the plane (z lines): compile-time for the cubic
// lengths of line_lengths.cuh, run-time otherwise.  keep_x(d, i): whether block
// i of x holds a stick, row_block(i): its place among the kept blocks.
template <int N1, int N2, int K, int COLUMNS>
struct StaticPlane {
  static constexpr int x1 = N1, x2 = N2, y1 = N1, y2 = N2, nx = N1 * N2, ny = N1 * N2;
  static constexpr int stride = ny | 1, columns = COLUMNS, rows = 2 * K * N2;
  static constexpr bool kStatic = true;
  static_assert(2 * K <= N1, "kept blocks");
  static constexpr unsigned kZero = ((1u << (N1 - K)) - 1u) & ~((1u << K) - 1u);
  template <class D>
  __device__ static constexpr int rows_of(const D&, const StaticPlane&) { return rows; }
  template <class D>
  __device__ static constexpr bool keep_x(const D&, int i) { return !((kZero >> i) & 1u); }
  template <class D>
  __device__ static constexpr bool keep_y(const D&, int i) { return !((kZero >> i) & 1u); }
  template <class D>
  __device__ static constexpr int row_block(const D&, int i) { return i < K ? i : i - (N1 - 2 * K); }
};
struct RuntimePlane {
  int x1, x2, y1, y2, nx, ny, stride, columns, rows;
  static constexpr bool kStatic = false;
  static constexpr unsigned kZero = 0;
  template <class D>
  __device__ static int rows_of(const D& d, const RuntimePlane&) { return d.rows; }
  template <class D>
  __device__ static bool keep_x(const D& d, int i) { return (d.xmask >> i) & 1u; }
  template <class D>
  __device__ static bool keep_y(const D& d, int i) { return (d.ymask >> i) & 1u; }
  template <class D>
  __device__ static int row_block(const D& d, int i) { return __popc(d.xmask & ((1u << i) - 1u)); }
};
template <int N1, int N2>
struct StaticZ {
  static constexpr int z1 = N1, z2 = N2, nz = N1 * N2, stride = nz | 1;
  static constexpr bool kStatic = true;
};
struct RuntimeZ {
  int z1, z2, nz, stride;
  static constexpr bool kStatic = false;
};

// fn(integral_constant<radix>) for a radix known at compile time or not.
template <int R, class Fn>
__device__ __forceinline__ void with_radix(std::integral_constant<int, R> r, Fn&& fn) {
  fn(r);
}
template <class Fn>
__device__ __forceinline__ void with_radix(int r, Fn&& fn) {
  switch (r) {
    case 2: fn(std::integral_constant<int, 2>{}); break;
    case 3: fn(std::integral_constant<int, 3>{}); break;
    case 4: fn(std::integral_constant<int, 4>{}); break;
    case 5: fn(std::integral_constant<int, 5>{}); break;
    case 6: fn(std::integral_constant<int, 6>{}); break;
    case 8: fn(std::integral_constant<int, 8>{}); break;
    case 9: fn(std::integral_constant<int, 9>{}); break;
    case 10: fn(std::integral_constant<int, 10>{}); break;
    case 12: fn(std::integral_constant<int, 12>{}); break;
    case 15: fn(std::integral_constant<int, 15>{}); break;
    default: fn(std::integral_constant<int, 16>{}); break;
  }
}
#define QEB_RADIX(P, field, ...)                                          \
  do {                                                                    \
    if constexpr (std::decay_t<decltype(P)>::kStatic)                     \
      with_radix(std::integral_constant<int, std::decay_t<decltype(P)>::field>{}, __VA_ARGS__); \
    else                                                                  \
      with_radix(static_cast<int>((P).field), __VA_ARGS__);               \
  } while (0)

// t / lines for t < 4096 and lines <= 256 with inv = ceil(2^20 / lines):
// t (lines inv - 2^20) < t lines < 2^20 keeps the quotient exact.
__device__ __forceinline__ int quotient(int t, unsigned inv) {
  return (int)(((unsigned)t * inv) >> 20);
}
inline __host__ __device__ constexpr unsigned inverse_of(int lines) {
  return ((1u << 20) + lines - 1) / lines;
}

template <typename T, class Z>
__device__ __forceinline__ void z_inverse_body(const KDesc<T>& d, const Z& g,
                                               const C2<T>* __restrict__ tw_z, int block_x,
                                               int64_t band) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<T>* lines = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* tw = lines + kSticks * g.stride;
  const int tid = threadIdx.x, threads = blockDim.x;
  const int s0 = block_x * kSticks;
  const int nsl = min(kSticks, d.nst - s0);
  // the first entries are on their way while the lines are zeroed
  const int e0 = d.stick_off[s0], e1 = d.stick_off[s0 + nsl];
  const C2<T>* col = d.psi + band * d.ld;
  int pos[kAhead];
  C2<T> value[kAhead];
#pragma unroll
  for (int u = 0; u < kAhead; ++u) {
    const int e = e0 + tid + u * threads;
    pos[u] = e < e1 ? d.entry_pos[e] : -1;
    if (pos[u] >= 0) value[u] = col[d.entry_g[e]];
  }
  for (int i = tid; i < g.nz; i += threads) tw[i] = tw_z[(i / g.z1) * (i % g.z1)];
  for (int i = tid; i < kSticks * g.stride; i += threads) lines[i] = mk<T>(0, 0);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kAhead; ++u)
    if (pos[u] >= 0) lines[pos[u]] = value[u];
  for (int e = e0 + tid + kAhead * threads; e < e1; e += threads)
    lines[d.entry_pos[e]] = col[d.entry_g[e]];
  __syncthreads();
  const uint32_t zmask = d.zmask;
  QEB_RADIX(g, z1, [&](auto r) {
    constexpr int R = decltype(r)::value;
    for (int t = tid; t < g.z2 * kSticks; t += threads) {
      const int j = t / kSticks, s = t % kSticks;
      C2<T>* p = lines + s * g.stride + j;
      C2<T> v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = ((zmask >> i) & 1u) ? p[i * g.z2] : mk<T>(0, 0);
      dft<T, R, true>(v);
      p[0] = v[0];
#pragma unroll
      for (int k = 1; k < R; ++k) p[k * g.z2] = twiddle_conj(v[k], tw[j * R + k]);
    }
  });
  __syncthreads();
  C2<T>* out = d.sticks + band * (int64_t)g.nz * d.nst + s0;
  QEB_RADIX(g, z2, [&](auto r) {
    constexpr int R = decltype(r)::value;
    for (int t = tid; t < g.z1 * kSticks; t += threads) {
      const int k = t / kSticks, s = t % kSticks;
      const C2<T>* p = lines + s * g.stride + R * k;
      C2<T> v[R];
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = p[j];
      dft<T, R, true>(v);
      if (s < nsl) {
#pragma unroll
        for (int q = 0; q < R; ++q) out[(int64_t)(k + g.z1 * q) * d.nst + s] = v[q];
      }
    }
  });
}

template <typename T, class Z>
__device__ __forceinline__ void z_forward_body(const KDesc<T>& d, const Z& g,
                                               const C2<T>* __restrict__ tw_z, T inv_n,
                                               int block_x, int64_t band) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<T>* lines = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* tw = lines + kSticks * g.stride;
  const int tid = threadIdx.x, threads = blockDim.x;
  const int s0 = block_x * kSticks;
  const int nsl = min(kSticks, d.nst - s0);
  for (int i = tid; i < g.nz; i += threads) tw[i] = tw_z[(i / g.z2) * (i % g.z2)];
  __syncthreads();
  const C2<T>* in = d.sticks + band * (int64_t)g.nz * d.nst + s0;
  QEB_RADIX(g, z2, [&](auto r) {
    constexpr int R = decltype(r)::value;
    for (int t = tid; t < g.z1 * kSticks; t += threads) {
      const int k = t / kSticks, s = t % kSticks;
      C2<T> v[R];
#pragma unroll
      for (int p = 0; p < R; ++p)
        v[p] = s < nsl ? in[(int64_t)(k + g.z1 * p) * d.nst + s] : mk<T>(0, 0);
      dft<T, R, false>(v);
      C2<T>* o = lines + s * g.stride + R * k;
      o[0] = v[0];
#pragma unroll
      for (int q = 1; q < R; ++q) o[q] = twiddle(v[q], tw[k * R + q]);
    }
  });
  __syncthreads();
  const uint32_t zmask = d.zmask;
  QEB_RADIX(g, z1, [&](auto r) {
    constexpr int R = decltype(r)::value;
    for (int t = tid; t < g.z2 * kSticks; t += threads) {
      const int j = t / kSticks, s = t % kSticks;
      C2<T>* p = lines + s * g.stride + j;
      C2<T> v[R];
#pragma unroll
      for (int k = 0; k < R; ++k) v[k] = p[k * g.z2];
      dft<T, R, false>(v);
#pragma unroll
      for (int i = 0; i < R; ++i)
        if ((zmask >> i) & 1u) p[i * g.z2] = v[i];
    }
  });
  const int e0 = d.stick_off[s0], e1 = d.stick_off[s0 + nsl];
  const C2<T>* col = d.psi + band * d.ld;
  C2<T>* dst = d.out + band * d.ldo;
  // the first entries' operands are on their way during the barrier
  int index[kAhead], pos[kAhead];
  C2<T> own[kAhead];
  T kinetic[kAhead];
#pragma unroll
  for (int u = 0; u < kAhead; ++u) {
    const int e = e0 + tid + u * threads;
    index[u] = e < e1 ? d.entry_g[e] : -1;
    if (index[u] < 0) continue;
    pos[u] = d.entry_pos[e];
    if (d.kinetic != nullptr) {
      kinetic[u] = d.kinetic[index[u]];
      own[u] = col[index[u]];
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kAhead; ++u) {
    if (index[u] < 0) continue;
    C2<T> v = scale(lines[pos[u]], inv_n);
    if (d.kinetic != nullptr) v = add_scaled(v, kinetic[u], own[u]);
    dst[index[u]] = v;
  }
  for (int e = e0 + tid + kAhead * threads; e < e1; e += threads) {
    const int gi = d.entry_g[e];
    C2<T> v = scale(lines[d.entry_pos[e]], inv_n);
    if (d.kinetic != nullptr) v = add_scaled(v, d.kinetic[gi], col[gi]);
    dst[gi] = v;
  }
}

// Density target of MODE 1: grid[x sx + y sy + z sz] += weights[band] |psi|^2.
struct DensityTarget {
  const double* weights;
  double* grid;
  int64_t sx, sy, sz;
};

constexpr __host__ __device__ int even(int n) { return (n + 1) & ~1; }

// Values of the twiddle tables [role][k] (rows padded to an even length):
// inverse n2 x n1, forward n1 x n2.
constexpr __host__ __device__ int twiddle_values(int n1, int n2) {
  return n2 * even(n1) + n1 * even(n2);
}

template <typename T>
constexpr size_t plane_smem(int x1, int x2, int y1, int y2, int rows, int columns) {
  return sizeof(C2<T>) * ((size_t)rows * ((y1 * y2) | 1) + (size_t)x1 * x2 * columns +
                          twiddle_values(x1, x2) + twiddle_values(y1, y2));
}

constexpr size_t kMaxSmem = 227 * 1024, kSmemPerSm = 228 * 1024;

// Launch bounds of a plane kernel: most threads per block and blocks per SM that
// its registers allow (FP32 64 per thread; FP64 80 up to DFT10, where three
// blocks of 256 threads measured faster than two, 64^3 0.387 -> 0.358 ms and
// 90^3 0.535 -> 0.491, and 128 for longer DFTs, which spill below that: 135^3
// 1.83 ms at 128, 2.68 at 80).  The run-time kernel holds every length.
struct PlaneBounds {
  int threads, blocks;
};
template <typename T>
constexpr PlaneBounds plane_bounds(int x1, int x2, int y1, int y2, bool compiled) {
  if (sizeof(T) == 4) return {512, 2};
  const bool small = x1 <= 10 && x2 <= 10 && y1 <= 10 && y2 <= 10;
  return compiled && small ? PlaneBounds{384, 2} : PlaneBounds{512, 1};
}

// Relative time of a plane with `columns` columns per batch and t threads,
// `resident` blocks per SM at most: every step's rounds of t small DFTs, each
// round weighted by its DFT's length and lasting t plus a latency that the
// resident blocks share, and a cost per barrier.  `whole` of a round's
// idle threads count (0: other blocks use their issue slots).  The constants
// were fitted to 51 timings (FP32: 64, 90 and 135 points; FP64: 64, 90, 108 and
// 135 points; batches of 16 to 90 columns, 96 to 512 threads; planes per
// second within 4 % rms, where the timings of one length span up to 1.4 x).
template <typename T>
constexpr double plane_cost(int x1, int x2, int y1, int y2, int rows, int columns, int t,
                            int budget, int resident, double whole) {
  constexpr bool single = sizeof(T) == 4;
  const int ny = y1 * y2, batches = (ny + columns - 1) / columns;
  const int by_smem =
      (int)(kSmemPerSm / (plane_smem<T>(x1, x2, y1, y2, rows, columns) + 1024));
  int blocks = budget / t;  // by registers
  blocks = blocks < by_smem ? blocks : by_smem;
  blocks = blocks < resident ? blocks : resident;
  if (blocks < 1) blocks = 1;
  const int tasks[4] = {x2 * columns, x1 * columns, y2 * rows, y1 * rows};
  const double weight[4] = {24.0 * x1 * batches, 30.0 * x2 * batches, 26.0 * y1, 29.0 * y2};
  double work = 0.0;
  for (int i = 0; i < 4; ++i)
    work += weight[i] * (whole * ((tasks[i] + t - 1) / t) + (1.0 - whole) * tasks[i] / t);
  return work * (t + (single ? 128.0 : 256.0) / blocks) + 2.0e4 * (3 * batches + 4) / blocks;
}

template <typename T>
constexpr double kWholeRounds = sizeof(T) == 4 ? 0.0 : 0.4;

// Columns of one batch, by the cost above; 0: the plane does not fit.
template <typename T>
constexpr int plane_columns(int x1, int x2, int y1, int y2, int rows, bool compiled) {
  const int ny = y1 * y2;
  const PlaneBounds bounds = plane_bounds<T>(x1, x2, y1, y2, compiled);
  const int budget = bounds.threads * bounds.blocks;
  int best = 0;
  double best_cost = 0.0;
  for (int batches = 1; batches <= ny; ++batches) {
    const int columns = (ny + batches - 1) / batches;
    if (batches > 8 && best > 0) break;
    if (plane_smem<T>(x1, x2, y1, y2, rows, columns) > kMaxSmem) continue;
    for (int t = 64; t <= bounds.threads; t += 32) {
      const double cost =
          plane_cost<T>(x1, x2, y1, y2, rows, columns, t, budget, 32, kWholeRounds<T>);
      if (best == 0 || cost < best_cost) best = columns, best_cost = cost;
    }
  }
  return best;
}

// Threads of a launch of `blocks` plane blocks: a launch that leaves less than
// two blocks per SM is bound by the rounds of one block.
template <typename T, class P>
int plane_threads(const P& g, int64_t blocks) {
  const int64_t per_sm = (blocks + 147) / 148;
  const int resident = per_sm < 32 ? (int)per_sm : 32;
  const double whole = per_sm < 2 ? 1.0 : kWholeRounds<T>;
  const PlaneBounds bounds = plane_bounds<T>(g.x1, g.x2, g.y1, g.y2, P::kStatic);
  const int budget = bounds.threads * bounds.blocks;
  int best = 64;
  double best_cost = 0.0;
  for (int t = 64; t <= bounds.threads; t += 32) {
    const double cost =
        plane_cost<T>(g.x1, g.x2, g.y1, g.y2, g.rows, g.columns, t, budget, resident, whole);
    if (t == 64 || cost < best_cost) best = t, best_cost = cost;
  }
  return best;
}

template <typename T>
RuntimePlane runtime_plane(const qeb_local_plan* p, int rows) {
  RuntimePlane g;
  line_split(p->nx, &g.x1, &g.x2);
  line_split(p->ny, &g.y1, &g.y2);
  g.nx = p->nx;
  g.ny = p->ny;
  g.stride = p->ny | 1;
  g.rows = rows;
  g.columns = rows == p->line_rows ? p->line_columns
                                   : plane_columns<T>(g.x1, g.x2, g.y1, g.y2, rows, false);
  return g;
}

// Launch of the plane pass (local_plane_f32.cu, local_plane_f64.cu) over nk k
// points of one line_k; nb == 0 prepares the kernel instead (plan creation).
int plane_pass(const KBatch<float>& kb, const qeb_local_plan* p, int mode, int nk, int nb,
               const float* potential, const DensityTarget& rho, cudaStream_t s);
int plane_pass(const KBatch<double>& kb, const qeb_local_plan* p, int mode, int nk, int nb,
               const double* potential, const DensityTarget& rho, cudaStream_t s);

template <typename T>
const C2<T>* tw_at(const qeb_local_plan* p, int which) {
  const C2<T>* base = static_cast<const C2<T>*>(p->tw);
  return which == 0 ? base : (which == 1 ? base + p->nx : base + p->nx + p->ny);
}

template <typename T>
__device__ __forceinline__ void load_twiddles(C2<T>* inverse, C2<T>* fwd,
                                              const C2<T>* __restrict__ tw, int n1, int n2) {
  for (int i = threadIdx.x; i < n1 * n2; i += blockDim.x) {
    const int j = i / n1, k = i - j * n1;
    const C2<T> w = tw[j * k];
    inverse[j * even(n1) + k] = w;
    fwd[k * even(n2) + j] = w;
  }
}

// The R twiddles of one role (rows of an even number of values: two complex64
// values a load; a load per value took 1 to 5 % of the plane pass).
template <typename T, int R>
__device__ __forceinline__ void load_role(C2<T> (&w)[even(R)], const C2<T>* p) {
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int k = 0; k < even(R); k += 2) {
      const float4 v = *reinterpret_cast<const float4*>(p + k);
      w[k] = mk<T>(v.x, v.y);
      w[k + 1] = mk<T>(v.z, v.w);
    }
  } else {
#pragma unroll
    for (int k = 0; k < R; ++k) w[k] = p[k];
  }
}

// MODE 0: local potential; MODE 1: density accumulation.
template <typename T, int MODE, class P>
__device__ __forceinline__ void plane_body(const KDesc<T>& d, const P& g, int nz,
                                           const C2<T>* __restrict__ tw_x,
                                           const C2<T>* __restrict__ tw_y,
                                           const T* __restrict__ potential,
                                           const DensityTarget& rho, int z, int64_t band) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, threads = blockDim.x;
  const int rows = P::rows_of(d, g);
  constexpr unsigned Z = P::kZero;
  C2<T>* twx_inv = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* twx_fwd = twx_inv + g.x2 * even(g.x1);
  C2<T>* twy_inv = twx_inv + twiddle_values(g.x1, g.x2);
  C2<T>* twy_fwd = twy_inv + g.y2 * even(g.y1);
  C2<T>* buf = twy_inv + twiddle_values(g.y1, g.y2);
  C2<T>* plane = buf + g.nx * g.columns;
  C2<T>* srow = d.sticks + (band * nz + z) * (int64_t)d.nst;
  const unsigned rinv = inverse_of(rows), cinv = inverse_of(g.columns);
  // rows 1; the first DFT's sticks are on their way while the tables load
  QEB_RADIX(g, y1, [&](auto r) {
    constexpr int R = decltype(r)::value;
    const int total = g.y2 * rows;
    C2<T> v[R];
    auto fetch = [&](int t) {
      int idx[R];
#pragma unroll
      for (int i = 0; i < R; ++i)
        idx[i] = P::keep_y(d, i) ? __ldg(d.stick_map + t + i * g.y2 * rows) : -1;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        v[i] = mk<T>(0, 0);
        if (P::keep_y(d, i) && idx[i] >= 0) v[i] = srow[idx[i]];
      }
    };
    if (tid < total) fetch(tid);
    load_twiddles(twx_inv, twx_fwd, tw_x, g.x1, g.x2);
    load_twiddles(twy_inv, twy_fwd, tw_y, g.y1, g.y2);
    __syncthreads();
    for (int t = tid; t < total; t += threads) {
      if (t != tid) fetch(t);
      const int j = quotient(t, rinv), a = t - j * rows;
      dft<T, R, true, Z>(v);
      C2<T>* o = plane + a * g.stride + j * R;
      C2<T> w[even(R)];
      load_role<T, R>(w, twy_inv + j * even(R));
      o[0] = v[0];
#pragma unroll
      for (int k = 1; k < R; ++k) o[k] = twiddle_conj(v[k], w[k]);
    }
  });
  __syncthreads();
  // rows 2
  QEB_RADIX(g, y2, [&](auto r) {
    constexpr int R = decltype(r)::value;
    for (int t = tid; t < g.y1 * rows; t += threads) {
      const int k = quotient(t, rinv), a = t - k * rows;
      C2<T>* p = plane + a * g.stride + k;
      C2<T> v[R];
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = p[j * g.y1];
      dft<T, R, true>(v);
#pragma unroll
      for (int j = 0; j < R; ++j) p[j * g.y1] = v[j];
    }
  });
  __syncthreads();
  double weight = 0.0;
  if (MODE == 1) weight = rho.weights[band];
  for (int c0 = 0; c0 < g.ny; c0 += g.columns) {
    const int nc = min(g.columns, g.ny - c0);
    // cols 1
    QEB_RADIX(g, x1, [&](auto r) {
      constexpr int R = decltype(r)::value;
      for (int t = tid; t < g.x2 * g.columns; t += threads) {
        const int j = quotient(t, cinv), c = t - j * g.columns;
        if (c >= nc) continue;
        const C2<T>* p = plane + j * g.stride + c0 + c;
        C2<T> v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
          v[i] = mk<T>(0, 0);
          if (P::keep_x(d, i)) v[i] = p[P::row_block(d, i) * g.x2 * g.stride];
        }
        dft<T, R, true, Z>(v);
        C2<T>* o = buf + j * R * g.columns + c;
        C2<T> w[even(R)];
        load_role<T, R>(w, twx_inv + j * even(R));
        o[0] = v[0];
#pragma unroll
        for (int k = 1; k < R; ++k) o[k * g.columns] = twiddle_conj(v[k], w[k]);
      }
    });
    __syncthreads();
    // cols 2
    QEB_RADIX(g, x2, [&](auto r) {
      constexpr int R = decltype(r)::value;
      for (int t = tid; t < g.x1 * g.columns; t += threads) {
        const int k = quotient(t, cinv), c = t - k * g.columns;
        if (c >= nc) continue;
        C2<T>* p = buf + t;
        C2<T> v[R];
#pragma unroll
        for (int j = 0; j < R; ++j) v[j] = p[j * g.x1 * g.columns];
        if constexpr (MODE == 0) {
          const T* vp = potential + (z * g.nx + k) * (int64_t)g.ny + c0 + c;
          T pot[R];
#pragma unroll
          for (int q = 0; q < R; ++q) pot[q] = __ldg(vp + q * g.x1 * g.ny);
          dft<T, R, true>(v);
#pragma unroll
          for (int q = 0; q < R; ++q) v[q] = scale(v[q], pot[q]);
          dft<T, R, false>(v);
          C2<T> w[even(R)];
          load_role<T, R>(w, twx_fwd + k * even(R));
          p[0] = v[0];
#pragma unroll
          for (int q = 1; q < R; ++q) p[q * g.x1 * g.columns] = twiddle(v[q], w[q]);
        } else {
          dft<T, R, true>(v);
          double* o = rho.grid + z * rho.sz + k * rho.sx + (c0 + c) * rho.sy;
#pragma unroll
          for (int q = 0; q < R; ++q) {
            const double m = (double)v[q].re * v[q].re + (double)v[q].im * v[q].im;
            atomicAdd(o + q * g.x1 * rho.sx, weight * m);
          }
        }
      }
    });
    __syncthreads();
    if constexpr (MODE == 0) {
      // cols 3
      QEB_RADIX(g, x1, [&](auto r) {
        constexpr int R = decltype(r)::value;
        for (int t = tid; t < g.x2 * g.columns; t += threads) {
          const int q = quotient(t, cinv), c = t - q * g.columns;
          if (c >= nc) continue;
          const C2<T>* p = buf + q * R * g.columns + c;
          C2<T> v[R];
#pragma unroll
          for (int k = 0; k < R; ++k) v[k] = p[k * g.columns];
          dft<T, R, false>(v);
          C2<T>* o = plane + q * g.stride + c0 + c;
#pragma unroll
          for (int i = 0; i < R; ++i)
            if (P::keep_x(d, i)) o[P::row_block(d, i) * g.x2 * g.stride] = v[i];
        }
      });
      __syncthreads();
    }
  }
  if constexpr (MODE == 0) {
    // rows 3
    QEB_RADIX(g, y2, [&](auto r) {
      constexpr int R = decltype(r)::value;
      for (int t = tid; t < g.y1 * rows; t += threads) {
        const int k = quotient(t, rinv), a = t - k * rows;
        C2<T>* p = plane + a * g.stride + k;
        C2<T> v[R];
#pragma unroll
        for (int j = 0; j < R; ++j) v[j] = p[j * g.y1];
        dft<T, R, false>(v);
        C2<T> w[even(R)];
        load_role<T, R>(w, twy_fwd + k * even(R));
        p[0] = v[0];
#pragma unroll
        for (int q = 1; q < R; ++q) p[q * g.y1] = twiddle(v[q], w[q]);
      }
    });
    __syncthreads();
    // rows 4
    QEB_RADIX(g, y1, [&](auto r) {
      constexpr int R = decltype(r)::value;
      for (int t = tid; t < g.y2 * rows; t += threads) {
        const int q = quotient(t, rinv), a = t - q * rows;
        int idx[R];
#pragma unroll
        for (int i = 0; i < R; ++i)
          idx[i] = P::keep_y(d, i) ? __ldg(d.stick_map + t + i * g.y2 * rows) : -1;
        const C2<T>* p = plane + a * g.stride + q * R;
        C2<T> v[R];
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = p[k];
        dft<T, R, false>(v);
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (P::keep_y(d, i) && idx[i] >= 0) srow[idx[i]] = v[i];
      }
    });
  }
}

}  // namespace lines
}  // namespace qeb
