// Complex GEMMs of the nonlocal projector and Davidson subspace contractions.
//
//   C = alpha * op(A) * B + beta * C,   op(A) = A ("N") or A^H ("C")
//
// All matrices are column-major with explicit leading dimensions.  The
// plain form (complex128) runs on the FP64 tensor pipe (mma.sync m8n8k4; a
// tcgen05 kind for FP64 does not exist) fed by a cp.async ring; complex64
// products too small for the split-TF32 tensor-core GEMM run on a
// register-tiled FP32 SIMT kernel (64 x 64 block tile, 4 x 4 complex micro
// tile per thread, 16-deep K tiles double-buffered in shared memory).
// Contractions over the long plane-wave dimension (calbec beta^H psi,
// Davidson V^H HV) split K across blocks; the partial tiles go to caller
// scratch and a second kernel reduces them in a fixed order, so results are
// deterministic.
//
// Reference calls replaced: projector_overlaps (ZGEMM ConjTrans/NoTrans,
// qepy_pw/_native_fft.pyx:694-731), add_projector_product (ZGEMM beta=1,
// :782-836), the Davidson reduced-matrix and Ritz products
// (qepy_pw/diagonalization.py:658-726) and coupling @ overlaps (:348).
#include <mutex>
#include <type_traits>

#include "qeb_common.cuh"
#include "../../include/qe_b200.h"

using qeb::C2;

namespace {

constexpr int BM = 64, BN = 64, BK = 16, THREADS = 256;

template <typename T>
struct Tile {
  C2<T> a[2][BK][BM];
  C2<T> b[2][BK][BN];
};

template <typename T, bool CONJ_A>
__device__ __forceinline__ void load_tiles(const C2<T>* __restrict__ A, int64_t lda,
                                           const C2<T>* __restrict__ B, int64_t ldb, int M,
                                           int N, int k0, int k1, int m0, int n0,
                                           C2<T> (&ra)[4], C2<T> (&rb)[4]) {
  const int t = threadIdx.x;
  const C2<T> zero = qeb::mk<T>(0, 0);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    if (CONJ_A) {
      // op(A)(m, k) = conj(A[k + m*lda]), contiguous along k
      const int k = t % BK, m = t / BK + 16 * r;
      const int gk = k0 + k, gm = m0 + m;
      C2<T> v = zero;
      if (gk < k1 && gm < M) {
        v = A[gk + (int64_t)gm * lda];
        v.im = -v.im;
      }
      ra[r] = v;
    } else {
      // op(A)(m, k) = A[m + k*lda], contiguous along m
      const int m = t % BM, k = t / BM + 4 * r;
      const int gk = k0 + k, gm = m0 + m;
      ra[r] = (gk < k1 && gm < M) ? A[gm + (int64_t)gk * lda] : zero;
    }
    const int k = t % BK, n = t / BK + 16 * r;
    const int gk = k0 + k, gn = n0 + n;
    rb[r] = (gk < k1 && gn < N) ? B[gk + (int64_t)gn * ldb] : zero;
  }
}

template <typename T, bool CONJ_A>
__device__ __forceinline__ void store_tiles(Tile<T>& s, int buf, const C2<T> (&ra)[4],
                                            const C2<T> (&rb)[4]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    if (CONJ_A) {
      s.a[buf][t % BK][t / BK + 16 * r] = ra[r];
    } else {
      s.a[buf][t / BM + 4 * r][t % BM] = ra[r];
    }
    s.b[buf][t % BK][t / BK + 16 * r] = rb[r];
  }
}

// One block computes a BM x BN tile of op(A) B over K range [kbeg, kend).
// split == 0: C = alpha*acc + beta*C.  split > 0: write acc to the partial
// buffer P (slice blockIdx.z, ldp = M).
template <typename T, bool CONJ_A>
__global__ void __launch_bounds__(THREADS) gemm_kernel(int M, int N, int K, int kchunk,
                                                       C2<T> alpha, const C2<T>* __restrict__ A,
                                                       int64_t lda, const C2<T>* __restrict__ B,
                                                       int64_t ldb, C2<T> beta, C2<T>* C,
                                                       int64_t ldc, C2<T>* __restrict__ P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Tile<T>& s = *reinterpret_cast<Tile<T>*>(smem_raw);
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int kbeg = blockIdx.z * kchunk;
  const int kend = min(K, kbeg + kchunk);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  C2<T> acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = qeb::mk<T>(0, 0);
  C2<T> ra[4], rb[4];
  int buf = 0;
  if (kbeg < kend) {
    load_tiles<T, CONJ_A>(A, lda, B, ldb, M, N, kbeg, kend, m0, n0, ra, rb);
    store_tiles<T, CONJ_A>(s, 0, ra, rb);
  }
  __syncthreads();
  for (int k0 = kbeg; k0 < kend; k0 += BK) {
    const bool more = k0 + BK < kend;
    if (more) load_tiles<T, CONJ_A>(A, lda, B, ldb, M, N, k0 + BK, kend, m0, n0, ra, rb);
#pragma unroll 4
    for (int kk = 0; kk < BK; ++kk) {
      C2<T> av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = s.a[buf][kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = s.b[buf][kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j].re = fma(av[i].re, bv[j].re, acc[i][j].re);
          acc[i][j].re = fma(-av[i].im, bv[j].im, acc[i][j].re);
          acc[i][j].im = fma(av[i].re, bv[j].im, acc[i][j].im);
          acc[i][j].im = fma(av[i].im, bv[j].re, acc[i][j].im);
        }
    }
    if (more) store_tiles<T, CONJ_A>(s, buf ^ 1, ra, rb);
    __syncthreads();
    buf ^= 1;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty + 16 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx + 16 * j;
      if (gn >= N) continue;
      if (P != nullptr) {
        P[(int64_t)blockIdx.z * M * N + gm + (int64_t)gn * M] = acc[i][j];
      } else {
        C2<T> v = qeb::cmul(alpha, acc[i][j]);
        C2<T>* c = C + gm + (int64_t)gn * ldc;
        if (beta.re != T(0) || beta.im != T(0)) v = v + qeb::cmul(beta, *c);
        *c = v;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// FP64 products on the tensor pipe.
//
// Bound by the FP64 pipe, whose rate is the same for FMA and mma.sync
// (measured 36.5 and 37.2 TFLOP/s): what the SIMT kernel lost to shared-memory
// loads (8 per 64 FMAs, bank conflicts on the transposed stores) and issue
// slots, one m8n8k4 instruction per 256 multiply-adds gives back.  Four warps
// (2 x 2) share a BM x BN complex tile; a warp's 8-row and 8-column fragments
// are single 16-byte loads (re and im together), and each 8 x 8 x 4 complex
// product is four real ones, op(A)'s conjugation being a sign flip of the
// imaginary fragment.  K advances in steps of kMmaK through kMmaStages
// cp.async buffers (16-byte copies: one complex value, so any leading
// dimension works; values past the edges are zero-filled).
// Shared layouts: K-contiguous operands are rows of kMmaK values at a stride
// of 12 (4 mod 8: the 2 rows x 4 k of a load phase cover all banks), the
// M-contiguous A of op N is rows of BM values at a stride of BM + 2 (2 mod 8).
// Measured against the SIMT kernel: the 23 847 x 184 x 184 rotation 0.373 ->
// 0.218 ms (29.6 TFLOP/s).
constexpr int kMmaK = 8, kMmaStages = 4, kMmaThreads = 128, kMmaStride = kMmaK + 4;

template <int BMT, int BNT, bool CONJ_A>
struct MmaTile {
  static constexpr int a_values = CONJ_A ? BMT * kMmaStride : kMmaK * (BMT + 2);
  static constexpr int b_values = BNT * kMmaStride;
  static constexpr size_t smem = sizeof(double2) * (size_t)kMmaStages * (a_values + b_values);
};

__device__ __forceinline__ void cp_async16(double2* dst, const double2* src, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// One block: the BM x BN tile of op(A) B at (tile_m, tile_n) over the K range
// of slice blockIdx.y.  P == nullptr: C = alpha*acc + beta*C, else the partial
// slice.  Tiles are numbered with n fastest, so the blocks that share rows of
// a tall A run side by side.
template <int BMT, int BNT, bool CONJ_A>
__global__ void __launch_bounds__(kMmaThreads, 2) zgemm_mma_kernel(
    int M, int N, int K, int kchunk, int ntiles, double2 alpha, const double2* __restrict__ A,
    int64_t lda, const double2* __restrict__ B, int64_t ldb, double2 beta, double2* C,
    int64_t ldc, double2* __restrict__ P) {
  using S = MmaTile<BMT, BNT, CONJ_A>;
  constexpr int TM = BMT / 16, TN = BNT / 16;  // 8 x 8 tiles per warp
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* as = reinterpret_cast<double2*>(smem_raw);
  double2* bs = as + kMmaStages * S::a_values;
  const int tile_m = blockIdx.x / ntiles, tile_n = blockIdx.x - tile_m * ntiles;
  const int m0 = tile_m * BMT, n0 = tile_n * BNT;
  const int kbeg = blockIdx.y * kchunk, kend = min(K, kbeg + kchunk);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int wm = (warp & 1) * (BMT / 2), wn = (warp >> 1) * (BNT / 2);
  const int row = lane >> 2, quad = lane & 3;
  const int steps = kend > kbeg ? (kend - kbeg + kMmaK - 1) / kMmaK : 0;

  auto load = [&](int step) {
    if (step < steps) {
      const int slot = step % kMmaStages, k0 = kbeg + step * kMmaK;
      double2* a = as + slot * S::a_values;
      double2* b = bs + slot * S::b_values;
#pragma unroll
      for (int r = 0; r < BMT * kMmaK / kMmaThreads; ++r) {
        const int i = t + r * kMmaThreads;
        const int k = CONJ_A ? i % kMmaK : i / BMT, m = CONJ_A ? i / kMmaK : i % BMT;
        const bool valid = k0 + k < kend && m0 + m < M;
        const double2* src = CONJ_A ? A + (k0 + k) + (int64_t)(m0 + m) * lda
                                    : A + (m0 + m) + (int64_t)(k0 + k) * lda;
        cp_async16(a + (CONJ_A ? m * kMmaStride + k : k * (BMT + 2) + m), valid ? src : A, valid);
      }
#pragma unroll
      for (int r = 0; r < BNT * kMmaK / kMmaThreads; ++r) {
        const int i = t + r * kMmaThreads, k = i % kMmaK, n = i / kMmaK;
        const bool valid = k0 + k < kend && n0 + n < N;
        cp_async16(b + n * kMmaStride + k, valid ? B + (k0 + k) + (int64_t)(n0 + n) * ldb : B,
                   valid);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  double re[TM][TN][2], im[TM][TN][2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;

#pragma unroll
  for (int s = 0; s < kMmaStages - 1; ++s) load(s);
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kMmaStages - 2) : "memory");
    __syncthreads();  // this step's values are in; the slot loaded next has been read
    load(step + kMmaStages - 1);
    const double2* a = as + (step % kMmaStages) * S::a_values;
    const double2* b = bs + (step % kMmaStages) * S::b_values;
#pragma unroll
    for (int kk = 0; kk < kMmaK; kk += 4) {
      double2 av[TM], bv[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int m = wm + 8 * i + row, k = kk + quad;
        av[i] = a[CONJ_A ? m * kMmaStride + k : k * (BMT + 2) + m];
      }
#pragma unroll
      for (int j = 0; j < TN; ++j) bv[j] = b[(wn + 8 * j + row) * kMmaStride + kk + quad];
      // re += ar br, im += ar bi, then re -+ ai bi, im +- ai br: an
      // accumulator is revisited only after all the others
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) mma_f64(re[i][j], av[i].x, bv[j].x);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) mma_f64(im[i][j], av[i].x, bv[j].y);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const double ai = CONJ_A ? av[i].y : -av[i].y;
#pragma unroll
        for (int j = 0; j < TN; ++j) mma_f64(re[i][j], ai, bv[j].y);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const double ai = CONJ_A ? -av[i].y : av[i].y;
#pragma unroll
        for (int j = 0; j < TN; ++j) mma_f64(im[i][j], ai, bv[j].x);
      }
    }
  }
  const bool use_beta = beta.x != 0.0 || beta.y != 0.0;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + wm + 8 * i + row;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int gn = n0 + wn + 8 * j + 2 * quad + c;
        if (gn >= N) continue;
        const double x = re[i][j][c], y = im[i][j][c];
        if (P != nullptr) {
          P[(int64_t)blockIdx.y * M * N + gm + (int64_t)gn * M] = make_double2(x, y);
        } else {
          double2* o = C + gm + (int64_t)gn * ldc;
          double2 v = make_double2(alpha.x * x - alpha.y * y, alpha.x * y + alpha.y * x);
          if (use_beta) {
            const double2 old = *o;
            v.x += beta.x * old.x - beta.y * old.y;
            v.y += beta.x * old.y + beta.y * old.x;
          }
          *o = v;
        }
      }
  }
}

// C = alpha * sum_s P[s] + beta * C, slices summed in ascending order.
template <typename T>
__global__ void reduce_partials(int M, int N, int splits, const C2<T>* __restrict__ P,
                                C2<T> alpha, C2<T> beta, C2<T>* C, int64_t ldc) {
  const int64_t total = (int64_t)M * N;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    C2<T> sum = P[i];
    for (int s = 1; s < splits; ++s) sum = sum + P[(int64_t)s * total + i];
    const int64_t m = i % M, n = i / M;
    C2<T> v = qeb::cmul(alpha, sum);
    C2<T>* c = C + m + n * ldc;
    if (beta.re != T(0) || beta.im != T(0)) v = v + qeb::cmul(beta, *c);
    *c = v;
  }
}

// ---------------------------------------------------------------------------
// Skinny products: one side of the output has at most 16 columns.  The tiled
// kernel above wastes most of a 64-wide tile there and reads the large
// operand once per tile column; these kernels stream the large operand once
// from HBM.  Cases of the hot path:
// calbec and the projector add for a few unconverged bands, the Davidson
// rows of a few correction vectors (new^H [HV, V]) and their Ritz columns.

constexpr int kSkinnyMax = 16;
constexpr int kSkinnyThreads = 256;
constexpr int kSkinnyWarps = kSkinnyThreads / 32;
constexpr int kSkinnyRows = 64;  // rows per block (OP_N), two per lane

// Columns of the large operand per warp (OP_C): each narrow value loaded
// serves that many of its multiply-adds.
constexpr int skinny_cols(int ns) { return ns <= 8 ? 4 : 2; }

// V consecutive values from p; `full` says that all of them are inside.
template <typename T, int V>
__device__ __forceinline__ void load_run(C2<T> (&v)[V], const C2<T>* __restrict__ p, bool full) {
  if constexpr (V == 2) {  // two complex64 values in one 16-byte load
    if (full) {
      const float4 w = __ldg(reinterpret_cast<const float4*>(p));
      v[0] = qeb::mk<T>(w.x, w.y);
      v[1] = qeb::mk<T>(w.z, w.w);
    } else {
      v[0] = p[0];
      v[1] = qeb::mk<T>(0, 0);
    }
  } else {
    v[0] = p[0];
  }
}

// Asynchronous copy of a run of V values (`valid` of them, the rest zero) to
// shared memory, and its reading.
template <typename T, int V>
__device__ __forceinline__ void copy_run(C2<T>* dst, const C2<T>* __restrict__ src, int valid) {
  constexpr int bytes = (int)sizeof(C2<T>) * V;
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int size = (int)sizeof(C2<T>) * valid;
  if constexpr (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(size)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(size)
                 : "memory");
}
template <typename T, int V>
__device__ __forceinline__ void read_run(C2<T> (&v)[V], const C2<T>* src) {
  if constexpr (V == 2) {
    const float4 w = *reinterpret_cast<const float4*>(src);
    v[0] = qeb::mk<T>(w.x, w.y);
    v[1] = qeb::mk<T>(w.z, w.w);
  } else {
    v[0] = src[0];
  }
}

constexpr int kSkinnyRing = 3;  // steps in the ring of skinny_c_kernel

template <typename T, int NS, int V>
constexpr size_t skinny_c_smem() {
  return sizeof(C2<T>) * V * (size_t)kSkinnyRing * (skinny_cols(NS) + NS) * kSkinnyThreads;
}

// D[mb, ns] = sum_k conj(X[k, mb]) Y[k, ns] over this block's K range.  A warp
// owns MC columns of X and reads them with MC + NS loads per 4 MC NS
// multiply-adds, lanes along k (one column per warp with Y staged in shared
// memory was bound by its NS shared-memory loads per value of X: beta^H psi of
// 5 bands, 80 725 x 864 complex64, 257 us).  WK warps share a column group and
// split the K range between them (short products, whose few columns would
// leave the loads of one warp in a chain).  splits == 1: the block writes C
// directly; else the partial slice blockIdx.y of P (Mb x Ns).
// Output mapping: swapped == 0: C[mb, ns] = alpha D + beta C;
//                 swapped == 1: C[ns, mb] = alpha conj(D) + beta C.
template <typename T, int NS, int V, int WK>
__global__ void __launch_bounds__(kSkinnyThreads) skinny_c_kernel(
    int Mb, int Ns, int K, int krange, const C2<T>* __restrict__ X, int64_t ldx,
    const C2<T>* __restrict__ Y, int64_t ldy, C2<T> alpha, C2<T> beta, C2<T>* C, int64_t ldc,
    int swapped, C2<T>* __restrict__ P) {
  constexpr int MC = skinny_cols(NS), WM = kSkinnyWarps / WK;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = (blockIdx.x * WM + warp / WK) * MC;
  const int kbeg = blockIdx.y * krange;
  const int kend = min(K, kbeg + krange);
  const C2<T>* x[MC];
  const C2<T>* y[NS];
#pragma unroll
  for (int i = 0; i < MC; ++i) x[i] = X + (int64_t)min(m0 + i, Mb - 1) * ldx;
#pragma unroll
  for (int n = 0; n < NS; ++n) y[n] = Y + (int64_t)min(n, Ns - 1) * ldy;
  C2<T> acc[MC][NS];
#pragma unroll
  for (int i = 0; i < MC; ++i)
#pragma unroll
    for (int n = 0; n < NS; ++n) acc[i][n] = qeb::mk<T>(0, 0);
  // a ring of runs in shared memory, private to the thread: copies of the next
  // kRing - 1 steps are in flight while one is multiplied, without a barrier
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<T>* ring = reinterpret_cast<C2<T>*>(smem_raw) + (size_t)threadIdx.x * V;
  constexpr int kSlot = kSkinnyThreads * V, kStep = WK * 32 * V;
  const int first = kbeg + ((warp % WK) * 32 + lane) * V;
  const int steps = m0 < Mb && first < kend ? (kend - first + kStep - 1) / kStep : 0;
  auto fetch = [&](int step) {
    if (step < steps) {
      const int k = first + step * kStep;
      const int valid = min(V, kend - k);
      C2<T>* slot = ring + (size_t)(step % kSkinnyRing) * (MC + NS) * kSlot;
#pragma unroll
      for (int i = 0; i < MC; ++i) copy_run<T, V>(slot + i * kSlot, x[i] + k, valid);
#pragma unroll
      for (int n = 0; n < NS; ++n) copy_run<T, V>(slot + (MC + n) * kSlot, y[n] + k, valid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int step = 0; step < kSkinnyRing - 1; ++step) fetch(step);
  for (int step = 0; step < steps; ++step) {
    fetch(step + kSkinnyRing - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kSkinnyRing - 1) : "memory");
    const C2<T>* slot = ring + (size_t)(step % kSkinnyRing) * (MC + NS) * kSlot;
    C2<T> xv[MC][V], yv[NS][V];
#pragma unroll
    for (int i = 0; i < MC; ++i) read_run<T, V>(xv[i], slot + i * kSlot);
#pragma unroll
    for (int n = 0; n < NS; ++n) read_run<T, V>(yv[n], slot + (MC + n) * kSlot);
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int i = 0; i < MC; ++i)
#pragma unroll
        for (int n = 0; n < NS; ++n) {  // conj(x) * y
          acc[i][n].re = fma(xv[i][v].re, yv[n][v].re, acc[i][n].re);
          acc[i][n].re = fma(xv[i][v].im, yv[n][v].im, acc[i][n].re);
          acc[i][n].im = fma(xv[i][v].re, yv[n][v].im, acc[i][n].im);
          acc[i][n].im = fma(-xv[i][v].im, yv[n][v].re, acc[i][n].im);
        }
  }
  C2<T> mine = qeb::mk<T>(0, 0);  // lane l: entry (l / NS, l % NS), then l + 32, ...
  __shared__ C2<T> part[WK > 1 ? kSkinnyWarps : 1][MC * NS];
#pragma unroll
  for (int i = 0; i < MC; ++i)
#pragma unroll
    for (int n = 0; n < NS; ++n) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        acc[i][n].re += __shfl_xor_sync(0xffffffffu, acc[i][n].re, off);
        acc[i][n].im += __shfl_xor_sync(0xffffffffu, acc[i][n].im, off);
      }
      if (lane == i * NS + n) mine = acc[i][n];
    }
  static_assert(MC * NS <= 32, "one entry per lane");
  if constexpr (WK > 1) {
    if (lane < MC * NS) part[warp][lane] = mine;
    __syncthreads();
    if (warp % WK != 0) return;
    if (lane < MC * NS)
#pragma unroll
      for (int w = 1; w < WK; ++w) mine = mine + part[warp + w][lane];
  }
  const int mb = m0 + lane / NS, n = lane % NS;
  if (lane >= MC * NS || mb >= Mb || n >= Ns) return;
  if (P != nullptr) {
    P[(int64_t)blockIdx.y * Mb * Ns + mb + (int64_t)n * Mb] = mine;
  } else {
    if (swapped) mine.im = -mine.im;
    C2<T>* c = swapped ? C + n + (int64_t)mb * ldc : C + mb + (int64_t)n * ldc;
    C2<T> v = qeb::cmul(alpha, mine);
    if (beta.re != T(0) || beta.im != T(0)) v = v + qeb::cmul(beta, *c);
    *c = v;
  }
}

// Sum of the skinny partial slices in ascending order, then the output
// mapping of skinny_c_kernel.
template <typename T>
__global__ void skinny_reduce(int Mb, int Ns, int splits, const C2<T>* __restrict__ P,
                              C2<T> alpha, C2<T> beta, C2<T>* C, int64_t ldc, int swapped) {
  const int64_t total = (int64_t)Mb * Ns;
  const bool use_beta = beta.re != T(0) || beta.im != T(0);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    C2<T> d = P[i];
    for (int s = 1; s < splits; ++s) d = d + P[(int64_t)s * total + i];
    const int64_t mb = i % Mb, n = i / Mb;
    if (swapped) d.im = -d.im;
    C2<T>* c = swapped ? C + n + mb * ldc : C + mb + n * ldc;
    C2<T> v = qeb::cmul(alpha, d);
    if (use_beta) v = v + qeb::cmul(beta, *c);
    *c = v;
  }
}

// C[m, n] = alpha sum_k A[m, k] B[k, n] + beta C[m, n] for N <= NS.  A block
// owns 64 rows, two per lane (V == 2: neighbouring complex64 rows in one
// 16-byte load, else rows 32 apart), and its warps split K; the partial sums
// meet in shared memory four columns at a time.  (One thread per row over the
// whole of K left 2.1 blocks of 256 rows per SM on the 216-atom cell's
// projector add, 80 725 x 864 x 5 complex64.)  With the kernel above: H|psi> of 5
// bands of that cell 0.607 -> 0.345 ms.
template <typename T, int NS, int V>
__global__ void __launch_bounds__(kSkinnyThreads) skinny_n_kernel(
    int M, int N, int K, C2<T> alpha, const C2<T>* __restrict__ A, int64_t lda,
    const C2<T>* __restrict__ B, int64_t ldb, C2<T> beta, C2<T>* C, int64_t ldc) {
  constexpr int kStep = 4;  // output columns reduced at a time
  __shared__ C2<T> part[kSkinnyWarps][kStep][kSkinnyRows];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kSkinnyRows;
  const int r0 = V == 2 ? 2 * lane : lane, r1 = V == 2 ? 2 * lane + 1 : lane + 32;
  const int kper = (K + kSkinnyWarps - 1) / kSkinnyWarps;
  const int kbeg = min(K, warp * kper), kend = min(K, kbeg + kper);
  C2<T> acc[2][NS];
#pragma unroll
  for (int n = 0; n < NS; ++n) acc[0][n] = acc[1][n] = qeb::mk<T>(0, 0);
  const C2<T>* a0 = A + min(m0 + r0, M - 1);
  const C2<T>* a1 = A + min(m0 + r1, M - 1);
  const bool full = m0 + r1 < M;
  const C2<T>* b[NS];
#pragma unroll
  for (int n = 0; n < NS; ++n) b[n] = B + (int64_t)min(n, N - 1) * ldb;
#pragma unroll 4
  for (int k = kbeg; k < kend; ++k) {
    C2<T> av[2];
    if constexpr (V == 2) {
      load_run<T, 2>(av, a0 + (int64_t)k * lda, full);
    } else {
      av[0] = a0[(int64_t)k * lda];
      av[1] = a1[(int64_t)k * lda];
    }
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      const C2<T> bv = b[n][k];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        acc[r][n].re = fma(av[r].re, bv.re, acc[r][n].re);
        acc[r][n].re = fma(-av[r].im, bv.im, acc[r][n].re);
        acc[r][n].im = fma(av[r].re, bv.im, acc[r][n].im);
        acc[r][n].im = fma(av[r].im, bv.re, acc[r][n].im);
      }
    }
  }
  const bool use_beta = beta.re != T(0) || beta.im != T(0);
#pragma unroll
  for (int n0 = 0; n0 < NS; n0 += kStep) {
    if (n0 > 0) __syncthreads();
#pragma unroll
    for (int j = 0; j < kStep; ++j)
      if (n0 + j < NS) {
        part[warp][j][r0] = acc[0][n0 + j];
        part[warp][j][r1] = acc[1][n0 + j];
      }
    __syncthreads();
    const int j = threadIdx.x / kSkinnyRows, r = threadIdx.x % kSkinnyRows;
    const int m = m0 + r, n = n0 + j;
    if (n < NS && n < N && m < M) {
      C2<T> sum = part[0][j][r];
#pragma unroll
      for (int w = 1; w < kSkinnyWarps; ++w) sum = sum + part[w][j][r];
      C2<T>* c = C + m + (int64_t)n * ldc;
      C2<T> v = qeb::cmul(alpha, sum);
      if (use_beta) v = v + qeb::cmul(beta, *c);
      *c = v;
    }
  }
}
static_assert(kSkinnyThreads == 4 * kSkinnyRows, "one output per thread and reduction step");

// C[m, n] as above for tall A: one thread per row over the whole of K, B staged
// in shared memory (every lane reads the same entry).  Sums of four K values are
// formed on their own and added: as many additions in a chain as in the kernel
// above (8 and K / 4; there 2 K / 8 and 8), so no more rounding.  Which of the
// two runs: skinny_row_threads.
constexpr int kSkinnyChunkN = 64;  // K rows staged per step
constexpr int kSkinnyGroup = 8;    // loads of A in flight per thread
// Blocks of 128 rows, registers for five (complex128 of 9 to 16 columns: three)
// per SM: the 631 blocks of 80 725 rows then run in one wave (two).
constexpr int kRowThreads = 128;
template <typename T, int NS>
__global__ void __launch_bounds__(kRowThreads, sizeof(T) * NS <= 64 ? 5 : 3) skinny_rows_kernel(
    int M, int N, int K, C2<T> alpha, const C2<T>* __restrict__ A, int64_t lda,
    const C2<T>* __restrict__ B, int64_t ldb, C2<T> beta, C2<T>* C, int64_t ldc) {
  __shared__ C2<T> bs[kSkinnyChunkN][NS];
  const int m = blockIdx.x * kRowThreads + threadIdx.x;
  const C2<T> zero = qeb::mk<T>(0, 0);
  C2<T> sum[NS];
#pragma unroll
  for (int n = 0; n < NS; ++n) sum[n] = zero;
  const C2<T>* arow = A + (m < M ? m : 0);
  auto add = [&](C2<T> (&acc)[NS], int kk, C2<T> a) {
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      const C2<T> b = bs[kk][n];
      acc[n].re = fma(a.re, b.re, acc[n].re);
      acc[n].re = fma(-a.im, b.im, acc[n].re);
      acc[n].im = fma(a.re, b.im, acc[n].im);
      acc[n].im = fma(a.im, b.re, acc[n].im);
    }
  };
  for (int k0 = 0; k0 < K; k0 += kSkinnyChunkN) {
    __syncthreads();
    for (int i = threadIdx.x; i < NS * kSkinnyChunkN; i += kRowThreads) {
      const int n = i / kSkinnyChunkN, kk = i - n * kSkinnyChunkN;
      const int k = k0 + kk;
      bs[kk][n] = (n < N && k < K) ? B[k + (int64_t)n * ldb] : zero;
    }
    __syncthreads();
    if (m < M) {
      const int kn = min(kSkinnyChunkN, K - k0);
      int kk = 0;
      for (; kk + kSkinnyGroup <= kn; kk += kSkinnyGroup) {
        C2<T> a[kSkinnyGroup];  // loads in flight
#pragma unroll
        for (int u = 0; u < kSkinnyGroup; ++u) a[u] = arow[(int64_t)(k0 + kk + u) * lda];
#pragma unroll
        for (int g = 0; g < kSkinnyGroup; g += 4) {
          C2<T> acc[NS];
#pragma unroll
          for (int n = 0; n < NS; ++n) acc[n] = zero;
#pragma unroll
          for (int u = g; u < g + 4; ++u) add(acc, kk + u, a[u]);
#pragma unroll
          for (int n = 0; n < NS; ++n) sum[n] = sum[n] + acc[n];
        }
      }
      while (kk < kn) {
        C2<T> acc[NS];
#pragma unroll
        for (int n = 0; n < NS; ++n) acc[n] = zero;
        for (const int stop = min(kk + 4, kn); kk < stop; ++kk)
          add(acc, kk, arow[(int64_t)(k0 + kk) * lda]);
#pragma unroll
        for (int n = 0; n < NS; ++n) sum[n] = sum[n] + acc[n];
      }
    }
  }
  if (m >= M) return;
  const bool use_beta = beta.re != T(0) || beta.im != T(0);
#pragma unroll
  for (int n = 0; n < NS; ++n) {
    if (n >= N) break;
    C2<T>* c = C + m + (int64_t)n * ldc;
    C2<T> v = qeb::cmul(alpha, sum[n]);
    if (use_beta) v = v + qeb::cmul(beta, *c);
    *c = v;
  }
}

int g_sm_count = 0;

int sm_count() {
  if (g_sm_count == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (g_sm_count <= 0) g_sm_count = 148;
  }
  return g_sm_count;
}

// Number of K slices: enough blocks for ~2 waves, each slice >= 256 deep.
int choose_splits(int M, int N, int K) {
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  const int want = (2 * sm_count() + tiles - 1) / tiles;
  int by_depth = K / 256;
  if (by_depth < 1) by_depth = 1;
  int s = want < by_depth ? want : by_depth;
  if (s > 64) s = 64;
  return s < 1 ? 1 : s;
}

// Tile edges (64, 48 or 32) and K slices of the FP64 tensor kernel.  The blocks
// of one SM share its FP64 pipe, so the time is that of the SM with the most
// tiles (at kSmRate complex multiply-adds per microsecond), plus writing and
// reading the partial slices of a split; slices are at least 64 deep.  Against
// that, A B runs faster in small tiles, of which more blocks are resident
// (23 847 x 184 x 184: 32 x 32 243 us, 48 x 48 260; 80 725 x 97 x 300: 32 x 32 804,
// 64 x 64 957), A^H B a little faster in large ones, which load less per product
// (512 x 256 x 11 019: 64 x 64 370 us, 32 x 32 385).  The rates only weigh the
// terms against each other.  No fewer slices than choose_splits: rounding grows
// with the length of a chain of additions, and the fewer slices that are often
// faster (512 x 256 x 6000 202 us, 263 so) doubled the error of narrow products
// (512 x 40 x 11 019: 1.7e-15 relative, 8.7e-16 so).
struct MmaPlan {
  int bm = 64, bn = 64, splits = 1;
};

MmaPlan mma_plan(int M, int N, int K, bool split) {
  constexpr double kSmRate = 30.0e3, kSliceBytes = 4.0e6;  // per SM; bytes per us
  const int least = split ? choose_splits(M, N, K) : 1;
  MmaPlan best;
  double best_time = 0.0;
  for (int bm : {64, 48, 32})
    for (int bn : {64, 48, 32}) {
      const int64_t tiles = (int64_t)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
      const double rate = kSmRate * (split ? 1.0 - 0.4 / bm - 0.4 / bn
                                           : 1.0 - 0.05 * (bm * bn / 1024.0 - 1.0));
      for (int s = least; s <= (split ? 64 : 1) && (s == least || K / s >= 64); ++s) {
        const int64_t per_sm = (tiles * s + sm_count() - 1) / sm_count();
        const int depth = ((K + s - 1) / s + kMmaK - 1) / kMmaK * kMmaK;
        double time = (double)per_sm * depth * bm * bn / rate;
        if (s > 1) time += 2.0 + 32.0 * s * M * N / kSliceBytes;  // a second launch, slices
        if (best_time == 0.0 || time < 0.99 * best_time)
          best.bm = bm, best.bn = bn, best.splits = s, best_time = time;
      }
    }
  return best;
}

// Compiled widths of the narrow side.
constexpr int kSkinnyWidths[] = {1, 2, 3, 4, 5, 6, 7, 8, 10, 12, 16};

int skinny_width(int n) {
  for (int w : kSkinnyWidths)
    if (n <= w) return w;
  return kSkinnyMax;
}

// Skinny OP_C plan: the narrow side (N, else M when N is wide), the large
// side mb, the number of K slices (up to four blocks per SM in all, each slice
// at least 1024 deep; by whole waves for 9 to 16 columns against few) and whether
// the warps of a block split K between them (wk: when the blocks would not fill
// the GPU otherwise).
struct SkinnyC {
  bool use = false, swapped = false;
  int mb = 0, ns = 0, splits = 1, wk = 1;
  int groups() const {  // blocks along the large side
    const int per = skinny_cols(skinny_width(ns)) * (kSkinnyWarps / wk);
    return (mb + per - 1) / per;
  }
};

SkinnyC skinny_c_plan(int M, int N, int K) {
  SkinnyC p;
  if (N <= kSkinnyMax) {
    p.use = true, p.mb = M, p.ns = N;
  } else if (M <= kSkinnyMax) {
    p.use = true, p.swapped = true, p.mb = N, p.ns = M;
  } else {
    return p;
  }
  const int by_depth = K / 1024 < 1 ? 1 : K / 1024;
  if (p.ns > 8 && p.mb <= 192) {
    // One block per SM (172 to 221 KB of ring): of four waves at most, and slices
    // of 3072 to 4096 values at most, as many slices as fill their waves best.
    // With slices for two blocks per SM, 80 725 x 97 x 16 ran 448 blocks in four
    // waves (complex64 91 us; 588 blocks, whole waves, 80) and 130 columns 576 (117
    // us; 585 blocks 101).
    p.wk = kSkinnyWarps;
    const int groups = p.groups(), sms = sm_count();
    const int most = 4 * sms / groups, deep = K / 4096;
    double best = 0.0;
    for (int s = deep < 1 ? 1 : (deep < most ? deep : most);
         s <= most && (best == 0.0 || s <= K / 3072); ++s) {
      const int waves = (groups * s + sms - 1) / sms;
      const double fill = (double)groups * s / (waves * sms);
      if (fill >= best) best = fill, p.splits = s;
    }
    return p;
  }
  if ((int64_t)p.groups() * by_depth < 2 * sm_count()) p.wk = kSkinnyWarps;
  const int fill = 4 * sm_count() / p.groups();
  // a split product needs a second launch: not for the depth one block
  // covers in a few loads per lane
  const int deep = p.wk > 1 ? K / 4096 : by_depth;
  p.splits = fill < deep ? fill : deep;
  if (p.splits > 64) p.splits = 64;
  if (p.splits < 1) p.splits = 1;
  return p;
}

template <typename T, int NS>
int launch_skinny_c(const SkinnyC& p, bool wide, int K, int krange, const C2<T>* X, int64_t ldx,
                     const C2<T>* Y, int64_t ldy, C2<T> al, C2<T> be, C2<T>* C, int64_t ldc,
                     C2<T>* partials, cudaStream_t stream) {
  const dim3 grid(p.groups(), p.splits);
  constexpr int V = sizeof(T) == 4 ? 2 : 1;
  const int sw = p.swapped ? 1 : 0;
  auto launch = [&](auto* kernel, size_t smem) {
    const cudaError_t e = qeb::raise_smem_limit(kernel, smem);
    if (e != cudaSuccess) return qeb::cuda_status(e, "skinny product shared memory");
    kernel<<<grid, kSkinnyThreads, smem, stream>>>(p.mb, p.ns, K, krange, X, ldx, Y, ldy, al, be,
                                                   C, ldc, sw, partials);
    return QEB_OK;
  };
  if (p.wk > 1)
    return wide ? launch(skinny_c_kernel<T, NS, V, kSkinnyWarps>, skinny_c_smem<T, NS, V>())
                : launch(skinny_c_kernel<T, NS, 1, kSkinnyWarps>, skinny_c_smem<T, NS, 1>());
  return wide ? launch(skinny_c_kernel<T, NS, V, 1>, skinny_c_smem<T, NS, V>())
              : launch(skinny_c_kernel<T, NS, 1, 1>, skinny_c_smem<T, NS, 1>());
}

// Whether complex64 columns start on 16-byte boundaries (two values a load);
// complex128 values are 16-byte loads in any case.
template <typename T>
bool wide_loads(const C2<T>* p, int64_t ld) {
  return sizeof(T) == 8 || (reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 2 == 0);
}

// Calls fn(integral_constant<width>) for the compiled width of n.
template <class Fn>
void with_width(int n, Fn&& fn) {
  switch (skinny_width(n)) {
    case 1: fn(std::integral_constant<int, 1>{}); break;
    case 2: fn(std::integral_constant<int, 2>{}); break;
    case 3: fn(std::integral_constant<int, 3>{}); break;
    case 4: fn(std::integral_constant<int, 4>{}); break;
    case 5: fn(std::integral_constant<int, 5>{}); break;
    case 6: fn(std::integral_constant<int, 6>{}); break;
    case 7: fn(std::integral_constant<int, 7>{}); break;
    case 8: fn(std::integral_constant<int, 8>{}); break;
    case 10: fn(std::integral_constant<int, 10>{}); break;
    case 12: fn(std::integral_constant<int, 12>{}); break;
    default: fn(std::integral_constant<int, 16>{}); break;
  }
}

template <typename T>
int gemm_skinny_c(int M, int N, int K, C2<T> al, const C2<T>* A, int64_t lda, const C2<T>* B,
                  int64_t ldb, C2<T> be, C2<T>* C, int64_t ldc, void* scratch,
                  int64_t scratch_bytes, cudaStream_t stream) {
  SkinnyC p = skinny_c_plan(M, N, K);
  const int64_t slice_bytes = (int64_t)p.mb * p.ns * (int64_t)sizeof(C2<T>);
  if (p.splits > 1) {
    const int64_t fit = (scratch == nullptr) ? 0 : scratch_bytes / slice_bytes;
    if (fit < p.splits) p.splits = (int)(fit < 1 ? 1 : fit);
  }
  constexpr int kChunk = 64;  // slices start on whole 16-byte loads of a warp
  int krange = (K + p.splits - 1) / p.splits;
  krange = (krange + kChunk - 1) / kChunk * kChunk;
  p.splits = (K + krange - 1) / krange;
  // large operand X and narrow operand Y of D = X^H Y
  const C2<T>* X = p.swapped ? B : A;
  const C2<T>* Y = p.swapped ? A : B;
  const int64_t ldx = p.swapped ? ldb : lda, ldy = p.swapped ? lda : ldb;
  const bool wide = wide_loads(X, ldx) && wide_loads(Y, ldy);
  C2<T>* partials = p.splits > 1 ? static_cast<C2<T>*>(scratch) : nullptr;
  int rc = QEB_OK;
  with_width(p.ns, [&](auto w) {
    rc = launch_skinny_c<T, decltype(w)::value>(p, wide, K, krange, X, ldx, Y, ldy, al, be, C, ldc,
                                                partials, stream);
  });
  if (rc) return rc;
  qeb::count_launches(p.splits > 1 ? 2 : 1);
  if (p.splits > 1) {
    const int64_t total = (int64_t)p.mb * p.ns;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 4 * sm_count()) blocks = 4 * sm_count();
    skinny_reduce<T><<<blocks, 256, 0, stream>>>(p.mb, p.ns, p.splits, partials, al, be, C, ldc,
                                                p.swapped ? 1 : 0);
  }
  return qeb::cuda_status(cudaGetLastError(), "zgemm skinny launch");
}

// Whether an OP_N product runs with one thread per row instead of a K range per
// warp: from some number of rows on, because its blocks then fill the GPU, sooner
// the shorter K is (a block's reduction over its warps costs as much as a few K
// steps) and the wider the narrow side (its values, loaded from global memory
// for every two rows, take over).  The table holds those rows in thousands by
// width of the narrow side and by K, from timings of both over 12 000 to 80 725
// rows, 2 to 900 K values and 1 to 16 columns.  Range per warp and thread per row:
// 80 725 x 600 x 8 complex128 562 and 286 us, 24 000 x 24 x 16 17 and 15; on the other
// side 80 725 x 600 x 9 complex128 468 and 620, 24 000 x 140 x 8 29 and 33.
bool skinny_row_threads(int M, int N, int K, bool single) {
  constexpr int X = 1 << 30;                                    // never
  constexpr int kWidths[] = {2, 3, 4, 5, 6, 7, 8, 10, 12, 16};  // columns up to
  constexpr int kDepths[] = {10, 24, 48, 150};                  // K up to, and above
  constexpr int kRows[2][10][5] = {{{46, X, X, X, X},           // complex128
                                    {32, 32, 36, 52, 36},
                                    {16, 36, 24, 24, 28},
                                    {36, 40, X, X, X},
                                    {16, 24, 32, 52, 60},
                                    {16, 20, 32, 36, 46},
                                    {20, 20, 24, 32, 40},
                                    {16, 24, X, X, X},
                                    {16, 20, 32, X, X},
                                    {12, 16, 24, X, X}},
                                   {{60, 60, X, X, 70},  // complex64
                                    {24, 40, 40, 70, 52},
                                    {24, 32, 32, 52, 60},
                                    {40, 32, X, X, X},
                                    {36, 32, 32, X, 60},
                                    {40, 20, 24, 36, 36},
                                    {40, 20, 20, 20, 20},
                                    {40, 40, X, X, X},
                                    {20, 20, 24, 32, 52},
                                    {20, 16, 24, 32, 40}}};
  int w = 0, d = 0;
  while (w < 9 && N > kWidths[w]) ++w;
  while (d < 4 && K > kDepths[d]) ++d;
  return M / 1000 >= kRows[single ? 1 : 0][w][d];
}

template <typename T>
int gemm_skinny_n(int M, int N, int K, C2<T> al, const C2<T>* A, int64_t lda, const C2<T>* B,
                  int64_t ldb, C2<T> be, C2<T>* C, int64_t ldc, cudaStream_t stream) {
  if (skinny_row_threads(M, N, K, sizeof(T) == 4)) {
    auto* kernel = N <= 4 ? skinny_rows_kernel<T, 4>
                          : (N <= 8 ? skinny_rows_kernel<T, 8> : skinny_rows_kernel<T, 16>);
    const unsigned blocks = (unsigned)(((int64_t)M + kRowThreads - 1) / kRowThreads);
    kernel<<<blocks, kRowThreads, 0, stream>>>(M, N, K, al, A, lda, B, ldb, be, C, ldc);
    qeb::count_launches(1);
    return qeb::cuda_status(cudaGetLastError(), "zgemm skinny launch");
  }
  const dim3 grid((M + kSkinnyRows - 1) / kSkinnyRows);
  const bool wide = sizeof(T) == 4 && wide_loads(A, lda);
  with_width(N, [&](auto w) {
    // complex128: the kernel of 16 columns is the faster one for 11 and 12 too
    // (80 725 x 600 x 12 562 us, compiled for 12 columns 773)
    constexpr int kW = decltype(w)::value;
    constexpr int NS = sizeof(T) == 8 && kW == 12 ? 16 : kW;
    if constexpr (sizeof(T) == 4) {
      if (wide) {
        skinny_n_kernel<T, NS, 2><<<grid, kSkinnyThreads, 0, stream>>>(M, N, K, al, A, lda, B,
                                                                       ldb, be, C, ldc);
        return;
      }
    }
    skinny_n_kernel<T, NS, 1><<<grid, kSkinnyThreads, 0, stream>>>(M, N, K, al, A, lda, B, ldb,
                                                                   be, C, ldc);
  });
  qeb::count_launches(1);
  return qeb::cuda_status(cudaGetLastError(), "zgemm skinny launch");
}

template <int BMT, int BNT, bool CONJ_A>
int launch_mma_tile(int M, int N, int K, int kchunk, int splits, double2 al, const double2* A,
                    int64_t lda, const double2* B, int64_t ldb, double2 be, double2* C,
                    int64_t ldc, double2* partials, cudaStream_t stream) {
  auto* kernel = zgemm_mma_kernel<BMT, BNT, CONJ_A>;
  constexpr size_t smem = MmaTile<BMT, BNT, CONJ_A>::smem;
  const cudaError_t e = qeb::raise_smem_limit(kernel, smem);
  if (e != cudaSuccess) return qeb::cuda_status(e, "zgemm shared-memory limit");
  const int mt = (M + BMT - 1) / BMT, nt = (N + BNT - 1) / BNT;
  if ((int64_t)mt * nt > 0x7fffffff) {
    qeb::set_error("zgemm: matrix too large for one launch");
    return QEB_EUNSUPPORTED;
  }
  kernel<<<dim3(mt * nt, splits), kMmaThreads, smem, stream>>>(M, N, K, kchunk, nt, al, A, lda, B,
                                                               ldb, be, C, ldc, partials);
  return QEB_OK;
}

template <class... Args>
int launch_mma(int opa, int bm, int bn, int M, int N, Args... args) {
  const bool conj = opa == QEB_OP_C;
#define QEB_TILE(m, n)                                                              \
  if (bm == m && bn == n)                                                           \
    return conj ? launch_mma_tile<m, n, true>(M, N, args...)                        \
                : launch_mma_tile<m, n, false>(M, N, args...);
  QEB_TILE(64, 64) QEB_TILE(64, 48) QEB_TILE(64, 32)
  QEB_TILE(48, 64) QEB_TILE(48, 48) QEB_TILE(48, 32)
  QEB_TILE(32, 64) QEB_TILE(32, 48) QEB_TILE(32, 32)
#undef QEB_TILE
  return QEB_EUNSUPPORTED;
}

template <typename T>
int gemm(int opa, int M, int N, int K, const double* alpha, const void* A, int64_t lda,
         const void* B, int64_t ldb, const double* beta, void* C, int64_t ldc, void* scratch,
         int64_t scratch_bytes, cudaStream_t stream) {
  if (M < 0 || N < 0 || K < 0 || (opa != QEB_OP_N && opa != QEB_OP_C)) {
    qeb::set_error("zgemm: invalid sizes or op");
    return QEB_EINVAL;
  }
  if (M == 0 || N == 0) return QEB_OK;
  const int64_t a_rows = (opa == QEB_OP_N) ? M : K;
  if (lda < (a_rows > 0 ? a_rows : 1) || ldb < (K > 0 ? K : 1) || ldc < M) {
    qeb::set_error("zgemm: leading dimension too small (lda=%lld ldb=%lld ldc=%lld)",
                   (long long)lda, (long long)ldb, (long long)ldc);
    return QEB_EINVAL;
  }
  if (C == nullptr || (K > 0 && (A == nullptr || B == nullptr))) {
    qeb::set_error("zgemm: null operand");
    return QEB_EINVAL;
  }
  const C2<T> al = qeb::mk<T>((T)alpha[0], (T)alpha[1]);
  const C2<T> be = qeb::mk<T>((T)beta[0], (T)beta[1]);
  if (K > 0 && opa == QEB_OP_C && (N <= kSkinnyMax || M <= kSkinnyMax))
    return gemm_skinny_c<T>(M, N, K, al, static_cast<const C2<T>*>(A), lda,
                            static_cast<const C2<T>*>(B), ldb, be, static_cast<C2<T>*>(C), ldc,
                            scratch, scratch_bytes, stream);
  if (K > 0 && opa == QEB_OP_N && N <= kSkinnyMax)
    return gemm_skinny_n<T>(M, N, K, al, static_cast<const C2<T>*>(A), lda,
                            static_cast<const C2<T>*>(B), ldb, be, static_cast<C2<T>*>(C), ldc,
                            stream);
  constexpr bool kMma = sizeof(T) == 8;
  const MmaPlan plan = kMma ? mma_plan(M, N, K, opa == QEB_OP_C) : MmaPlan{};
  int splits = kMma ? plan.splits : (opa == QEB_OP_C ? choose_splits(M, N, K) : 1);
  const int64_t slice_bytes = (int64_t)M * N * (int64_t)sizeof(C2<T>);
  if (splits > 1) {
    const int64_t fit = (scratch == nullptr) ? 0 : scratch_bytes / slice_bytes;
    if (fit < splits) splits = (int)(fit < 1 ? 1 : fit);
  }
  constexpr int kStep = kMma ? kMmaK : BK;
  int kchunk = K;
  if (splits > 1) {
    kchunk = (K + splits - 1) / splits;
    kchunk = (kchunk + kStep - 1) / kStep * kStep;
    splits = (K + kchunk - 1) / kchunk;
  }
  if (K == 0) kchunk = 1;
  C2<T>* partials = (splits > 1) ? static_cast<C2<T>*>(scratch) : nullptr;
  if constexpr (kMma) {
    const int rc = launch_mma(opa, plan.bm, plan.bn, M, N, K, kchunk, splits, make_double2(al.re, al.im),
                              static_cast<const double2*>(A), lda,
                              static_cast<const double2*>(B), ldb, make_double2(be.re, be.im),
                              static_cast<double2*>(C), ldc,
                              reinterpret_cast<double2*>(partials), stream);
    if (rc) return rc;
  } else {
    const size_t smem = sizeof(Tile<T>);
    const dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN, splits);
    auto* kernel = opa == QEB_OP_C ? gemm_kernel<T, true> : gemm_kernel<T, false>;
    const cudaError_t e = qeb::raise_smem_limit(kernel, smem);
    if (e != cudaSuccess) return qeb::cuda_status(e, "cgemm shared-memory limit");
    kernel<<<grid, THREADS, smem, stream>>>(
        M, N, K, kchunk, al, static_cast<const C2<T>*>(A), lda, static_cast<const C2<T>*>(B), ldb,
        be, static_cast<C2<T>*>(C), ldc, partials);
  }
  qeb::count_launches(splits > 1 ? 2 : 1);
  if (splits > 1) {
    const int64_t total = (int64_t)M * N;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 4 * sm_count()) blocks = 4 * sm_count();
    reduce_partials<T><<<blocks, 256, 0, stream>>>(M, N, splits, partials, al, be,
                                                   static_cast<C2<T>*>(C), ldc);
  }
  return qeb::cuda_status(cudaGetLastError(), "zgemm launch");
}

}  // namespace

extern "C" int64_t qeb_zgemm_scratch_bytes(int opa, int M, int N, int K, int precision) {
  if (opa != QEB_OP_C || M <= 0 || N <= 0 || K <= 0) return 0;
  const int64_t elem = (precision == QEB_F64) ? 16 : 8;
  if (N <= kSkinnyMax || M <= kSkinnyMax) {
    const SkinnyC p = skinny_c_plan(M, N, K);
    return p.splits > 1 ? (int64_t)p.splits * p.mb * p.ns * elem : 0;
  }
  const int splits =
      precision == QEB_F64 ? mma_plan(M, N, K, true).splits : choose_splits(M, N, K);
  return splits > 1 ? (int64_t)splits * M * N * elem : 0;
}

extern "C" int qeb_zgemm(int opa, int M, int N, int K, const double* alpha, const void* A,
                         int64_t lda, const void* B, int64_t ldb, const double* beta, void* C,
                         int64_t ldc, void* scratch, int64_t scratch_bytes, void* stream) {
  return gemm<double>(opa, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, scratch, scratch_bytes,
                      static_cast<cudaStream_t>(stream));
}

extern "C" int qeb_cgemm(int opa, int M, int N, int K, const double* alpha, const void* A,
                         int64_t lda, const void* B, int64_t ldb, const double* beta, void* C,
                         int64_t ldc, void* scratch, int64_t scratch_bytes, void* stream) {
  return gemm<float>(opa, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, scratch, scratch_bytes,
                     static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the split-K product C = alpha A^H B + beta C.
//
// For callers that must not allocate device memory themselves, for example a
// host code that runs inside a memory pool it does not own, a process whose
// allocator is reserved for other data, or a driver that forbids cudaMalloc
// between set-up and shutdown.  Instead of caller scratch, the partial K
// tiles live in the fixed array below, which every GPU that loads this
// library holds until the process exits.
namespace {

constexpr int64_t kStaticPartialBytes = 16ll << 20;  // 16 MiB per device
constexpr int kMaxDevices = 64;

__device__ __align__(256) unsigned char g_static_partials[kStaticPartialBytes];

std::mutex g_static_mutex;
void* g_static_address[kMaxDevices] = {nullptr};

// Device address of g_static_partials on the current device.  The host-side
// symbol is only a stand-in, so the address is looked up once per device
// (with that device current) and cached for the life of the process; the
// cache assumes the primary context of each device throughout (a
// cudaDeviceReset or another current context leaves it stale).
int static_partials(void** out) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return qeb::cuda_status(err, "zgemm_static_scratch: cudaGetDevice");
  if (device < 0 || device >= kMaxDevices) {
    qeb::set_error("zgemm_static_scratch: device index %d above %d", device, kMaxDevices);
    return QEB_EUNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (g_static_address[device] == nullptr) {
    void* address = nullptr;
    err = cudaGetSymbolAddress(&address, g_static_partials);
    if (err != cudaSuccess) return qeb::cuda_status(err, "zgemm_static_scratch: cudaGetSymbolAddress");
    g_static_address[device] = address;
  }
  *out = g_static_address[device];
  return QEB_OK;
}

}  // namespace

extern "C" int64_t qeb_zgemm_static_scratch_capacity(void) { return kStaticPartialBytes; }

extern "C" int qeb_zgemm_static_scratch(int M, int N, int K, const double* alpha, const void* A,
                                        int64_t lda, const void* B, int64_t ldb,
                                        const double* beta, void* C, int64_t ldc, void* stream) {
  // Two partial slices of M x N complex128 values must fit the array.
  if (M > 0 && N > 0 && (int64_t)M * N * 16 * 2 > kStaticPartialBytes) {
    qeb::set_error(
        "zgemm_static_scratch: M*N = %lld exceeds the %lld complex128 entries the static "
        "partial buffer allows (M*N*16*2 <= %lld bytes)",
        (long long)M * N, (long long)(kStaticPartialBytes / 32), (long long)kStaticPartialBytes);
    return QEB_EUNSUPPORTED;
  }
  void* scratch = nullptr;
  const int rc = static_partials(&scratch);
  if (rc != QEB_OK) return rc;
  return gemm<double>(QEB_OP_C, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, scratch,
                      kStaticPartialBytes, static_cast<cudaStream_t>(stream));
}
