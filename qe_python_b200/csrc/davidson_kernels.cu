// Davidson column kernels: QE g_psi preconditioner, column norms, inner
// products, normalisation and residual formation.
//
// Reference: qepy_pw/_native_fft.pyx qe_precondition (:852-899),
// column_squared_norms (:1153-1190), subtract_band_energies (:1193-1234),
// column_inner_products (:1237-1291), column_diagonal_expectations
// (:1294-1343), normalize_selected_columns (:1495-1530).
// Column reductions accumulate in FP64 whatever the vector precision, in a
// fixed order, so they are deterministic.
#include <type_traits>

#include "qeb_common.cuh"
#include "../../include/qe_b200.h"

using qeb::C2;

namespace {

constexpr int kReduceThreads = 256;
constexpr int kMaxCluster = 8;

// V consecutive values: one 16-byte access for two complex64 or one
// complex128 value.
template <typename T, int V>
__device__ __forceinline__ void load_run(C2<T> (&v)[V], const C2<T>* p) {
  if constexpr (V == 2) {
    const float4 w = *reinterpret_cast<const float4*>(p);
    v[0] = qeb::mk<T>(w.x, w.y);
    v[1] = qeb::mk<T>(w.z, w.w);
  } else {
    v[0] = p[0];
  }
}
template <typename T, int V>
__device__ __forceinline__ void store_run(C2<T>* p, const C2<T> (&v)[V]) {
  if constexpr (V == 2)
    *reinterpret_cast<float4*>(p) = make_float4(v[0].re, v[0].im, v[1].re, v[1].im);
  else
    p[0] = v[0];
}

__device__ __forceinline__ double block_sum(double v, double* shared) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (lane == 0) shared[warp] = v;
  __syncthreads();
  double total = 0.0;
  if (threadIdx.x == 0) {
    for (int w = 0; w < (int)(blockDim.x / 32); ++w) total += shared[w];
  }
  __syncthreads();
  return total;
}

// Not the .aligned form, which wants every warp converged: thread 0 comes here
// from branches that it alone takes.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The double at `p` of this block's shared memory as block `rank` holds it.
__device__ __forceinline__ double cluster_read(const double* p, unsigned rank) {
  const unsigned local = (unsigned)__cvta_generic_to_shared(p);
  unsigned remote;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote));
  return v;
}

// mode 0: sum |v|^2; mode 1: sum diag |v|^2; mode 2: sum conj(l) r (complex).
// A cluster of `parts` blocks shares a column: each sums a run of its rows and
// the first adds the partial sums in block order through distributed shared
// memory, so there is neither scratch nor a second launch.  Bound by the
// reads: one block per column left 131 blocks on 148 SMs for the corrections
// of the 216-atom cell (80 725 x 131 complex64: 57 us, 1.5 TB/s).  With the
// column kernels below: g_psi, norms and normalisation of that block 0.173 ->
// 0.087 ms.
template <typename T, int MODE, int V>
__global__ void __launch_bounds__(kReduceThreads) column_reduce(
    int64_t rows, int parts, int64_t part_rows, const C2<T>* __restrict__ left, int64_t ldl,
    const C2<T>* __restrict__ right, int64_t ldr, const double* __restrict__ diag,
    double* __restrict__ out) {
  __shared__ double shared[2][32];
  __shared__ double sums[2];
  const int64_t col = blockIdx.x / parts;
  const int part = (int)(blockIdx.x - col * parts);
  const int64_t first = part * part_rows, last = min(rows, first + part_rows);
  const C2<T>* l = left + col * ldl;
  const C2<T>* r = MODE == 2 ? right + col * ldr : nullptr;
  double re2[2] = {0.0, 0.0}, im2[2] = {0.0, 0.0};  // of the even and the odd runs
  auto add = [&](int c, int64_t g, C2<T> a, C2<T> b) {
    if (MODE == 2) {
      re2[c] += (double)a.re * b.re + (double)a.im * b.im;
      im2[c] += (double)a.re * b.im - (double)a.im * b.re;
    } else {
      const double m = (double)a.re * a.re + (double)a.im * a.im;
      re2[c] += (MODE == 1) ? diag[g] * m : m;
    }
  };
  constexpr int kStep = kReduceThreads * V;
  int64_t g = first + threadIdx.x * V;
  // four loads in flight per thread, two from each operand of an inner product
  // (four from each took 160 us on 50 000 x 480 complex128, two 118); two sums,
  // half the chain of additions, make up for the longer parts
  constexpr int kRuns = MODE == 2 ? 2 : 4;
  for (; g + (kRuns - 1) * kStep + V <= last; g += kRuns * kStep) {
    C2<T> a[kRuns][V], b[kRuns][V];
#pragma unroll
    for (int u = 0; u < kRuns; ++u) {
      load_run<T, V>(a[u], l + g + u * kStep);
      if constexpr (MODE == 2) load_run<T, V>(b[u], r + g + u * kStep);
    }
#pragma unroll
    for (int u = 0; u < kRuns; ++u)
#pragma unroll
      for (int v = 0; v < V; ++v)
        add(u & 1, g + u * kStep + v, a[u][v], MODE == 2 ? b[u][v] : a[u][v]);
  }
  for (; g < last; g += kStep)
    for (int v = 0; v < V && g + v < last; ++v)
      add(0, g + v, l[g + v], MODE == 2 ? r[g + v] : l[g + v]);
  double re = re2[0] + re2[1], im = im2[0] + im2[1];
  re = block_sum(re, shared[0]);
  if (MODE == 2) im = block_sum(im, shared[1]);
  if (parts > 1) {
    if (threadIdx.x == 0) {
      sums[0] = re;
      sums[1] = im;
    }
    cluster_sync();
    if (part == 0 && threadIdx.x == 0) {
      for (int p = 1; p < parts; ++p) {
        re += cluster_read(&sums[0], p);
        if (MODE == 2) im += cluster_read(&sums[1], p);
      }
    }
    cluster_sync();  // the other blocks' shared memory stays until it has been read
  }
  if (part == 0 && threadIdx.x == 0) {
    if (MODE == 2) {
      out[2 * col] = re;
      out[2 * col + 1] = im;
    } else {
      out[col] = re;
    }
  }
}

// Column kernels: a block handles kRunRows consecutive rows of one column
// (blockIdx.x = column * blocks per column + row block: one division per
// block), in 16-byte runs where the columns allow it.
constexpr int kRunThreads = 256, kRunRows = 1024;

template <typename T, int V, class Fn>
__device__ __forceinline__ void for_runs(int64_t rows, int64_t first, Fn&& fn) {
  const int64_t last = min(rows, first + kRunRows);
#pragma unroll
  for (int u = 0; u < kRunRows / (kRunThreads * V); ++u) {
    const int64_t g = first + (u * kRunThreads + threadIdx.x) * V;
    if (g + V <= last) fn(g, std::integral_constant<int, V>{});
    else
      for (int64_t h = g; h < last; ++h) fn(h, std::integral_constant<int, 1>{});
  }
}

// x = 2 (H_GG - e_b) [Ry], d = (1 + x + sqrt(1 + (x - 1)^2)) / 2, out = 2 r / d,
// in FP64 whatever the vectors' precision.
template <typename T, int V>
__global__ void __launch_bounds__(kRunThreads) precondition_kernel(
    int64_t rows, int64_t blocks, const C2<T>* __restrict__ r, int64_t ldr,
    const double* __restrict__ e, const double* __restrict__ diag, C2<T>* __restrict__ out,
    int64_t ldo) {
  const int64_t b = blockIdx.x / blocks, first = (blockIdx.x - b * blocks) * kRunRows;
  const double eb = e[b];
  const C2<T>* src = r + b * ldr;
  C2<T>* dst = out + b * ldo;
  for_runs<T, V>(rows, first, [&](int64_t g, auto width) {
    constexpr int W = decltype(width)::value;
    C2<T> v[W];
    load_run<T, W>(v, src + g);
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const double x = 2.0 * (diag[g + i] - eb);
      const double d = 0.5 * (1.0 + x + sqrt(1.0 + (x - 1.0) * (x - 1.0)));
      const double s = 2.0 / d;
      v[i] = qeb::mk<T>((T)(s * (double)v[i].re), (T)(s * (double)v[i].im));
    }
    store_run<T, W>(dst + g, v);
  });
}

// out[:, j] = v[:, sel[j]] / sqrt(norms2[sel[j]])
template <typename T, int V>
__global__ void __launch_bounds__(kRunThreads) normalize_kernel(
    int64_t rows, int64_t blocks, const C2<T>* __restrict__ v, int64_t ldv,
    const double* __restrict__ norms2, const int64_t* __restrict__ sel, C2<T>* __restrict__ out,
    int64_t ldo) {
  const int64_t j = blockIdx.x / blocks, first = (blockIdx.x - j * blocks) * kRunRows;
  const int64_t col = sel ? sel[j] : j;
  const double s = 1.0 / sqrt(norms2[col]);
  const C2<T>* src = v + col * ldv;
  C2<T>* dst = out + j * ldo;
  for_runs<T, V>(rows, first, [&](int64_t g, auto width) {
    constexpr int W = decltype(width)::value;
    C2<T> a[W];
    load_run<T, W>(a, src + g);
#pragma unroll
    for (int i = 0; i < W; ++i)
      a[i] = qeb::mk<T>((T)(s * (double)a[i].re), (T)(s * (double)a[i].im));
    store_run<T, W>(dst + g, a);
  });
}

// r[:, b] -= e[b] v[:, b]
template <typename T, int V>
__global__ void __launch_bounds__(kRunThreads) subtract_kernel(
    int64_t rows, int64_t blocks, C2<T>* __restrict__ r, int64_t ldr, const C2<T>* __restrict__ v,
    int64_t ldv, const double* __restrict__ e) {
  const int64_t b = blockIdx.x / blocks, first = (blockIdx.x - b * blocks) * kRunRows;
  const T eb = (T)e[b];
  const C2<T>* src = v + b * ldv;
  C2<T>* dst = r + b * ldr;
  for_runs<T, V>(rows, first, [&](int64_t g, auto width) {
    constexpr int W = decltype(width)::value;
    C2<T> a[W], t[W];
    load_run<T, W>(a, src + g);
    load_run<T, W>(t, dst + g);
#pragma unroll
    for (int i = 0; i < W; ++i) {
      t[i].re -= eb * a[i].re;
      t[i].im -= eb * a[i].im;
    }
    store_run<T, W>(dst + g, t);
  });
}

// Whether complex64 columns start on 16-byte boundaries.
bool wide(const void* p, int64_t ld) {
  return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 2 == 0;
}

// Grid of the column kernels, or a negative status when it is too large.
int64_t run_blocks(int64_t rows, int64_t cols, int64_t* per_column) {
  *per_column = (rows + kRunRows - 1) / kRunRows;
  const int64_t total = *per_column * cols;
  if (total > 0x7fffffff) {
    qeb::set_error("column kernel: matrix too large for one launch");
    return QEB_EUNSUPPORTED;
  }
  return total;
}

template <typename T, int MODE>
int launch_reduce(int64_t rows, int64_t cols, const void* left, int64_t ldl, const void* right,
                  int64_t ldr, const double* diag, double* out, cudaStream_t stream) {
  // blocks per column: about four per SM in all for complex64 values, three for
  // complex128, each with at least 4096 rows, or 8192 once there are three per SM.
  // Columns that fill the GPU alone stay whole (squared norms, one block a column
  // against two: 80 725 x 480 complex128 97 and 109 us, 11 019 x 480 complex64 8.6
  // and 10.6); fewer gain by the split (80 725 x 131 complex128, one and four, 57 and 31).
  constexpr int kFill = (sizeof(T) == 4 ? 4 : 3) * 148;
  int parts = 1;
  while (parts < kMaxCluster && cols * parts < kFill &&
         rows / (2 * parts) >= (cols * parts < 3 * 148 ? 4096 : 8192))
    parts *= 2;
  int64_t part_rows = (rows + parts - 1) / parts;
  part_rows = (part_rows + 1) & ~int64_t(1);  // every part starts on a whole run
  if (cols * parts > 0x7fffffff) {
    qeb::set_error("column reduction: too many columns for one launch");
    return QEB_EUNSUPPORTED;
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)(cols * parts));
  config.blockDim = dim3(kReduceThreads);
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeClusterDimension;
  attribute.val.clusterDim.x = (unsigned)parts;
  attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  const C2<T>* l = static_cast<const C2<T>*>(left);
  const C2<T>* r = static_cast<const C2<T>*>(right);
  const bool runs = sizeof(T) == 4 && wide(left, ldl) && (MODE != 2 || wide(right, ldr));
  cudaError_t e;
  if constexpr (sizeof(T) == 4) {
    e = runs ? cudaLaunchKernelEx(&config, column_reduce<T, MODE, 2>, rows, parts, part_rows, l, ldl,
                                  r, ldr, diag, out)
             : cudaLaunchKernelEx(&config, column_reduce<T, MODE, 1>, rows, parts, part_rows, l, ldl,
                                  r, ldr, diag, out);
  } else {
    e = cudaLaunchKernelEx(&config, column_reduce<T, MODE, 1>, rows, parts, part_rows, l, ldl, r,
                           ldr, diag, out);
  }
  qeb::count_launches(1);
  return qeb::cuda_status(e, "column reduction");
}

int grid_for(int64_t total) {
  int64_t blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  return (int)(blocks < 1 ? 1 : blocks);
}

bool bad(int64_t rows, int64_t cols, int64_t ld) { return rows < 0 || cols < 0 || ld < rows; }

}  // namespace

#define QEB_DISPATCH(prec, call_f64, call_f32)                      \
  do {                                                              \
    if ((prec) == QEB_F64) {                                        \
      call_f64;                                                     \
    } else if ((prec) == QEB_F32) {                                 \
      call_f32;                                                     \
    } else {                                                        \
      qeb::set_error("unknown precision %d", (int)(prec));          \
      return QEB_EINVAL;                                            \
    }                                                               \
  } while (0)

extern "C" int qeb_column_squared_norms(int precision, int64_t rows, int64_t cols,
                                        const void* v, int64_t ld, double* out, void* stream) {
  if (bad(rows, cols, ld) || (cols > 0 && (v == nullptr || out == nullptr))) {
    qeb::set_error("column_squared_norms: invalid arguments");
    return QEB_EINVAL;
  }
  if (cols == 0) return QEB_OK;
  int rc = QEB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  QEB_DISPATCH(precision,
               (rc = launch_reduce<double, 0>(rows, cols, v, ld, nullptr, 0, nullptr, out, s)),
               (rc = launch_reduce<float, 0>(rows, cols, v, ld, nullptr, 0, nullptr, out, s)));
  return rc;
}

extern "C" int qeb_column_diagonal_expectations(int precision, int64_t rows, int64_t cols,
                                                const void* v, int64_t ld, const double* diag,
                                                double* out, void* stream) {
  if (bad(rows, cols, ld) || (cols > 0 && (v == nullptr || out == nullptr || diag == nullptr))) {
    qeb::set_error("column_diagonal_expectations: invalid arguments");
    return QEB_EINVAL;
  }
  if (cols == 0) return QEB_OK;
  int rc = QEB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  QEB_DISPATCH(precision,
               (rc = launch_reduce<double, 1>(rows, cols, v, ld, nullptr, 0, diag, out, s)),
               (rc = launch_reduce<float, 1>(rows, cols, v, ld, nullptr, 0, diag, out, s)));
  return rc;
}

extern "C" int qeb_column_inner_products(int precision, int64_t rows, int64_t cols,
                                         const void* left, int64_t ldl, const void* right,
                                         int64_t ldr, double* out_complex, void* stream) {
  if (bad(rows, cols, ldl) || ldr < rows ||
      (cols > 0 && (left == nullptr || right == nullptr || out_complex == nullptr))) {
    qeb::set_error("column_inner_products: invalid arguments");
    return QEB_EINVAL;
  }
  if (cols == 0) return QEB_OK;
  int rc = QEB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  QEB_DISPATCH(precision,
               (rc = launch_reduce<double, 2>(rows, cols, left, ldl, right, ldr, nullptr,
                                              out_complex, s)),
               (rc = launch_reduce<float, 2>(rows, cols, left, ldl, right, ldr, nullptr,
                                             out_complex, s)));
  return rc;
}

extern "C" int qeb_precondition(int precision, int64_t rows, int64_t cols, const void* residuals,
                                int64_t ldr, const double* eigenvalues, const double* diagonal,
                                void* out, int64_t ldo, void* stream) {
  if (bad(rows, cols, ldr) || ldo < rows ||
      (cols > 0 && (!residuals || !eigenvalues || !diagonal || !out))) {
    qeb::set_error("precondition: invalid arguments");
    return QEB_EINVAL;
  }
  if (cols == 0 || rows == 0) return QEB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int64_t per_column = 0;
  const int64_t total = run_blocks(rows, cols, &per_column);
  if (total < 0) return (int)total;
  const unsigned blocks = (unsigned)total;
  const bool runs = wide(residuals, ldr) && wide(out, ldo);
  QEB_DISPATCH(precision,
               (precondition_kernel<double, 1><<<blocks, kRunThreads, 0, s>>>(
                   rows, per_column, static_cast<const C2<double>*>(residuals), ldr, eigenvalues,
                   diagonal, static_cast<C2<double>*>(out), ldo)),
               (runs ? precondition_kernel<float, 2><<<blocks, kRunThreads, 0, s>>>(
                   rows, per_column, static_cast<const C2<float>*>(residuals), ldr, eigenvalues,
                   diagonal, static_cast<C2<float>*>(out), ldo)
                     : precondition_kernel<float, 1><<<blocks, kRunThreads, 0, s>>>(
                   rows, per_column, static_cast<const C2<float>*>(residuals), ldr, eigenvalues,
                   diagonal, static_cast<C2<float>*>(out), ldo)));
  qeb::count_launches(1);
  return qeb::cuda_status(cudaGetLastError(), "precondition");
}

extern "C" int qeb_normalize_columns(int precision, int64_t rows, int64_t cols, const void* v,
                                     int64_t ldv, const double* norms2, const int64_t* selected,
                                     void* out, int64_t ldo, void* stream) {
  if (rows < 0 || cols < 0 || ldo < rows || ldv < rows ||
      (cols > 0 && (!v || !norms2 || !out))) {
    qeb::set_error("normalize_columns: invalid arguments");
    return QEB_EINVAL;
  }
  if (cols == 0 || rows == 0) return QEB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int64_t per_column = 0;
  const int64_t total = run_blocks(rows, cols, &per_column);
  if (total < 0) return (int)total;
  const unsigned blocks = (unsigned)total;
  const bool runs = wide(v, ldv) && wide(out, ldo);
  QEB_DISPATCH(precision,
               (normalize_kernel<double, 1><<<blocks, kRunThreads, 0, s>>>(
                   rows, per_column, static_cast<const C2<double>*>(v), ldv, norms2, selected,
                   static_cast<C2<double>*>(out), ldo)),
               (runs ? normalize_kernel<float, 2><<<blocks, kRunThreads, 0, s>>>(
                   rows, per_column, static_cast<const C2<float>*>(v), ldv, norms2, selected,
                   static_cast<C2<float>*>(out), ldo)
                     : normalize_kernel<float, 1><<<blocks, kRunThreads, 0, s>>>(
                   rows, per_column, static_cast<const C2<float>*>(v), ldv, norms2, selected,
                   static_cast<C2<float>*>(out), ldo)));
  qeb::count_launches(1);
  return qeb::cuda_status(cudaGetLastError(), "normalize_columns");
}

extern "C" int qeb_subtract_band_energies(int precision, int64_t rows, int64_t cols,
                                          void* residual, int64_t ldr, const void* v,
                                          int64_t ldv, const double* energies, void* stream) {
  if (bad(rows, cols, ldr) || ldv < rows || (cols > 0 && (!residual || !v || !energies))) {
    qeb::set_error("subtract_band_energies: invalid arguments");
    return QEB_EINVAL;
  }
  if (cols == 0 || rows == 0) return QEB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int64_t per_column = 0;
  const int64_t total = run_blocks(rows, cols, &per_column);
  if (total < 0) return (int)total;
  const unsigned blocks = (unsigned)total;
  const bool runs = wide(residual, ldr) && wide(v, ldv);
  QEB_DISPATCH(precision,
               (subtract_kernel<double, 1><<<blocks, kRunThreads, 0, s>>>(
                   rows, per_column, static_cast<C2<double>*>(residual), ldr,
                   static_cast<const C2<double>*>(v), ldv, energies)),
               (runs ? subtract_kernel<float, 2><<<blocks, kRunThreads, 0, s>>>(
                   rows, per_column, static_cast<C2<float>*>(residual), ldr,
                   static_cast<const C2<float>*>(v), ldv, energies)
                     : subtract_kernel<float, 1><<<blocks, kRunThreads, 0, s>>>(
                   rows, per_column, static_cast<C2<float>*>(residual), ldr,
                   static_cast<const C2<float>*>(v), ldv, energies)));
  qeb::count_launches(1);
  return qeb::cuda_status(cudaGetLastError(), "subtract_band_energies");
}

namespace {

// diag[g] += m * Re sum_i coupled[g, i] conj(beta[g, i])
template <typename T>
__global__ void projector_diagonal_kernel(int64_t rows, int64_t channels,
                                          const C2<T>* __restrict__ coupled, int64_t ldc,
                                          const C2<T>* __restrict__ beta, int64_t ldb,
                                          double multiplicity, double* __restrict__ diag) {
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < rows;
       g += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int64_t i = 0; i < channels; ++i) {
      const C2<T> c = coupled[g + i * ldc], b = beta[g + i * ldb];
      acc += (double)c.re * b.re + (double)c.im * b.im;
    }
    diag[g] += multiplicity * acc;
  }
}

}  // namespace

extern "C" int qeb_accumulate_projector_diagonal(int precision, int64_t rows, int64_t channels,
                                                 const void* coupled, int64_t ldc,
                                                 const void* beta, int64_t ldb,
                                                 double multiplicity, double* diagonal,
                                                 void* stream) {
  if (rows < 0 || channels < 0 || ldc < rows || ldb < rows ||
      (rows > 0 && channels > 0 && (!coupled || !beta || !diagonal))) {
    qeb::set_error("accumulate_projector_diagonal: invalid arguments");
    return QEB_EINVAL;
  }
  if (rows == 0 || channels == 0) return QEB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int blocks = grid_for(rows);
  QEB_DISPATCH(precision,
               (projector_diagonal_kernel<double><<<blocks, 256, 0, s>>>(
                   rows, channels, static_cast<const C2<double>*>(coupled), ldc,
                   static_cast<const C2<double>*>(beta), ldb, multiplicity, diagonal)),
               (projector_diagonal_kernel<float><<<blocks, 256, 0, s>>>(
                   rows, channels, static_cast<const C2<float>*>(coupled), ldc,
                   static_cast<const C2<float>*>(beta), ldb, multiplicity, diagonal)));
  qeb::count_launches(1);
  return qeb::cuda_status(cudaGetLastError(), "accumulate_projector_diagonal");
}
