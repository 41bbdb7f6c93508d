// The Davidson reduced problem in one launch: the lowest pairs of
// H c = e S c for a small Hermitian pencil, and the update of the reduced
// matrices by the rows of a new correction block.
//
// qeb_small_generalized_eigh: as LAPACK zhegv (the reference's solver,
// qepy_pw/diagonalization.py:83-110): S = L L^H, A = L^-1 H L^-H, A z = e z,
// c = L^-H z, here by one block with all matrices in shared memory and the
// Hermitian eigensolve by cyclic Jacobi rotations (Golub and Van Loan, Matrix
// Computations, section 8.5) over a round-robin ordering: a round rotates n / 2
// disjoint index pairs at once, one thread per 2 x 2 block of A.  Bound by the
// latency of the rounds (n - 1 per sweep, six to nine sweeps).  The library
// route (Cholesky, three triangular solves, zheevd) is a chain of about sixty
// launches, which the host of a small cell's SCF could not issue as fast as
// the GPU ran them.
#include "qeb_common.cuh"
#include "../../include/qe_b200.h"

using qeb::C2;
using Z = C2<double>;

namespace {

// Largest n: one thread per 2 x 2 block of A and per row and pair of V.  The
// rounds' latency grows with n and the library's route does not: measured 0.17
// against 0.39 ms at n = 16, 0.39 and 0.51 ms at 32 (host time of a whole
// solve); with more rows than threads, before this split, 1.27 and 1.01 ms at 48.
constexpr int kMaxN = 32;
constexpr int kMaxSweeps = 30;
constexpr int kMaxThreads = (kMaxN / 2) * (kMaxN / 2) + kMaxN * (kMaxN / 2);

__device__ __forceinline__ Z conj(Z a) { return qeb::mk<double>(a.re, -a.im); }
__device__ __forceinline__ Z mul(Z a, Z b) {
  return qeb::mk<double>(fma(a.re, b.re, -(a.im * b.im)), fma(a.re, b.im, a.im * b.re));
}
// a - b c
__device__ __forceinline__ Z sub_mul(Z a, Z b, Z c) {
  return qeb::mk<double>(fma(b.im, c.im, fma(-b.re, c.re, a.re)),
                         fma(-b.im, c.re, fma(-b.re, c.im, a.im)));
}

// Index pair `k` of round `r` of a round-robin over m indices (m even):
// index m - 1 stays, the others rotate.
__device__ __forceinline__ void round_pair(int m, int r, int k, int* p, int* q) {
  const int a = k == 0 ? m - 1 : (r + k) % (m - 1);
  const int b = (r + m - 1 - k) % (m - 1);
  *p = a < b ? a : b;
  *q = a < b ? b : a;
}

struct Rotation {
  double c;
  Z s;  // sine times the phase of the rotated off-diagonal entry
  int p, q;
};

__global__ void __launch_bounds__(kMaxThreads) small_eigh_kernel(
    int n, int roots, const Z* __restrict__ h, int64_t ldh, const Z* __restrict__ s, int64_t lds,
    double* __restrict__ values, Z* __restrict__ vectors, int64_t ldv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m = (n + 1) & ~1, ld = m | 1;  // padded to even; odd row stride
  Z* a = reinterpret_cast<Z*>(smem_raw);
  Z* l = a + m * ld;
  Z* v = l + m * ld;
  Rotation* rot = reinterpret_cast<Rotation*>(v + m * ld);
  __shared__ double diagonal[kMaxN];
  __shared__ int rank_of[kMaxN];
  __shared__ int failed;
  __shared__ double norm2, off2;
  const int tid = threadIdx.x, threads = blockDim.x;
  if (tid == 0) failed = 0;
  for (int i = tid; i < m * m; i += threads) {
    const int r = i / m, c = i - r * m;
    const bool in = r < n && c < n;
    a[r * ld + c] = in ? h[r * ldh + c] : qeb::mk<double>(0, 0);
    l[r * ld + c] = in && c <= r ? s[r * lds + c] : qeb::mk<double>(0, 0);
    v[r * ld + c] = qeb::mk<double>(r == c ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  // Cholesky of the lower triangle, column by column
  for (int k = 0; k < n; ++k) {
    const double pivot = l[k * ld + k].re;
    if (!(pivot > 0.0)) {
      if (tid == 0) failed = k + 1;
      break;  // the same on every thread
    }
    const double inv = 1.0 / sqrt(pivot);
    __syncthreads();
    for (int i = k + tid; i < n; i += threads) l[i * ld + k] = qeb::scale(l[i * ld + k], inv);
    __syncthreads();
    const int rest = n - k - 1;
    for (int t = tid; t < rest * rest; t += threads) {
      const int i = k + 1 + t / rest, j = k + 1 + t % rest;
      if (j <= i) l[i * ld + j] = sub_mul(l[i * ld + j], l[i * ld + k], conj(l[j * ld + k]));
    }
    __syncthreads();
  }
  __syncthreads();
  if (failed) {
    if (tid == 0) values[roots] = failed;
    return;
  }
  // A <- L^-1 A, then A <- A L^-H (row and column substitution)
  for (int k = 0; k < n; ++k) {
    const double inv = 1.0 / l[k * ld + k].re;
    for (int c = tid; c < n; c += threads) a[k * ld + c] = qeb::scale(a[k * ld + c], inv);
    __syncthreads();
    for (int t = tid; t < (n - k - 1) * n; t += threads) {
      const int i = k + 1 + t / n, c = t % n;
      a[i * ld + c] = sub_mul(a[i * ld + c], l[i * ld + k], a[k * ld + c]);
    }
    __syncthreads();
  }
  for (int k = 0; k < n; ++k) {
    const double inv = 1.0 / l[k * ld + k].re;
    for (int r = tid; r < n; r += threads) a[r * ld + k] = qeb::scale(a[r * ld + k], inv);
    __syncthreads();
    for (int t = tid; t < (n - k - 1) * n; t += threads) {
      const int j = k + 1 + t / n, r = t % n;
      a[r * ld + j] = sub_mul(a[r * ld + j], conj(l[j * ld + k]), a[r * ld + k]);
    }
    __syncthreads();
  }
  // Hermitian part
  for (int t = tid; t < n * n; t += threads) {
    const int i = t / n, j = t % n;
    if (j < i) {
      const Z x = a[i * ld + j], y = a[j * ld + i];
      const Z w = qeb::mk<double>(0.5 * (x.re + y.re), 0.5 * (x.im - y.im));
      a[i * ld + j] = w;
      a[j * ld + i] = conj(w);
    } else if (j == i) {
      a[i * ld + i].im = 0.0;
    }
  }
  __syncthreads();
  const int pairs = m / 2, blocks = pairs * pairs;
  // this thread's part of every round: the 2 x 2 block (ki, kj) of A, or row
  // `row` of V for pair ki
  const int ki = tid < blocks ? tid / pairs : (tid - blocks) / m;
  const int kj = tid - ki * pairs, row = tid - blocks - ki * m;
  bool converged = false;
  for (int sweep = 0; sweep < kMaxSweeps; ++sweep) {
    // off-diagonal against the whole: below n eps the eigenvalues stand
    if (tid < 32) {
      double off = 0.0, all = 0.0;
      for (int i = 0; i < n; ++i)
        for (int j = tid; j < n; j += 32) {
          const Z x = a[i * ld + j];
          const double w = x.re * x.re + x.im * x.im;
          all += w;
          if (i != j) off += w;
        }
      for (int o = 16; o > 0; o >>= 1) {
        off += __shfl_xor_sync(0xffffffffu, off, o);
        all += __shfl_xor_sync(0xffffffffu, all, o);
      }
      if (tid == 0) {
        off2 = off;
        norm2 = all;
      }
    }
    __syncthreads();
    // (squares outside the exponent range, infinities, NaN: not for this kernel)
    if (!(norm2 > 1.0e-250 && norm2 < 1.0e250)) break;
    converged = off2 <= 1.0e-31 * norm2;  // the same on every thread
    if (converged) break;
    for (int round = 0; round < m - 1; ++round) {
      if (tid < pairs) {
        Rotation r = {1.0, qeb::mk<double>(0, 0), 0, 0};
        round_pair(m, round, tid, &r.p, &r.q);
        const Z b = a[r.p * ld + r.q];
        const double w = b.re * b.re + b.im * b.im;
        if (w > 1.0e-300) {
          // tan of the angle: 2 |b| / (d +- sqrt(d^2 + 4 |b|^2)), d = a_qq - a_pp
          const double d = a[r.q * ld + r.q].re - a[r.p * ld + r.p].re;
          const double inv = rsqrt(w), root = sqrt(fma(d, d, 4.0 * w));
          const double t = copysign(2.0 * w * inv, d) / (fabs(d) + root);
          r.c = rsqrt(fma(t, t, 1.0));
          r.s = qeb::scale(b, t * r.c * inv);
        }
        rot[tid] = r;
      }
      __syncthreads();
      // A <- J^H A J per 2 x 2 block; V <- V J per row and pair
      if (tid < blocks) {
        const Rotation ri = rot[ki], rj = rot[kj];
        Z* top = a + ri.p * ld;
        Z* bottom = a + ri.q * ld;
        const Z pp = top[rj.p], pq = top[rj.q], qp = bottom[rj.p], qq = bottom[rj.q];
        // columns: x_p = c u_p - conj(s) u_q, x_q = s u_p + c u_q
        const Z cpp = sub_mul(qeb::scale(pp, rj.c), conj(rj.s), pq);
        const Z cpq = qeb::scale(pq, rj.c) + mul(rj.s, pp);
        const Z cqp = sub_mul(qeb::scale(qp, rj.c), conj(rj.s), qq);
        const Z cqq = qeb::scale(qq, rj.c) + mul(rj.s, qp);
        // rows: the conjugates
        Z npp = sub_mul(qeb::scale(cpp, ri.c), ri.s, cqp);
        Z npq = sub_mul(qeb::scale(cpq, ri.c), ri.s, cqq);
        Z nqp = qeb::scale(cqp, ri.c) + mul(conj(ri.s), cpp);
        Z nqq = qeb::scale(cqq, ri.c) + mul(conj(ri.s), cpq);
        if (ki == kj) {  // the rotated pair: exactly diagonal
          npq = nqp = qeb::mk<double>(0, 0);
          npp.im = nqq.im = 0.0;
        }
        top[rj.p] = npp;
        top[rj.q] = npq;
        bottom[rj.p] = nqp;
        bottom[rj.q] = nqq;
      } else if (ki < pairs) {
        const Rotation r = rot[ki];
        const Z x = v[row * ld + r.p], y = v[row * ld + r.q];
        v[row * ld + r.p] = sub_mul(qeb::scale(x, r.c), conj(r.s), y);
        v[row * ld + r.q] = qeb::scale(y, r.c) + mul(r.s, x);
      }
      __syncthreads();
    }
  }
  if (!converged) {
    if (tid == 0) values[roots] = -1.0;
    return;
  }
  // ascending order (ties by index)
  for (int i = tid; i < n; i += threads) diagonal[i] = a[i * ld + i].re;
  __syncthreads();
  for (int i = tid; i < n; i += threads) {
    int rank = 0;
    for (int j = 0; j < n; ++j)
      rank += diagonal[j] < diagonal[i] || (diagonal[j] == diagonal[i] && j < i);
    rank_of[rank] = i;
  }
  __syncthreads();
  // the wanted vectors into A, then L^-H by back substitution
  for (int t = tid; t < n * roots; t += threads) {
    const int r = t / roots, c = t - r * roots;
    a[r * ld + c] = v[r * ld + rank_of[c]];
  }
  __syncthreads();
  for (int k = n - 1; k >= 0; --k) {
    const double inv = 1.0 / l[k * ld + k].re;
    for (int c = tid; c < roots; c += threads) a[k * ld + c] = qeb::scale(a[k * ld + c], inv);
    __syncthreads();
    for (int t = tid; t < k * roots; t += threads) {
      const int i = t / roots, c = t - i * roots;
      a[i * ld + c] = sub_mul(a[i * ld + c], conj(l[k * ld + i]), a[k * ld + c]);
    }
    __syncthreads();
  }
  for (int i = tid; i < roots; i += threads) values[i] = diagonal[rank_of[i]];
  for (int t = tid; t < n * roots; t += threads) {
    const int c = t / n, r = t - c * n;
    vectors[r + c * ldv] = a[r * ld + c];
  }
  if (tid == 0) values[roots] = 0.0;
}

size_t small_smem(int n) {
  const int m = (n + 1) & ~1, ld = m | 1;
  return sizeof(Z) * 3 * (size_t)m * ld + sizeof(Rotation) * (m / 2);
}

// New rows [first, active) of the reduced matrices (row-major, ld) from the
// products new^H [H V, V] (column-major, `rows` x active): the Hermitian
// counterparts in the columns above them, the new diagonal block averaged with
// its conjugate transpose.  lam: h_rows += s_rows lam on the first nlam
// columns (refined Davidson), or null.
template <typename T>
__global__ void update_reduced_kernel(int first, int active, const C2<T>* __restrict__ h_rows,
                                      int64_t ldh, const C2<T>* __restrict__ s_rows, int64_t lds,
                                      const double* __restrict__ lam, int nlam,
                                      Z* __restrict__ projected, Z* __restrict__ overlap,
                                      int64_t ld) {
  const int64_t rows = active - first;
  auto entry = [&](const C2<T>* m, int64_t ldm, int64_t i, int64_t j, bool shifted) {
    const C2<T> x = m[i + j * ldm];
    Z z = qeb::mk<double>(x.re, x.im);
    if (shifted && j < nlam) {
      const C2<T> w = s_rows[i + j * lds];
      z.re = fma((double)w.re, lam[j], z.re);
      z.im = fma((double)w.im, lam[j], z.im);
    }
    return z;
  };
  const bool shifted = lam != nullptr;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < rows * active;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = t / rows, i = t - j * rows;
    Z hv = entry(h_rows, ldh, i, j, shifted), sv = entry(s_rows, lds, i, j, false);
    if (j >= first) {
      const Z hc = entry(h_rows, ldh, j - first, first + i, shifted);
      const Z sc = entry(s_rows, lds, j - first, first + i, false);
      hv = qeb::mk<double>(0.5 * (hv.re + hc.re), 0.5 * (hv.im - hc.im));
      sv = qeb::mk<double>(0.5 * (sv.re + sc.re), 0.5 * (sv.im - sc.im));
    } else {
      projected[j * ld + first + i] = conj(hv);
      overlap[j * ld + first + i] = conj(sv);
    }
    projected[(first + i) * ld + j] = hv;
    overlap[(first + i) * ld + j] = sv;
  }
}

}  // namespace

extern "C" int qeb_small_eigh_max(void) { return kMaxN; }

extern "C" int qeb_small_generalized_eigh(int n, int roots, const void* h, int64_t ldh,
                                          const void* s, int64_t lds, double* values,
                                          void* vectors, int64_t ldv, void* stream) {
  if (n < 1 || roots < 1 || roots > n || ldh < n || lds < n || ldv < n || h == nullptr ||
      s == nullptr || values == nullptr || vectors == nullptr) {
    qeb::set_error("small_generalized_eigh: invalid arguments (n=%d roots=%d)", n, roots);
    return QEB_EINVAL;
  }
  if (n > kMaxN) {
    qeb::set_error("small_generalized_eigh: n = %d exceeds %d", n, kMaxN);
    return QEB_EUNSUPPORTED;
  }
  const size_t smem = small_smem(n);
  cudaError_t e = qeb::raise_smem_limit(small_eigh_kernel, smem);
  if (e != cudaSuccess) return qeb::cuda_status(e, "small_generalized_eigh shared memory");
  const int m = (n + 1) & ~1, threads = (m / 2 * (m / 2) + m * (m / 2) + 31) / 32 * 32;
  small_eigh_kernel<<<1, threads, smem, static_cast<cudaStream_t>(stream)>>>(
      n, roots, static_cast<const Z*>(h), ldh, static_cast<const Z*>(s), lds, values,
      static_cast<Z*>(vectors), ldv);
  qeb::count_launches(1);
  return qeb::cuda_status(cudaGetLastError(), "small_generalized_eigh launch");
}

extern "C" int qeb_update_reduced(int precision, int first, int active, const void* h_rows,
                                  int64_t ldh, const void* s_rows, int64_t lds, const double* lam,
                                  int nlam, void* projected, void* overlap, int64_t ld,
                                  void* stream) {
  const int64_t rows = (int64_t)active - first;
  if (first < 0 || rows < 0 || ldh < rows || lds < rows || ld < active || nlam < 0 ||
      (rows > 0 && (h_rows == nullptr || s_rows == nullptr || projected == nullptr ||
                    overlap == nullptr))) {
    qeb::set_error("update_reduced: invalid arguments (first=%d active=%d)", first, active);
    return QEB_EINVAL;
  }
  if (rows == 0) return QEB_OK;
  const int64_t want = (rows * active + 255) / 256;
  const int blocks = (int)(want < 148 * 8 ? want : 148 * 8);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (precision == QEB_F64) {
    update_reduced_kernel<double><<<blocks, 256, 0, st>>>(
        first, active, static_cast<const Z*>(h_rows), ldh, static_cast<const Z*>(s_rows), lds, lam,
        nlam, static_cast<Z*>(projected), static_cast<Z*>(overlap), ld);
  } else if (precision == QEB_F32) {
    update_reduced_kernel<float><<<blocks, 256, 0, st>>>(
        first, active, static_cast<const C2<float>*>(h_rows), ldh,
        static_cast<const C2<float>*>(s_rows), lds, lam, nlam, static_cast<Z*>(projected),
        static_cast<Z*>(overlap), ld);
  } else {
    qeb::set_error("update_reduced: unknown precision %d", precision);
    return QEB_EINVAL;
  }
  qeb::count_launches(1);
  return qeb::cuda_status(cudaGetLastError(), "update_reduced launch");
}
