// Plane-pass kernels of one precision and their launch (included by
// local_plane_f32.cu and local_plane_f64.cu, which instantiate it).
#pragma once

#include <algorithm>
#include <cstdlib>

#include "line_lengths.cuh"
#include "local_lines.cuh"
#include "../../include/qe_b200.h"

namespace qeb {
namespace lines {

template <typename T, class P>
constexpr PlaneBounds bounds_of() {
  if constexpr (P::kStatic)
    return plane_bounds<T>(P::x1, P::x2, P::y1, P::y2, true);
  else
    return plane_bounds<T>(16, 16, 16, 16, false);
}

template <typename T, int MODE, class P>
__global__ void __launch_bounds__((bounds_of<T, P>().threads), (bounds_of<T, P>().blocks)) plane_kernel(
    const __grid_constant__ KBatch<T> kb, const __grid_constant__ P g, int nz, const C2<T>* tw_x,
    const C2<T>* tw_y, const T* potential, const __grid_constant__ DensityTarget rho) {
  const KDesc<T>& d = kb.k[blockIdx.z];
  if ((int)blockIdx.y >= d.nb) return;
  plane_body<T, MODE, P>(d, g, nz, tw_x, tw_y, potential, rho, blockIdx.x, blockIdx.y);
}

// nb == 0: only raise the kernel's shared-memory limit (plan creation, so that
// a launch makes no other call and may be captured first thing).
template <typename T, int MODE, class P>
int launch_one(const KBatch<T>& kb, const P& g, int nz, int nk, int nb, const C2<T>* tw_x,
               const C2<T>* tw_y, const T* potential, const DensityTarget& rho, cudaStream_t s) {
  const size_t smem = plane_smem<T>(g.x1, g.x2, g.y1, g.y2, g.rows, g.columns);
  if (nb == 0)
    return cuda_status(raise_smem_limit(plane_kernel<T, MODE, P>, smem),
                       "plane pass shared memory");
  const int threads = plane_threads<T>(g, (int64_t)nz * nb * nk);
  plane_kernel<T, MODE, P><<<dim3(nz, nb, nk), threads, smem, s>>>(kb, g, nz, tw_x, tw_y,
                                                                   potential, rho);
  return QEB_OK;
}

template <typename T, int MODE, int N1, int N2, int K>
int launch_static(const KBatch<T>& kb, const qeb_local_plan* p, int nk, int nb, const C2<T>* tw_x,
                  const C2<T>* tw_y, const T* potential, const DensityTarget& rho,
                  cudaStream_t s) {
  using P = StaticPlane<N1, N2, K, plane_columns<T>(N1, N2, N1, N2, 2 * K * N2, true)>;
  return launch_one<T, MODE, P>(kb, P{}, p->nz, nk, nb, tw_x, tw_y, potential, rho, s);
}

template <typename T, int MODE>
int launch_plane(const KBatch<T>& kb, const qeb_local_plan* p, int nk, int nb,
                 const T* potential, const DensityTarget& rho, cudaStream_t s) {
  const C2<T>* tw_x = tw_at<T>(p, 0);
  const C2<T>* tw_y = tw_at<T>(p, 1);
#define QEB_CASE(n, a, b, k1, k2)                                                             \
  if constexpr (plane_columns<T>(a, b, a, b, 2 * k1 * b, true) > 0) {                               \
    if (p->nx == n && p->line_k == k1)                                                        \
      return launch_static<T, MODE, a, b, k1>(kb, p, nk, nb, tw_x, tw_y, potential, rho, s);  \
  }                                                                                           \
  if constexpr (k2 > k1 && plane_columns<T>(a, b, a, b, 2 * k2 * b, true) > 0) {                    \
    if (p->nx == n && p->line_k == k2)                                                        \
      return launch_static<T, MODE, a, b, k2>(kb, p, nk, nb, tw_x, tw_y, potential, rho, s);  \
  }
  QEB_LINE_LENGTHS(QEB_CASE)
#undef QEB_CASE
  int rows = 0;
  for (int k = 0; k < nk; ++k) rows = std::max(rows, kb.k[k].rows);
  const RuntimePlane g = runtime_plane<T>(p, rows);
  return launch_one<T, MODE, RuntimePlane>(kb, g, p->nz, nk, nb, tw_x, tw_y, potential, rho, s);
}

}  // namespace lines
}  // namespace qeb
