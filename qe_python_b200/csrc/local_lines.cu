// The z passes of the line transforms and the launch sequence of the local
// H|psi> and the density (local_lines.cuh).
#include <algorithm>
#include <atomic>

#include "line_lengths.cuh"
#include "local_lines.cuh"
#include "../../include/qe_b200.h"

namespace qeb {

// The device word of bounded waits that gave up (tf32_gemm.cu).
int tensor_error_word(int** out);

namespace lines {
namespace {

template <typename T, class Z>
__global__ void __launch_bounds__(kZThreads) z_inverse_kernel(
    const __grid_constant__ KBatch<T> kb, const __grid_constant__ Z g, const C2<T>* tw_z) {
  const KDesc<T>& d = kb.k[blockIdx.z];
  if ((int)blockIdx.x * kSticks >= d.nst || (int)blockIdx.y >= d.nb) return;
  z_inverse_body<T, Z>(d, g, tw_z, blockIdx.x, blockIdx.y);
}

template <typename T, class Z>
__global__ void __launch_bounds__(kZThreads) z_forward_kernel(
    const __grid_constant__ KBatch<T> kb, const __grid_constant__ Z g, const C2<T>* tw_z, T inv_n) {
  const KDesc<T>& d = kb.k[blockIdx.z];
  if ((int)blockIdx.x * kSticks >= d.nst || (int)blockIdx.y >= d.nb) return;
  z_forward_body<T, Z>(d, g, tw_z, inv_n, blockIdx.x, blockIdx.y);
}

// nb == 0: only raise the kernels' shared-memory limits (plan creation).
template <typename T, class Z>
int launch_z(const KBatch<T>& kb, const Z& g, bool inverse, dim3 grid, const C2<T>* tw, T inv_n,
             cudaStream_t s) {
  const size_t smem = sizeof(C2<T>) * ((size_t)kSticks * g.stride + g.nz);
  if (grid.y == 0) {
    cudaError_t e = raise_smem_limit(z_inverse_kernel<T, Z>, smem);
    if (e == cudaSuccess) e = raise_smem_limit(z_forward_kernel<T, Z>, smem);
    return cuda_status(e, "z pass shared memory");
  }
  if (inverse)
    z_inverse_kernel<T, Z><<<grid, kZThreads, smem, s>>>(kb, g, tw);
  else
    z_forward_kernel<T, Z><<<grid, kZThreads, smem, s>>>(kb, g, tw, inv_n);
  return QEB_OK;
}

template <typename T>
RuntimeZ runtime_z(const qeb_local_plan* p) {
  RuntimeZ g;
  line_split(p->nz, &g.z1, &g.z2);
  g.nz = p->nz;
  g.stride = p->nz | 1;
  return g;
}

template <typename T>
int z_pass(const KBatch<T>& kb, const qeb_local_plan* p, bool inverse, int nk, int nb, int blocks,
           cudaStream_t s) {
  const dim3 grid(blocks, nb, nk);
  const T inv_n = T(1.0 / ((double)p->nx * p->ny * p->nz));
  const C2<T>* tw = tw_at<T>(p, 2);
#define QEB_CASE(n, a, b, k1, k2) \
  if (p->nz == n) return launch_z<T>(kb, StaticZ<a, b>{}, inverse, grid, tw, inv_n, s);
  QEB_LINE_LENGTHS(QEB_CASE)
#undef QEB_CASE
  return launch_z<T>(kb, runtime_z<T>(p), inverse, grid, tw, inv_n, s);
}

template <typename T>
KDesc<T> describe(const qeb_local_plan* p, void* sticks, const void* psi, int64_t ld, int64_t nb,
                  const void* kinetic, void* out, int64_t ldo) {
  KDesc<T> d;
  d.psi = static_cast<const C2<T>*>(psi);
  d.out = static_cast<C2<T>*>(out);
  d.kinetic = static_cast<const T*>(kinetic);
  d.sticks = static_cast<C2<T>*>(sticks);
  d.entry_g = p->entry_g;
  d.entry_pos = p->entry_pos;
  d.stick_off = p->stick_off;
  d.stick_map = p->stick_map;
  d.ld = ld;
  d.ldo = ldo;
  d.nst = p->nst;
  d.rows = p->line_rows;
  d.nb = (int)nb;
  d.xmask = p->xmask;
  d.ymask = p->ymask;
  d.zmask = p->zmask;
  return d;
}

// ---------------------------------------------------------------------------
// Persistent form: the three passes of every k point in one cooperative launch
// of as many blocks as fit on the GPU at once; each block takes work items (a
// stick block or a z plane of one band of one k point) in turn, and a grid
// barrier separates the passes.  Run-time sizes, same bodies and bits as the
// three launches.

constexpr long long kBarrierLimit = 1ll << 24;  // polls before a barrier gives up

// Grid barrier over `nblocks` co-resident blocks on two words of global
// memory (arrival count, generation), bounded: false when the wait gave up,
// which the caller records.  The last block to arrive resets the count and
// advances the generation; the others wait for the generation to change.
__device__ __forceinline__ bool grid_barrier(unsigned int* words, unsigned int nblocks) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    volatile unsigned int* generation = words + 1;
    const unsigned int g = *generation;
    __threadfence();  // this block's writes before its arrival
    if (atomicAdd(words, 1u) == nblocks - 1) {
      words[0] = 0u;
      __threadfence();
      atomicAdd(words + 1, 1u);
    } else {
      long long polls = 0;
      while (*generation == g) {
        if (++polls > kBarrierLimit) {
          ok = 0;
          break;
        }
      }
    }
    __threadfence();  // the other blocks' writes before this block reads
  }
  __syncthreads();
  return ok != 0;
}

template <typename T>
__global__ void __launch_bounds__(kZThreads) persistent_kernel(
    const __grid_constant__ KBatch<T> kb, const __grid_constant__ RuntimePlane gp,
    const __grid_constant__ RuntimeZ gz, int nk, int sblocks, int max_nb, const C2<T>* tw_x,
    const C2<T>* tw_y, const C2<T>* tw_z, const T* potential, T inv_n, unsigned int* barrier,
    int* error) {
  const int64_t per_k_z = (int64_t)max_nb * sblocks, items_z = nk * per_k_z;
  const int64_t per_k_p = (int64_t)max_nb * gz.nz, items_p = nk * per_k_p;
  const DensityTarget none{};
  for (int pass = 0; pass < 3; ++pass) {
    if (pass > 0 && !grid_barrier(barrier, gridDim.x) && threadIdx.x == 0) atomicExch(error, 21);
    const int64_t items = pass == 1 ? items_p : items_z, per_k = pass == 1 ? per_k_p : per_k_z;
    const int per_band = pass == 1 ? gz.nz : sblocks;
    for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
      const int k = (int)(it / per_k);
      const int64_t r = it - k * per_k;
      const int band = (int)(r / per_band), x = (int)(r - (int64_t)band * per_band);
      const KDesc<T>& d = kb.k[k];
      if (band >= d.nb || (pass != 1 && x * kSticks >= d.nst)) continue;
      __syncthreads();  // shared memory of the previous item
      if (pass == 0) z_inverse_body<T, RuntimeZ>(d, gz, tw_z, x, band);
      if (pass == 1)
        plane_body<T, 0, RuntimePlane>(d, gp, gz.nz, tw_x, tw_y, potential, none, x, band);
      if (pass == 2) z_forward_body<T, RuntimeZ>(d, gz, tw_z, inv_n, x, band);
    }
  }
}

std::atomic<int> g_persistent{0};

template <typename T>
int launch_persistent(const KBatch<T>& kb, const qeb_local_plan* p, int nk, int nb, int blocks,
                      int rows, const T* potential, unsigned int* barrier, cudaStream_t s) {
  RuntimePlane gp = runtime_plane<T>(p, rows);
  RuntimeZ gz = runtime_z<T>(p);
  // dynamic and the barrier's static shared memory together stay below a
  // block's limit
  const size_t limit = kMaxSmem - 1024;
  while (gp.columns > 1 &&
         plane_smem<T>(gp.x1, gp.x2, gp.y1, gp.y2, gp.rows, gp.columns) > limit)
    --gp.columns;
  const size_t smem =
      std::max(plane_smem<T>(gp.x1, gp.x2, gp.y1, gp.y2, gp.rows, gp.columns),
               sizeof(C2<T>) * ((size_t)kSticks * gz.stride + gz.nz));
  int per_sm = 0, device = 0, sms = 0;
  cudaError_t e = raise_smem_limit(persistent_kernel<T>, smem);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, persistent_kernel<T>, kZThreads,
                                                      smem);
  if (e == cudaSuccess) e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return cuda_status(e, "persistent passes: occupancy");
  if (per_sm < 1) {
    set_error("persistent passes: a block of %zu bytes of shared memory does not fit", smem);
    return QEB_EUNSUPPORTED;
  }
  int* error = nullptr;
  int rc = tensor_error_word(&error);
  if (rc) return rc;
  e = cudaMemsetAsync(barrier, 0, 2 * sizeof(unsigned int), s);
  if (e != cudaSuccess) return cuda_status(e, "persistent passes: barrier reset");
  KBatch<T> batch = kb;
  const C2<T>*tw_x = tw_at<T>(p, 0), *tw_y = tw_at<T>(p, 1), *tw_z = tw_at<T>(p, 2);
  T inv_n = T(1.0 / ((double)p->nx * p->ny * p->nz));
  void* args[] = {&batch, &gp,   &gz,   &nk,        &blocks, &nb,     &tw_x,
                  &tw_y,  &tw_z, &potential, &inv_n,  &barrier, &error};
  // cooperative: every block of the grid is resident at once, which the grid
  // barrier needs
  e = cudaLaunchCooperativeKernel(reinterpret_cast<void*>(persistent_kernel<T>),
                                  dim3(per_sm * sms), dim3(kZThreads), args, smem, s);
  count_launches(1);
  return cuda_status(e, "persistent passes launch");
}

template <typename T>
int apply_t(int nk, const qeb_local_plan* const* plans, void* const* sticks,
            const void* const* psi, const int64_t* ld, const int64_t* nb, const void* potential,
            const void* const* kinetic, void* const* out, const int64_t* ldo, cudaStream_t s,
            cudaEvent_t* ev, unsigned int* barrier) {
  KBatch<T> kb;
  const T* v = static_cast<const T*>(potential);
  int max_nb = 0, blocks = 0, rows = 0;
  bool one_k = true;  // one static plane kernel serves every k point
  for (int k = 0; k < nk; ++k) {
    const qeb_local_plan* p = plans[k];
    kb.k[k] = describe<T>(p, sticks[k], psi[k], ld[k], nb[k], kinetic[k], out[k], ldo[k]);
    max_nb = std::max(max_nb, kb.k[k].nb);
    blocks = std::max(blocks, (p->nst + kSticks - 1) / kSticks);
    rows = std::max(rows, p->line_rows);
    one_k = one_k && p->line_k == plans[0]->line_k;
  }
  if (max_nb == 0) return QEB_OK;
  const qeb_local_plan* p0 = plans[0];
  if (g_persistent.load() && ev == nullptr && barrier != nullptr)
    return launch_persistent<T>(kb, p0, nk, max_nb, blocks, rows, v, barrier, s);
  int rc, launches = 2;
  if (ev) cudaEventRecord(ev[0], s);
  if ((rc = z_pass<T>(kb, p0, true, nk, max_nb, blocks, s))) return rc;
  if (ev) cudaEventRecord(ev[1], s);
  if (one_k) {
    if ((rc = plane_pass(kb, p0, 0, nk, max_nb, v, DensityTarget{}, s))) return rc;
    ++launches;
  } else {  // one launch per number of kept blocks
    bool done[QEB_MAX_KBATCH] = {false};
    for (int k = 0; k < nk; ++k) {
      if (done[k]) continue;
      KBatch<T> part;
      int n = 0, part_nb = 0;
      for (int j = k; j < nk; ++j) {
        if (plans[j]->line_k != plans[k]->line_k) continue;
        done[j] = true;
        part.k[n++] = kb.k[j];
        part_nb = std::max(part_nb, kb.k[j].nb);
      }
      if (part_nb == 0) continue;
      if ((rc = plane_pass(part, plans[k], 0, n, part_nb, v, DensityTarget{}, s))) return rc;
      ++launches;
    }
  }
  if (ev) cudaEventRecord(ev[2], s);
  if ((rc = z_pass<T>(kb, p0, false, nk, max_nb, blocks, s))) return rc;
  if (ev) cudaEventRecord(ev[3], s);
  count_launches(launches);
  return cuda_status(cudaGetLastError(), "local apply launch");
}

// density[x, y, z] += grid[z, x, y]: 32 x 32 tiles of (y, z) through shared
// memory, both sides coalesced.  Atomic, as the straight form is: calls on
// several streams, each with scratch of its own, may add to one density.
__global__ void __launch_bounds__(256) density_add_kernel(int nx, int ny, int nz,
                                                          const double* __restrict__ grid,
                                                          double* __restrict__ density) {
  __shared__ double tile[32][33];
  const int x = blockIdx.z, y0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  for (int j = ty; j < 32; j += 8)
    if (z0 + j < nz && y0 + tx < ny)
      tile[j][tx] = grid[((int64_t)(z0 + j) * nx + x) * ny + y0 + tx];
  __syncthreads();
  for (int j = ty; j < 32; j += 8)
    if (y0 + j < ny && z0 + tx < nz)
      atomicAdd(density + ((int64_t)x * ny + y0 + j) * nz + z0 + tx, tile[tx][j]);
}

// grid: nx ny nz doubles of scratch in which the bands' contributions are
// added in the plane pass's own (z, x, y) order, so that the atomics of a warp
// fall on consecutive values, or null: atomics straight into the density, one
// 32-byte sector per point (480 bands
// on 135^3, FP64: 10.3 ms against 7.7 ms with the grid).
template <typename T>
int density_t(const qeb_local_plan* p, void* sticks, double* grid, const void* psi, int64_t ld,
              int64_t nb, const double* weights, double* density, cudaStream_t s) {
  KBatch<T> kb;
  kb.k[0] = describe<T>(p, sticks, psi, ld, nb, nullptr, nullptr, 0);
  int rc = z_pass<T>(kb, p, true, 1, (int)nb, (p->nst + kSticks - 1) / kSticks, s);
  if (rc) return rc;
  DensityTarget rho{weights, density, (int64_t)p->ny * p->nz, p->nz, 1};
  if (grid != nullptr) {
    const size_t bytes = sizeof(double) * (size_t)p->nx * p->ny * p->nz;
    const cudaError_t e = cudaMemsetAsync(grid, 0, bytes, s);
    if (e != cudaSuccess) return cuda_status(e, "density scratch");
    rho = DensityTarget{weights, grid, p->ny, 1, (int64_t)p->nx * p->ny};
  }
  if ((rc = plane_pass(kb, p, 1, 1, (int)nb, (const T*)nullptr, rho, s))) return rc;
  if (grid != nullptr)
    density_add_kernel<<<dim3((p->ny + 31) / 32, (p->nz + 31) / 32, p->nx), 256, 0, s>>>(
        p->nx, p->ny, p->nz, grid, density);
  count_launches(grid != nullptr ? 3 : 2);
  return cuda_status(cudaGetLastError(), "density launch");
}

template <typename T>
int prepare_t(const qeb_local_plan* p) {
  KBatch<T> kb;
  kb.k[0] = describe<T>(p, nullptr, nullptr, 0, 0, nullptr, nullptr, 0);
  int rc = z_pass<T>(kb, p, true, 1, 0, 0, nullptr);
  for (int mode = 0; mode < 2 && rc == QEB_OK; ++mode)
    rc = plane_pass(kb, p, mode, 1, 0, (const T*)nullptr, DensityTarget{}, nullptr);
  return rc;
}

}  // namespace
}  // namespace lines

bool line_split(int n, int* n1, int* n2) {
#define QEB_CASE(len, a, b, k1, k2) \
  if (n == len) {           \
    *n1 = a;                \
    *n2 = b;                \
    return true;            \
  }
  QEB_LINE_LENGTHS(QEB_CASE)
#undef QEB_CASE
  return false;
}

int line_keep(int n, int reach) {
#define QEB_CASE(len, a, b, k1, k2) \
  if (n == len) return reach <= k1 * b ? k1 : (reach <= k2 * b ? k2 : 0);
  QEB_LINE_LENGTHS(QEB_CASE)
#undef QEB_CASE
  return 0;
}

int line_columns(const qeb_local_plan* p) {
  int x1, x2, y1, y2;
  if (!line_split(p->nx, &x1, &x2) || !line_split(p->ny, &y1, &y2)) return 0;
  return p->precision == QEB_F64 ? lines::plane_columns<double>(x1, x2, y1, y2, p->line_rows, false)
                                 : lines::plane_columns<float>(x1, x2, y1, y2, p->line_rows, false);
}

int lines_prepare(const qeb_local_plan* p) {
  return p->precision == QEB_F64 ? lines::prepare_t<double>(p) : lines::prepare_t<float>(p);
}

int lines_apply(int nk, const qeb_local_plan* const* plans, void* const* sticks,
                const void* const* psi, const int64_t* ld, const int64_t* nb,
                const void* potential, const void* const* kinetic, void* const* out,
                const int64_t* ldo, cudaStream_t stream, cudaEvent_t* events,
                unsigned int* barrier) {
  return plans[0]->precision == QEB_F64
             ? lines::apply_t<double>(nk, plans, sticks, psi, ld, nb, potential, kinetic, out, ldo,
                                      stream, events, barrier)
             : lines::apply_t<float>(nk, plans, sticks, psi, ld, nb, potential, kinetic, out, ldo,
                                     stream, events, barrier);
}

int lines_density(const qeb_local_plan* p, void* sticks, double* grid, const void* psi, int64_t ld,
                  int64_t nb, const double* weights, double* density, cudaStream_t stream) {
  return p->precision == QEB_F64
             ? lines::density_t<double>(p, sticks, grid, psi, ld, nb, weights, density, stream)
             : lines::density_t<float>(p, sticks, grid, psi, ld, nb, weights, density, stream);
}

}  // namespace qeb

extern "C" int qeb_set_persistent_passes(int enabled) {
  qeb::lines::g_persistent.store(enabled ? 1 : 0);
  return QEB_OK;
}

extern "C" int qeb_persistent_passes(void) { return qeb::lines::g_persistent.load(); }
