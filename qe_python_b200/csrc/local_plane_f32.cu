// The plane pass in FP32 (local_lines.cuh).
#include "local_plane_launch.cuh"

int qeb::lines::plane_pass(const KBatch<float>& kb, const qeb_local_plan* p, int mode, int nk, int nb,
                           const float* potential, const DensityTarget& rho, cudaStream_t s) {
  return mode == 0 ? launch_plane<float, 0>(kb, p, nk, nb, potential, rho, s)
                   : launch_plane<float, 1>(kb, p, nk, nb, potential, rho, s);
}
