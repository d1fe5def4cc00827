// cpm_sweep3d.cu — the 3D sweep kernels (cpm_sweep.cuh): 26 neighbours, the
// terms of copyAttempt3d (src/kernels3d.cu:51-594).
#include "cpm_sweep.cuh"

namespace gpucpm {

cudaError_t launch_sweep3d(const SweepArgs& a, bool batch, int grid, int warps, cudaStream_t s) {
  return launch_sweep_nd<3>(a, batch, false, grid, warps, s);
}

}  // namespace gpucpm
