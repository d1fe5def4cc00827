// cpm_sweep2d.cu — the 2D sweep kernels (cpm_sweep.cuh): Moore-8
// neighbourhood, the terms of copyAttempt (src/kernels2d.cu:44-583), and the
// score kernels of the differentiable ensembles.
#include "cpm_sweep.cuh"

namespace gpucpm {

cudaError_t launch_sweep2d(const SweepArgs& a, bool batch, bool scores, int grid, int warps,
                           cudaStream_t s) {
  return launch_sweep_nd<2>(a, batch, scores, grid, warps, s);
}

}  // namespace gpucpm
