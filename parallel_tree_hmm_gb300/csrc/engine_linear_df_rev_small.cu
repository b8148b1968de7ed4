// Sum-product kernels, double inputs/outputs with float arithmetic, adjoint sweep,
// padded state counts 4, 8 and 16 (one translation unit per instance group so
// the build compiles them in parallel).
#include "engine_launch.cuh"

namespace thmm {

cudaError_t LaunchLinearDFReverseSmall(unsigned kmax, const EngineArgs &args, int grid,
                          LaunchStream stream, int *blocks_per_sm) {
  return LaunchLinearHalf<double, float, kLinearReverse, true>(kmax, args, grid, stream, blocks_per_sm);
}

} // namespace thmm
