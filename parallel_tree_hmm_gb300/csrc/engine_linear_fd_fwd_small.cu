// Sum-product kernels, float inputs/outputs with double arithmetic, forward sweep,
// padded state counts 4, 8 and 16 (one translation unit per instance group so
// the build compiles them in parallel).
#include "engine_launch.cuh"

namespace thmm {

cudaError_t LaunchLinearFDForwardSmall(unsigned kmax, const EngineArgs &args, int grid,
                          LaunchStream stream, int *blocks_per_sm) {
  return LaunchLinearHalf<float, double, kLinearForward, true>(kmax, args, grid, stream, blocks_per_sm);
}

} // namespace thmm
