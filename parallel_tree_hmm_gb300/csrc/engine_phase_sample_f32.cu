// Posterior sampling phase kernels (phase_log.cuh), float arithmetic.
#include "phase_log.cuh"

namespace thmm {

cudaError_t LaunchPhaseSampleF32(int kind, const PhaseArgs &args, LaunchStream stream,
                                  int *blocks_per_sm) {
  return LaunchLog<float, true>(kind, args, stream, blocks_per_sm);
}

} // namespace thmm
