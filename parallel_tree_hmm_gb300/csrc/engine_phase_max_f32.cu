// MAP phase kernels (phase_log.cuh), float arithmetic.
#include "phase_log.cuh"

namespace thmm {

cudaError_t LaunchPhaseMaximumF32(int kind, const PhaseArgs &args, LaunchStream stream,
                                  int *blocks_per_sm) {
  return LaunchLog<float, false>(kind, args, stream, blocks_per_sm);
}

} // namespace thmm
