// MAP phase kernels (phase_log.cuh), double arithmetic.
#include "phase_log.cuh"

namespace thmm {

cudaError_t LaunchPhaseMaximumF64(int kind, const PhaseArgs &args, LaunchStream stream,
                                  int *blocks_per_sm) {
  return LaunchLog<double, false>(kind, args, stream, blocks_per_sm);
}

} // namespace thmm
