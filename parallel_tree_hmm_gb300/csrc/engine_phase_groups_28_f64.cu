// Lane-group phase kernels for padded state count 28, double arithmetic.
#include "phase_groups_launch.cuh"

namespace thmm {

cudaError_t LaunchGroupPhase28F64(int scalar_bytes, int kind, const PhaseArgs &args,
                                   LaunchStream stream, int *blocks_per_sm) {
  return group_phase::Launch<double, 28>(scalar_bytes, kind, args, stream, blocks_per_sm);
}

} // namespace thmm
