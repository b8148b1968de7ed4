// Lane-group phase kernels for padded state count 8, float arithmetic.
#include "phase_groups_launch.cuh"

namespace thmm {

cudaError_t LaunchGroupPhase8F32(int scalar_bytes, int kind, const PhaseArgs &args,
                                   LaunchStream stream, int *blocks_per_sm) {
  return group_phase::Launch<float, 8>(scalar_bytes, kind, args, stream, blocks_per_sm);
}

} // namespace thmm
