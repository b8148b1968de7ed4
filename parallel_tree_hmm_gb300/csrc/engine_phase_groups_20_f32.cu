// Lane-group phase kernels with register rows of 20 (K in (16, 20]), float
// arithmetic.
#include "phase_groups_launch.cuh"

namespace thmm {

cudaError_t LaunchGroupPhase20F32(int scalar_bytes, int kind, const PhaseArgs &args,
                                   LaunchStream stream, int *blocks_per_sm) {
  return group_phase::Launch<float, 20>(scalar_bytes, kind, args, stream, blocks_per_sm);
}

} // namespace thmm
