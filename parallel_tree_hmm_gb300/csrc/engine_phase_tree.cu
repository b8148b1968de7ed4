// Launchers of the tree-per-block kernels (phase_tree.cuh).
#include "phase_tree.cuh"

namespace thmm {
namespace {

template <typename Scalar, typename Compute, int K>
cudaError_t LaunchTree(const TreePhaseArgs &args, LaunchStream stream) {
  auto kernel = TreePhaseKernel<Scalar, Compute, K>;
  if (args.at.bytes > 48 * 1024) {
    // The limit belongs to the kernel and not to the launch: every workspace and
    // thread sets the same one, or one would lower it under another's launch.
    const cudaError_t status = cudaFuncSetAttribute(
        kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTreePhaseMaxBytes));
    if (status != cudaSuccess)
      return status;
  }
  if (args.phase.items == 0)
    return cudaSuccess;
  return LaunchOn(stream, kernel, args.phase.items, kTreePhaseThreads, args.at.bytes, args);
}

template <typename Scalar, typename Compute>
cudaError_t LaunchStates(const TreePhaseArgs &args, LaunchStream stream) {
  switch (args.phase.states) {
  case 1:
    return LaunchTree<Scalar, Compute, 1>(args, stream);
  case 2:
    return LaunchTree<Scalar, Compute, 2>(args, stream);
  case 3:
    return LaunchTree<Scalar, Compute, 3>(args, stream);
  case 4:
    return LaunchTree<Scalar, Compute, 4>(args, stream);
  default:
    return cudaErrorInvalidValue;
  }
}

} // namespace

cudaError_t LaunchTreePhase(int scalar_bytes, bool compute_f64, const TreePhaseArgs &args,
                            LaunchStream stream) {
  if (scalar_bytes == 8)
    return compute_f64 ? LaunchStates<double, double>(args, stream)
                       : LaunchStates<double, float>(args, stream);
  return compute_f64 ? LaunchStates<float, double>(args, stream)
                     : LaunchStates<float, float>(args, stream);
}

} // namespace thmm
