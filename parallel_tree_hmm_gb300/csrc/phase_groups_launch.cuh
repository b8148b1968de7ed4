// Launchers of the lane-group phase kernels (phase_groups.cuh) for one
// padded state count; included by engine_phase_groups_*.cu, one translation
// unit per padded state count so that the build compiles them in parallel.
#ifndef THMM_PHASE_GROUPS_LAUNCH_CUH_
#define THMM_PHASE_GROUPS_LAUNCH_CUH_

#include "phase_groups.cuh"
#include "phase_items.cuh"

namespace thmm {
namespace group_phase {

// Warps of 32 items from which a launch runs an item per lane: one per SM
// sub-partition (608). Fewer are bound by a warp's own chain. Marginals at
// K = 20, lane groups -> an item per lane: 61 nodes, 64 items (some 60 warps)
// 66 -> 96 us; 399 nodes, 64 items (400) 119 -> 123; 128 items (800) 160 -> 162;
// 500 items (3,200) 449 -> 402; 1,999 nodes, 64 items (2,000) 328 -> 300, 500
// items 1,899 -> 1,614. K = 8, 1,000 items of 1,999 nodes 1,273 -> 989; K = 32,
// 200 items of 999 nodes 745 -> 686.
constexpr std::uint64_t kItemWarps = 608;
template <typename Scalar, typename Compute, int KMAX, int kKind>
cudaError_t LaunchKind(const PhaseArgs &args, LaunchStream stream, int *blocks_per_sm) {
  // Single precision is bound by instruction issue (53-60 % of the issue
  // slots in the large rounds), which folded bounds shorten: a marginal step
  // of 256 trees of 5,000 nodes at K = 20 2,202 -> 2,141 us, 500 items on a
  // 399-node tree 386 -> 377 us. Double is bound by its pipe and keeps one variant.
  auto kernel = GroupPhaseKernel<Scalar, Compute, KMAX, kKind, kGeneralForm>;
  if constexpr (sizeof(Compute) == 4) {
    if (args.states == KMAX)
      kernel = args.batch ? GroupPhaseKernel<Scalar, Compute, KMAX, kKind, kBatchForm>
                          : GroupPhaseKernel<Scalar, Compute, KMAX, kKind, kForestForm>;
  }
  constexpr unsigned lanes = GroupLanes<KMAX>();
  constexpr unsigned smem = kGroupPhaseThreads / lanes * kGroupPhaseElements<KMAX, kKind> *
                            static_cast<unsigned>(sizeof(Compute));
  static_assert(smem <= 227 * 1024, "shared memory per block");
  if (smem > 48 * 1024) {
    const cudaError_t status = cudaFuncSetAttribute(
        kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (status != cudaSuccess)
      return status;
  }
  if (blocks_per_sm != nullptr)
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel,
                                                         kGroupPhaseThreads, smem);
  if (args.count == 0 || args.items == 0)
    return cudaSuccess;
  if constexpr (sizeof(Compute) == 4 &&
                (kKind == kPhaseGather || kKind == kPhaseRakeReverse)) {
    const std::uint64_t warps =
        static_cast<std::uint64_t>(args.count) * ((args.items + 31) / 32);
    auto by_item = ItemPhaseKernel<Scalar, KMAX, kKind, true>;
    if constexpr (kKind == kPhaseGather) {
      if (args.states != KMAX)
        by_item = ItemPhaseKernel<Scalar, KMAX, kKind, false>;
    }
    // Rake adjoints of other K write unaligned rows and gain nothing (K = 13,
    // 500 items of 399 nodes: 308 us, with both kinds 337, with gathers 287).
    if (args.batch && args.input_paths && args.items >= 32 && warps >= kItemWarps &&
        (kKind == kPhaseGather || args.states == KMAX)) {
      constexpr unsigned per_block = kItemPhaseThreads / 32;
      return LaunchOn(stream, by_item, static_cast<unsigned>((warps + per_block - 1) / per_block),
                      kItemPhaseThreads, 0, args);
    }
  }
  // One lane group per operation (finish: instance, or a thread) and item.
  const std::uint64_t threads = static_cast<std::uint64_t>(args.count) * args.items *
                                (kKind == kPhaseFinish && !args.reverse ? 1u : lanes);
  const std::uint64_t grid = (threads + kGroupPhaseThreads - 1) / kGroupPhaseThreads;
  if (grid > 0x7fffffffull)
    return cudaErrorInvalidConfiguration;
  return LaunchOn(stream, kernel, static_cast<unsigned>(grid), kGroupPhaseThreads, smem, args);
}

template <typename Scalar, typename Compute, int KMAX>
cudaError_t LaunchTyped(int kind, const PhaseArgs &args, LaunchStream stream,
                        int *blocks_per_sm) {
  switch (kind) {
  case kPhaseGather:
    return LaunchKind<Scalar, Compute, KMAX, kPhaseGather>(args, stream, blocks_per_sm);
  case kPhaseCompress:
    return LaunchKind<Scalar, Compute, KMAX, kPhaseCompress>(args, stream, blocks_per_sm);
  case kPhaseFinish:
    return LaunchKind<Scalar, Compute, KMAX, kPhaseFinish>(args, stream, blocks_per_sm);
  case kPhaseRakeReverse:
    return LaunchKind<Scalar, Compute, KMAX, kPhaseRakeReverse>(args, stream, blocks_per_sm);
  case kPhaseCompressReverse:
    return LaunchKind<Scalar, Compute, KMAX, kPhaseCompressReverse>(args, stream,
                                                                    blocks_per_sm);
  default:
    return cudaErrorInvalidValue; // no tail kinds: every round runs grid-wide
  }
}

// Compute type fixed by the translation unit; scalar_bytes picks the
// input/output type.
template <typename Compute, int KMAX>
cudaError_t Launch(int scalar_bytes, int kind, const PhaseArgs &args, LaunchStream stream,
                   int *blocks_per_sm) {
  return scalar_bytes == 8
             ? LaunchTyped<double, Compute, KMAX>(kind, args, stream, blocks_per_sm)
             : LaunchTyped<float, Compute, KMAX>(kind, args, stream, blocks_per_sm);
}

} // namespace group_phase
} // namespace thmm

#endif // THMM_PHASE_GROUPS_LAUNCH_CUH_
