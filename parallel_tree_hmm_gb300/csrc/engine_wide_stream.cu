// Launchers of the pipelined compress kinds (wide_stream.cuh), 32 < K <= 128 and
// K a multiple of 4.
#include "wide_stream.cuh"

namespace thmm {
namespace {

template <int KP, bool kReverse>
cudaError_t LaunchStreamKind(const PhaseArgs &args, LaunchStream stream, int *blocks_per_sm) {
  using S = wide::StreamLayout<KP, kReverse>;
  const bool exact = args.states == KP;
  auto kernel = args.bf16 ? (exact ? wide::WideStreamKernel<KP, kReverse, true, true>
                                   : wide::WideStreamKernel<KP, kReverse, true, false>)
                          : (exact ? wide::WideStreamKernel<KP, kReverse, false, true>
                                   : wide::WideStreamKernel<KP, kReverse, false, false>);
  cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(S::kBytes));
  if (status == cudaSuccess)
    status = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                  cudaSharedmemCarveoutMaxShared);
  if (status != cudaSuccess)
    return status;
  if (blocks_per_sm != nullptr) {
    *blocks_per_sm = S::kResident;
    return cudaSuccess;
  }
  if (args.count == 0)
    return cudaSuccess;
  int device = 0, sms = 0;
  status = cudaGetDevice(&device);
  if (status == cudaSuccess)
    status = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (status != cudaSuccess)
    return status;
  const std::uint64_t slots = static_cast<std::uint64_t>(sms) * S::kResident;
  const unsigned grid = static_cast<unsigned>(args.count < slots ? args.count : slots);
  return LaunchOn(stream, kernel, grid, S::kThreads, S::kBytes, args);
}

} // namespace

cudaError_t LaunchWideStream(int kind, const PhaseArgs &args, LaunchStream stream,
                             int *blocks_per_sm) {
  const bool reverse = kind == kPhaseCompressReverse;
  if (args.states <= 64)
    return reverse ? LaunchStreamKind<64, true>(args, stream, blocks_per_sm)
                   : LaunchStreamKind<64, false>(args, stream, blocks_per_sm);
  return reverse ? LaunchStreamKind<128, true>(args, stream, blocks_per_sm)
                 : LaunchStreamKind<128, false>(args, stream, blocks_per_sm);
}

} // namespace thmm
