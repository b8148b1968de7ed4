// A whole tree per block: the sum-product of one item of a small batch (the
// batch API, K <= 4) in one launch.
//
// What bounds a small item is the chain of its rounds. A launch per round and
// kind takes some 5 us however little it does, most of it in three or four
// dependent trips to L2 or DRAM per operation. Here a block loads the records,
// the factors (in compute width) and the input node values of its item into
// shared memory once, and only the results leave it. Four lanes run one
// operation, lane r holding row r: a quarter of the instructions per thread of
// the one-thread form, whose unrolled code spent a round's time on instruction
// fetches (64 items of 999 nodes, double inputs: 90 us a kernel in that form, 40 in
// this one, 157 us in 29 launches).
//
// Each operation performs the floating-point operations of the one-thread form
// (phase_engine.cuh) in the same order, so every schedule agrees bit for bit.
// Input values are put where absorbed values go, with exponent 0: a node has
// one value, and which records read the input does not matter.
#ifndef THMM_PHASE_TREE_CUH_
#define THMM_PHASE_TREE_CUH_

#include <cstdint>
#include <cuda_runtime.h>

#include "engine.cuh"
#include "phase.h"

namespace thmm {

template <typename Scalar, typename Compute, int K> struct TreeOps {
  static constexpr int KK = K * K;
  uint4 *rakes, *gathers, *compress;
  Compute *edges, *comps, *comp_mu, *nodes;
  Scalar *node_out;   // in shared memory, copied out at the end
  Scalar *edge_out;   // the caller's, of this item
  int *node_exp, *comp_exp;
  unsigned r;    // row of this lane (lanes past K hold zeros)
  unsigned mask; // the four lanes of the operation

  // K values at p (a row of a matrix or a vector).
  template <typename T> __device__ __forceinline__ static void Row(const T *p, T (&out)[K]) {
    if constexpr (K == 4) {
      const T *q = static_cast<const T *>(__builtin_assume_aligned(p, 16));
      if constexpr (sizeof(T) == 4) {
        const float4 v = *reinterpret_cast<const float4 *>(q);
        out[0] = v.x, out[1] = v.y, out[2] = v.z, out[3] = v.w;
      } else {
        const double2 v = reinterpret_cast<const double2 *>(q)[0];
        const double2 w = reinterpret_cast<const double2 *>(q)[1];
        out[0] = v.x, out[1] = v.y, out[2] = w.x, out[3] = w.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < K; ++j)
        out[j] = p[j];
    }
  }
  __device__ __forceinline__ unsigned Own() const { return r < K ? r : 0u; }
  __device__ __forceinline__ const Compute *Path(std::uint32_t ref) const {
    return (ref & kFlag) ? comps + (ref & kMask) * KK : edges + ref * KK;
  }
  __device__ __forceinline__ int PathExp(std::uint32_t ref) const {
    return (ref & kFlag) ? comp_exp[ref & kMask] : 0;
  }
  __device__ __forceinline__ static int Exponent(Compute m) {
    return m > Compute(0) ? Pow2Exponent(m) : 0;
  }
  __device__ __forceinline__ Compute Max(Compute v) const {
#pragma unroll
    for (int offset = 2; offset > 0; offset >>= 1) {
      const Compute other = __shfl_xor_sync(mask, v, offset, 4);
      v = v < other ? other : v;
    }
    return v;
  }
  // Row r of the adjoint of path `ref`.
  __device__ __forceinline__ void PutAdjoint(std::uint32_t ref, const Compute (&row)[K]) const {
    if (r >= K)
      return;
    if (ref & kFlag) {
#pragma unroll
      for (int j = 0; j < K; ++j)
        comp_mu[(ref & kMask) * KK + r * K + j] = row[j];
    } else {
      Scalar *out = edge_out + static_cast<std::size_t>(ref) * KK + r * K;
      if constexpr (K == 4) {
        StoreRowStreaming<4>(out, 4u, row);
      } else {
#pragma unroll
        for (int j = 0; j < K; ++j)
          out[j] = static_cast<Scalar>(row[j]);
      }
    }
  }

  __device__ __forceinline__ void Gather(std::uint32_t i) const {
    const uint4 op = gathers[i];
    const std::uint32_t node = op.x & kMask, count = op.w & kCountMask;
    Compute v = r < K ? nodes[node * K + r] : Compute(0);
    int e = node_exp[node];
    for (std::uint32_t k = 0; k < count; ++k) {
      const uint4 rake = rakes[op.z + k];
      const std::uint32_t leaf_node = rake.y & kMask;
      Compute leaf[K], row[K];
      Row(nodes + leaf_node * K, leaf);
      Row(Path(rake.x) + Own() * K, row);
      e += node_exp[leaf_node] + PathExp(rake.x);
      Compute dot = Compute(0);
#pragma unroll
      for (int j = 0; j < K; ++j)
        dot = fma(row[j], leaf[j], dot);
      if (r >= K)
        dot = Compute(0);
      const int s1 = Exponent(Max(dot));
      const Compute value = v * ScalePow2(dot, -s1);
      const int s2 = Exponent(Max(value));
      v = ScalePow2(value, -s2);
      e += s1 + s2;
    }
    if (r < K)
      nodes[node * K + r] = v;
    if (r == 0)
      node_exp[node] = e;
  }

  // left * diag(middle) * right, row r.
  __device__ __forceinline__ static void Product(const Compute (&left)[K],
                                                 const Compute (&middle)[K],
                                                 const Compute (&right)[K][K],
                                                 Compute (&out)[K]) {
#pragma unroll
    for (int j = 0; j < K; ++j)
      out[j] = Compute(0);
#pragma unroll
    for (int m = 0; m < K; ++m) {
      const Compute weight = left[m] * middle[m];
#pragma unroll
      for (int j = 0; j < K; ++j)
        out[j] = fma(weight, right[m][j], out[j]);
    }
  }

  __device__ __forceinline__ void Compress(std::uint32_t i) const {
    const uint4 op = compress[i];
    const std::uint32_t node = op.y & kMask;
    Compute left[K], middle[K], right[K][K], out[K];
    Row(Path(op.x) + Own() * K, left);
    Row(nodes + node * K, middle);
#pragma unroll
    for (int m = 0; m < K; ++m)
      Row(Path(op.z) + m * K, right[m]);
    const int e = PathExp(op.x) + PathExp(op.z) + node_exp[node];
    Product(left, middle, right, out);
    Compute m = Compute(0);
#pragma unroll
    for (int j = 0; j < K; ++j)
      m = m < out[j] ? out[j] : m;
    const int s = Exponent(Max(r < K ? m : Compute(0)));
    if (r < K) {
#pragma unroll
      for (int j = 0; j < K; ++j)
        comps[i * KK + r * K + j] = ScalePow2(out[j], -s);
    }
    if (r == 0)
      comp_exp[i] = e + s;
  }

  __device__ __forceinline__ void RakeReverse(std::uint32_t i) const {
    const uint4 op = rakes[i];
    const std::uint32_t leaf_node = op.y & kMask;
    const Compute *path = Path(op.x);
    Compute leaf[K], row[K];
    Row(nodes + leaf_node * K, leaf);
    Row(path + Own() * K, row);
    Compute unnormalised = Compute(0);
#pragma unroll
    for (int j = 0; j < K; ++j)
      unnormalised = fma(row[j], leaf[j], unnormalised);
    const Compute parent_adjoint =
        r < K ? static_cast<Compute>(node_out[op.w * K + r]) : Compute(0);
    const Compute ratio =
        r < K && unnormalised > Compute(0) ? parent_adjoint / unnormalised : Compute(0);
#pragma unroll
    for (int j = 0; j < K; ++j)
      row[j] = ratio * row[j] * leaf[j];
    PutAdjoint(op.x, row);
    Compute column = Compute(0);
#pragma unroll
    for (int p = 0; p < K; ++p)
      column = fma(__shfl_sync(mask, ratio, p, 4), path[p * K + Own()], column);
    if (r < K)
      node_out[leaf_node * K + r] = static_cast<Scalar>(nodes[leaf_node * K + r] * column);
  }

  __device__ __forceinline__ void CompressReverse(std::uint32_t i) const {
    const uint4 op = compress[i];
    const std::uint32_t node = op.y & kMask;
    const Compute *left_path = Path(op.x);
    Compute left[K], middle[K], right[K][K], ratio[K], adjoint[K];
    Row(left_path + Own() * K, left);
    Row(nodes + node * K, middle);
#pragma unroll
    for (int m = 0; m < K; ++m)
      Row(Path(op.z) + m * K, right[m]);
    Row(static_cast<const Compute *>(comp_mu) + i * KK + Own() * K, adjoint);
    Product(left, middle, right, ratio);
#pragma unroll
    for (int j = 0; j < K; ++j)
      ratio[j] = ratio[j] > Compute(0) ? adjoint[j] / ratio[j] : Compute(0);
    Compute out[K];
#pragma unroll
    for (int m = 0; m < K; ++m) {
      Compute dot = Compute(0);
#pragma unroll
      for (int j = 0; j < K; ++j)
        dot = fma(right[m][j], ratio[j], dot);
      out[m] = left[m] * middle[m] * dot;
    }
    PutAdjoint(op.x, out);
    // Right adjoint, row m = r.
#pragma unroll
    for (int j = 0; j < K; ++j)
      out[j] = Compute(0);
#pragma unroll
    for (int p = 0; p < K; ++p) {
      const Compute left_p = left_path[p * K + Own()];
#pragma unroll
      for (int j = 0; j < K; ++j)
        out[j] = fma(left_p, __shfl_sync(mask, ratio[j], p, 4), out[j]);
    }
    Compute own[K];
    Row(Path(op.z) + Own() * K, own);
    const Compute middle_r = nodes[node * K + Own()];
    Compute total = Compute(0);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      out[j] = own[j] * middle_r * out[j];
      total += out[j];
    }
    PutAdjoint(op.z, out);
    if (r < K)
      node_out[node * K + r] = static_cast<Scalar>(total);
  }
};

// put(i, load(i)) for every i < count, each thread with eight loads in flight.
template <typename T, class Load, class Put>
__device__ __forceinline__ void CopyIn(std::uint32_t count, Load load, Put put) {
  constexpr unsigned kDeep = 8;
  for (std::uint32_t first = threadIdx.x; first < count; first += kDeep * kTreePhaseThreads) {
    T v[kDeep];
#pragma unroll
    for (unsigned b = 0; b < kDeep; ++b)
      if (const std::uint32_t i = first + b * kTreePhaseThreads; i < count)
        v[b] = load(i);
#pragma unroll
    for (unsigned b = 0; b < kDeep; ++b)
      if (const std::uint32_t i = first + b * kTreePhaseThreads; i < count)
        put(i, v[b]);
  }
}

// Starts copying `count` records (of 8 or 16 bytes) into shared memory.
template <typename T>
__device__ __forceinline__ void CopyAsyncAll(T *dst, const T *src, std::uint32_t count) {
  for (std::uint32_t i = threadIdx.x; i < count; i += kTreePhaseThreads)
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(dst + i))),
                 "l"(src + i), "n"(sizeof(T))
                 : "memory");
}

// Block b takes item first_item + b.
template <typename Scalar, typename Compute, int K>
__global__ void __launch_bounds__(kTreePhaseThreads) TreePhaseKernel(TreePhaseArgs args) {
  extern __shared__ __align__(16) unsigned char tree_smem[];
  const PhaseArgs &in = args.phase;
  const TreePhaseLayout &at = args.at;
  const std::uint64_t item = in.first_item + blockIdx.x;
  const unsigned t = threadIdx.x;
  TreeOps<Scalar, Compute, K> ops;
  ops.rakes = reinterpret_cast<uint4 *>(tree_smem);
  ops.gathers = reinterpret_cast<uint4 *>(tree_smem + at.gathers);
  ops.compress = reinterpret_cast<uint4 *>(tree_smem + at.compress);
  ops.edges = reinterpret_cast<Compute *>(tree_smem + at.edges);
  ops.comps = reinterpret_cast<Compute *>(tree_smem + at.comps);
  ops.comp_mu = reinterpret_cast<Compute *>(tree_smem + at.comp_mu);
  ops.nodes = reinterpret_cast<Compute *>(tree_smem + at.nodes);
  ops.node_out = reinterpret_cast<Scalar *>(tree_smem + at.node_out);
  ops.node_exp = reinterpret_cast<int *>(tree_smem + at.node_exp);
  ops.comp_exp = reinterpret_cast<int *>(tree_smem + at.comp_exp);
  ops.edge_out = static_cast<Scalar *>(in.edge_out) + item * in.item_edges * (K * K);
  ops.r = t & 3u;
  ops.mask = 0xfu << (t & 28u);

  const Scalar *edge_in = static_cast<const Scalar *>(in.edge_in);
  // The records by asynchronous copies, under the loads of the factors.
  uint4 *rounds = reinterpret_cast<uint4 *>(tree_smem + at.rounds);
  uint2 *round_rakes = reinterpret_cast<uint2 *>(tree_smem + at.round_rakes);
  CopyAsyncAll(ops.rakes, in.rakes, args.rakes);
  CopyAsyncAll(ops.gathers, in.gathers, args.gathers);
  CopyAsyncAll(ops.compress, in.compress, args.compressions);
  CopyAsyncAll(rounds, args.round_ops, args.rounds);
  CopyAsyncAll(round_rakes, args.round_rakes, args.rounds);
  const std::uint32_t root = in.roots[0].x & kMask;
  CopyIn<Scalar>(
      args.edges * (K * K), [&](std::uint32_t i) { return edge_in[i]; },
      [&](std::uint32_t i, Scalar v) { ops.edges[i] = static_cast<Compute>(v); });
  for (std::uint32_t i = t; i < args.nodes; i += kTreePhaseThreads)
    ops.node_exp[i] = 0;
  if (!in.categorical) {
    const Scalar *node_in = static_cast<const Scalar *>(in.node_in) + item * args.nodes * K;
    CopyIn<Scalar>(
        args.nodes * K, [&](std::uint32_t i) { return node_in[i]; },
        [&](std::uint32_t i, Scalar v) { ops.nodes[i] = static_cast<Compute>(v); });
  } else { // as PhaseOps::Input
    const Scalar *root_potential = static_cast<const Scalar *>(in.root_potential);
    const Scalar *emission = static_cast<const Scalar *>(in.emission);
    for (std::uint32_t i = t; i < args.nodes * K; i += kTreePhaseThreads)
      ops.nodes[i] =
          static_cast<Compute>(i / K == root ? root_potential[i % K] : Scalar(1));
    __syncthreads();
    CopyIn<uint2>(
        args.observed,
        [&](std::uint32_t k) {
          return make_uint2(args.observed_nodes[k],
                            args.observations[item * args.observed + k]);
        },
        [&](std::uint32_t, uint2 v) {
#pragma unroll
          for (int j = 0; j < K; ++j) {
            Scalar value = Scalar(0);
            if (v.y < in.categories) {
              value = emission[v.y * K + j];
              if (v.x == root)
                value = root_potential[j] * value;
            }
            ops.nodes[v.x * K + j] = static_cast<Compute>(value);
          }
        });
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  constexpr unsigned kGroups = kTreePhaseThreads / 4;
  const unsigned g = t / 4;
  for (std::uint32_t e = 0; e < args.rounds; ++e) {
    const uint4 round = rounds[e];
    for (std::uint32_t i = g; i < round.y; i += kGroups)
      ops.Gather(round.x + i);
    __syncthreads();
    if (round.w != 0) {
      for (std::uint32_t i = g; i < round.w; i += kGroups)
        ops.Compress(round.z + i);
      __syncthreads();
    }
  }
  if (t == 0) { // log Z and the root marginal, as PhaseOps::Finish
    double sum = 0.0;
    for (int j = 0; j < K; ++j)
      sum += static_cast<double>(ops.nodes[root * K + j]);
    const double log_z =
        !(sum > 0.0) ? -INFINITY
                     : fma(static_cast<double>(ops.node_exp[root]), 0.6931471805599453094,
                           log(sum));
    static_cast<Scalar *>(in.values)[item] = static_cast<Scalar>(in.raw ? exp(log_z) : log_z);
    if (in.reverse) {
      const bool finite = log_z > -INFINITY;
      for (int j = 0; j < K; ++j)
        ops.node_out[root * K + j] = static_cast<Scalar>(
            finite ? static_cast<double>(ops.nodes[root * K + j]) / sum : 0.0);
    }
  }
  if (!in.reverse)
    return;
  __syncthreads();
  for (std::uint32_t e = args.rounds; e-- > 0;) {
    const uint4 round = rounds[e];
    if (round.w != 0) {
      for (std::uint32_t i = g; i < round.w; i += kGroups)
        ops.CompressReverse(round.z + i);
      __syncthreads();
    }
    const uint2 leaves = round_rakes[e];
    for (std::uint32_t i = g; i < leaves.y; i += kGroups)
      ops.RakeReverse(leaves.x + i);
    __syncthreads();
  }
  Scalar *out = static_cast<Scalar *>(in.node_out) + item * args.nodes * K;
  for (std::uint32_t i = t; i < args.nodes * K; i += kTreePhaseThreads)
    out[i] = ops.node_out[i];
}

} // namespace thmm

#endif // THMM_PHASE_TREE_CUH_
