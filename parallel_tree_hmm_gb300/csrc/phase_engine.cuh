// Phase kernels of the level-synchronous schedule (phase.h) for padded state
// count 4 (K <= 4): one thread per operation (one warp or block per tree in the
// tail rounds), the K-vectors and K x K matrices in registers, 16-byte vector
// loads and stores.
//
// Each kernel performs exactly the floating-point operations of the
// one-thread-per-operation (G = 1) branch of LinearEngine (engine.cuh) in
// the same order, so the two schedules agree bit for bit; only the
// bookkeeping of the power-of-two exponents differs (carried per stored
// object here, summed per team there; both are exact integer sums).
#ifndef THMM_PHASE_ENGINE_CUH_
#define THMM_PHASE_ENGINE_CUH_

#include <cstdint>
#include <cuda_runtime.h>

#include "engine.cuh"
#include "phase.h"

namespace thmm {

constexpr int kPhaseThreads = 128;

// Where the operands of one operation live. Forest layout: the records hold
// absolute indices of every tree's nodes, edges and compressions, so every
// map is the identity.
struct ForestIndex {
  static constexpr bool kKeepMarginals = false;
  __device__ __forceinline__ std::size_t Store(std::uint32_t node) const { return node; }
  __device__ __forceinline__ std::size_t Io(std::uint32_t node) const { return node; }
  __device__ __forceinline__ std::size_t Comp(std::uint32_t tape) const { return tape; }
  __device__ __forceinline__ std::size_t Out(std::uint32_t edge) const { return edge; }
  __device__ __forceinline__ std::size_t In(std::uint32_t edge) const { return edge; }
  __device__ __forceinline__ std::size_t Obs(std::uint32_t slot) const { return slot; }
};

// Shared-topology layout (the reference's batch API: one plan, B node-factor
// sets, one edge input): the records are those of ONE tree and are read by
// every batch item, and consecutive threads take consecutive batch items of
// the same operation, so a warp reads each record and each edge row once
// (the addresses coincide) instead of once per item. Stored values are
// item-minor ([node][item]) so the warp's accesses are contiguous; the
// phase-ordered observations likewise ([slot][item]). Caller-visible arrays
// keep the reference's item-major layouts.
struct BatchIndex {
  // The children of a node read its marginal from where its value was stored
  // and not from the caller's array, where the items of a warp are a tree apart
  // (marginals of 4,096 items on 1,999 nodes 612 -> 581 us).
  static constexpr bool kKeepMarginals = true;
  std::uint32_t item;   // batch item of this thread
  std::uint64_t stride; // items per stored object (the batch capacity)
  std::uint64_t nodes;  // nodes per item
  std::uint64_t edges;  // edges per item
  __device__ __forceinline__ std::size_t Store(std::uint32_t node) const {
    return node * stride + item;
  }
  __device__ __forceinline__ std::size_t Io(std::uint32_t node) const {
    return item * nodes + node;
  }
  __device__ __forceinline__ std::size_t Comp(std::uint32_t tape) const {
    return tape * stride + item;
  }
  __device__ __forceinline__ std::size_t Out(std::uint32_t edge) const {
    return item * edges + edge;
  }
  __device__ __forceinline__ std::size_t In(std::uint32_t edge) const { return edge; }
  __device__ __forceinline__ std::size_t Obs(std::uint32_t slot) const {
    return slot * stride + item;
  }
};

// Shared memory of a block for the matrix stores below: one 4 x 4 matrix per
// thread at a pitch of 20 floats, whose 16-byte rows fall on different banks.
constexpr int kMatrixPitch = 20;
constexpr int kMatrixTile = 32 * kMatrixPitch; // one warp

// kWarpStores: every lane of a warp runs an operation (some perhaps not live),
// and the lanes store their matrices together (single-precision K = 4).
template <typename Scalar, typename Compute, class Index, bool kWarpStores = false>
struct PhaseOps {
  static constexpr int KMAX = 4;
  const PhaseArgs &a;
  Index ix;
  unsigned K;
  unsigned KK;
  bool live;
  float *tile; // this warp's kMatrixTile floats

  __device__ PhaseOps(const PhaseArgs &args, const Index &index, bool is_live = true,
                      float *warp_tile = nullptr)
      : a(args), ix(index), K(args.states), KK(args.states * args.states), live(is_live),
        tile(warp_tile) {}

  // A matrix leaves row by row: BeginMatrix, PutRow for every row, EndMatrix.
  // A thread's own four 16-byte stores would each write half a sector in 32
  // places; through shared memory, four lanes write a matrix as two whole
  // sectors.
  __device__ __forceinline__ bool Together() const {
    return kWarpStores && sizeof(Scalar) == 4 && sizeof(Compute) == 4 && K == KMAX;
  }
  __device__ __forceinline__ void BeginMatrix() const {
    if (Together())
      __syncwarp(); // the tile's last matrices have left
  }
  template <bool kStreaming, typename D>
  __device__ __forceinline__ void PutRow(D *dst, unsigned q, const Compute (&row)[KMAX]) const {
    if (Together())
      StoreRow<KMAX>(tile + (threadIdx.x & 31u) * kMatrixPitch + 4 * q, K, row);
    else if (live && q < K) {
      if constexpr (kStreaming)
        StoreRowStreaming<KMAX>(dst + q * K, K, row);
      else
        StoreRow<KMAX>(dst + q * K, K, row);
    }
  }
  // `dst`: where this lane's matrix goes. Ordinary stores: evicted first, the
  // marginals of 4,096 sites left L2 before their neighbours came (622 against
  // 610 us a step).
  __device__ __forceinline__ void EndMatrix(void *dst) const {
    if (!Together())
      return;
    const unsigned lane = threadIdx.x & 31u;
    __syncwarp();
    const unsigned long long own = live ? reinterpret_cast<unsigned long long>(dst) : 0ull;
#pragma unroll
    for (unsigned s = 0; s < 4; ++s) {
      const unsigned from = 8 * s + lane / 4, row = lane % 4;
      const unsigned long long to = __shfl_sync(kFull, own, from);
      if (to != 0) {
        const float4 v =
            *reinterpret_cast<const float4 *>(tile + from * kMatrixPitch + 4 * row);
        reinterpret_cast<float4 *>(to)[row] = v;
      }
    }
  }

  // Input factor vector of `node`: dense row, or the reference's categorical
  // (root ? root_potential : 1) * emission[observation]
  // (src/gpu_backend_impl.inc:326-382), as Context::InputNode.
  __device__ __forceinline__ void Input(std::uint32_t node, std::uint32_t obs, bool root,
                                        Compute (&out)[KMAX]) const {
    Scalar raw[KMAX];
    if (!a.categorical) {
      LoadRow<KMAX>(static_cast<const Scalar *>(a.node_in) + ix.Io(node) * K, K, raw);
    } else {
      const Scalar *root_potential = static_cast<const Scalar *>(a.root_potential);
      if (obs == kNone) {
#pragma unroll
        for (unsigned j = 0; j < KMAX; ++j)
          raw[j] = j < K ? (root ? root_potential[j] : Scalar(1)) : Scalar(0);
      } else {
        const unsigned category = a.observations[ix.Obs(obs)];
        if (category >= a.categories) {
#pragma unroll
          for (unsigned j = 0; j < KMAX; ++j)
            raw[j] = Scalar(0);
        } else {
          LoadRow<KMAX>(static_cast<const Scalar *>(a.emission) + category * K, K, raw);
          if (root) {
#pragma unroll
            for (unsigned j = 0; j < KMAX; ++j)
              raw[j] = j < K ? root_potential[j] * raw[j] : Scalar(0);
          }
        }
      }
    }
#pragma unroll
    for (unsigned j = 0; j < KMAX; ++j)
      out[j] = static_cast<Compute>(raw[j]);
  }

  // Value of a rake leaf or compression middle: the stored value (adding its
  // exponent to `e`) or the input factor.
  __device__ __forceinline__ void Node(std::uint32_t ref, std::uint32_t obs,
                                       Compute (&out)[KMAX], int &e) const {
    if (ref & kFlag) {
      const std::size_t at = ix.Store(ref & kMask);
      LoadRow<KMAX>(static_cast<const Compute *>(a.nodes) + at * K, K, out);
      e += a.node_exp[at];
    } else {
      Input(ref, obs, false, out);
    }
  }

  __device__ __forceinline__ const Scalar *EdgeIn(std::uint32_t path) const {
    return static_cast<const Scalar *>(a.edge_in) + ix.In(path) * KK;
  }

  // Row r of path `ref` (zero for padded rows).
  __device__ __forceinline__ void PathRow(std::uint32_t ref, unsigned r,
                                          Compute (&out)[KMAX]) const {
    if (r >= K) {
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        out[j] = Compute(0);
    } else if (ref & kFlag) {
      LoadRow<KMAX>(static_cast<const Compute *>(a.comps) + ix.Comp(ref & kMask) * KK + r * K,
                    K, out);
    } else {
      LoadRow<KMAX>(EdgeIn(ref) + r * K, K, out);
    }
  }
  __device__ __forceinline__ int PathExp(std::uint32_t ref) const {
    return (ref & kFlag) ? a.comp_exp[ix.Comp(ref & kMask)] : 0;
  }

  __device__ __forceinline__ static int Exponent(Compute m) {
    return m > Compute(0) ? Pow2Exponent(m) : 0;
  }
  // FP64 arithmetic is bound by its pipe (a warp instruction every 14 cycles
  // per SM), so it skips the terms past K; FP32 runs them, which is cheaper
  // than the tests.
  __device__ __forceinline__ bool Counts(unsigned j) const {
    return sizeof(Compute) == 4 || j < K;
  }
  // Exponent of the largest of v (0 where none is positive), without FP64
  // comparisons where that one is a normal number.
  template <int N> __device__ __forceinline__ static int MaxExponent(const Compute (&v)[N]) {
    if constexpr (sizeof(Compute) == 8) {
      int hi = 0;
#pragma unroll
      for (int j = 0; j < N; ++j)
        hi = max(hi, __double2hiint(v[j]));
      if (hi >= 0x00100000 && hi < 0x7ff00000)
        return (hi >> 20) - 1022;
    }
    Compute m = Compute(0);
#pragma unroll
    for (int j = 0; j < N; ++j)
      m = m < v[j] ? v[j] : m;
    return Exponent(m);
  }

  // ---------------------------------------------------------- forward
  __device__ __forceinline__ void Gather(std::uint32_t i) const {
    const uint4 op = a.gathers[i];
    const std::uint32_t node = op.x & kMask;
    const std::size_t at = ix.Store(node);
    Compute *dst = static_cast<Compute *>(a.nodes) + at * K;
    Compute v[KMAX];
    int e = 0;
    if (op.x & kFlag) {
      Input(node, op.y, (op.w & kRootBit) != 0, v);
    } else {
      LoadRow<KMAX>(dst, K, v);
      e = a.node_exp[at];
    }
    const std::uint32_t count = op.w & kCountMask;
    for (std::uint32_t k = 0; k < count; ++k) {
      const uint4 rake = a.rakes[op.z + k];
      Compute leaf[KMAX];
      Node(rake.y, rake.z, leaf, e);
      e += PathExp(rake.x);
      Compute message[KMAX];
#pragma unroll
      for (int q = 0; q < KMAX; ++q) {
        Compute row[KMAX];
        PathRow(rake.x, q, row);
        Compute dot = Compute(0);
#pragma unroll
        for (unsigned j = 0; j < KMAX; ++j)
          if (Counts(q) && Counts(j))
            dot = fma(row[j], leaf[j], dot);
        message[q] = dot;
      }
      int s = MaxExponent(message);
      e += s;
#pragma unroll
      for (int q = 0; q < KMAX; ++q)
        if (Counts(q))
          v[q] = v[q] * ScalePow2(message[q], -s);
      s = MaxExponent(v);
      e += s;
#pragma unroll
      for (int q = 0; q < KMAX; ++q)
        if (Counts(q))
          v[q] = ScalePow2(v[q], -s);
    }
    StoreRow<KMAX>(dst, K, v);
    a.node_exp[at] = e;
  }

  __device__ __forceinline__ void Compress(std::uint32_t i) const {
    const uint4 op = a.compress[i];
    int e = PathExp(op.x) + PathExp(op.z);
    Compute middle[KMAX];
    Node(op.y, op.w, middle, e);
    Compute left[KMAX][KMAX];
    Compute out[KMAX][KMAX];
#pragma unroll
    for (int q = 0; q < KMAX; ++q) {
      PathRow(op.x, q, left[q]);
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        out[q][j] = Compute(0);
    }
#pragma unroll
    for (unsigned mid = 0; mid < KMAX; ++mid) {
      if (mid < K) {
        Compute right[KMAX];
        PathRow(op.z, mid, right);
#pragma unroll
        for (int q = 0; q < KMAX; ++q) {
          if (Counts(q)) {
            const Compute weight = left[q][mid] * middle[mid];
#pragma unroll
            for (unsigned j = 0; j < KMAX; ++j)
              if (Counts(j))
                out[q][j] = fma(weight, right[j], out[q][j]);
          }
        }
      }
    }
    const int s = MaxExponent(reinterpret_cast<const Compute(&)[KMAX * KMAX]>(out));
    const std::size_t at = ix.Comp(i);
    Compute *dst = static_cast<Compute *>(a.comps) + at * KK;
    BeginMatrix();
#pragma unroll
    for (int q = 0; q < KMAX; ++q) {
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        if (Counts(q) && Counts(j))
          out[q][j] = ScalePow2(out[q][j], -s);
      PutRow<false>(dst, q, out[q]);
    }
    EndMatrix(dst);
    if (live)
      a.comp_exp[at] = e + s;
  }

  // Puts the marginal of node `ref` (as the caller's array holds it) in the
  // place of its stored value, which no operation reads again.
  __device__ __forceinline__ void KeepMarginal(std::uint32_t ref,
                                               const Compute (&marginal)[KMAX]) const {
    if constexpr (Index::kKeepMarginals) {
      if (ref & kFlag) {
        Compute kept[KMAX];
#pragma unroll
        for (int j = 0; j < KMAX; ++j)
          kept[j] = static_cast<Compute>(static_cast<Scalar>(marginal[j]));
        StoreRow<KMAX>(static_cast<Compute *>(a.nodes) + ix.Store(ref & kMask) * K, K, kept);
      }
    }
  }

  // log Z = ln 2 * (root exponent) + log(sum(root)), as LinearEngine::Run.
  // Root record `i`; the result is instance `value`'s.
  __device__ __forceinline__ void Finish(std::uint32_t i, std::uint32_t value) const {
    const uint2 rec = a.roots[i];
    const std::uint32_t node = rec.x & kMask;
    Compute root[KMAX];
    long long total = 0;
    if (rec.x & kFlag) {
      const std::size_t at = ix.Store(node);
      LoadRow<KMAX>(static_cast<const Compute *>(a.nodes) + at * K, K, root);
      total = a.node_exp[at];
    } else {
      Input(node, rec.y, true, root);
    }
    double sum = 0.0;
    for (unsigned j = 0; j < KMAX; ++j)
      sum += static_cast<double>(root[j]);
    const double log_z = !(sum > 0.0)
                             ? -INFINITY
                             : fma(static_cast<double>(total), 0.6931471805599453094, log(sum));
    static_cast<Scalar *>(a.values)[value] = static_cast<Scalar>(a.raw ? exp(log_z) : log_z);
    if (a.reverse) {
      Scalar *root_out = static_cast<Scalar *>(a.node_out) + ix.Io(node) * K;
      const bool finite = log_z > -INFINITY;
      for (unsigned j = 0; j < K; ++j) {
        double value = 0.0;
#pragma unroll
        for (unsigned k = 0; k < KMAX; ++k)
          if (k == j)
            value = static_cast<double>(root[k]);
        const Scalar marginal = static_cast<Scalar>(finite ? value / sum : 0.0);
        root_out[j] = marginal;
        if (Index::kKeepMarginals && (rec.x & kFlag))
          static_cast<Compute *>(a.nodes)[ix.Store(node) * K + j] = static_cast<Compute>(marginal);
      }
    }
  }

  // ---------------------------------------------------------- adjoint
  // The adjoint of path `ref`, row by row as above.
  __device__ __forceinline__ Compute *MuAt(std::uint32_t ref) const {
    return static_cast<Compute *>(a.comp_mu) + ix.Comp(ref & kMask) * KK;
  }
  __device__ __forceinline__ Scalar *EdgeOutAt(std::uint32_t ref) const {
    return static_cast<Scalar *>(a.edge_out) + ix.Out(ref) * KK;
  }
  __device__ __forceinline__ void PutAdjointRow(std::uint32_t ref, unsigned q,
                                                const Compute (&row)[KMAX]) const {
    if (ref & kFlag)
      PutRow<false>(MuAt(ref), q, row);
    else
      PutRow<true>(EdgeOutAt(ref), q, row);
  }
  __device__ __forceinline__ void EndAdjoint(std::uint32_t ref) const {
    const bool stored = (ref & kFlag) != 0;
    EndMatrix(stored ? static_cast<void *>(MuAt(ref)) : static_cast<void *>(EdgeOutAt(ref)));
  }

  __device__ __forceinline__ void RakeReverse(std::uint32_t i) const {
    const uint4 op = a.rakes[i];
    Scalar *node_out = static_cast<Scalar *>(a.node_out);
    Compute leaf[KMAX];
    int unused = 0;
    Node(op.y, op.z, leaf, unused);
    Compute parent_adjoint[KMAX];
    if constexpr (Index::kKeepMarginals)
      LoadRow<KMAX>(static_cast<const Compute *>(a.nodes) + ix.Store(op.w) * K, K, parent_adjoint);
    else
      LoadRow<KMAX>(node_out + ix.Io(op.w) * K, K, parent_adjoint);
    Compute ratio[KMAX];
    Compute rows[KMAX][KMAX];
    BeginMatrix();
#pragma unroll
    for (int q = 0; q < KMAX; ++q) {
      PathRow(op.x, q, rows[q]);
      Compute unnormalised = Compute(0);
      Compute w[KMAX] = {};
      ratio[q] = Compute(0);
      if (Counts(q)) {
#pragma unroll
        for (unsigned j = 0; j < KMAX; ++j)
          if (Counts(j))
            unnormalised = fma(rows[q][j], leaf[j], unnormalised);
        ratio[q] = unnormalised > Compute(0) ? parent_adjoint[q] / unnormalised : Compute(0);
#pragma unroll
        for (unsigned j = 0; j < KMAX; ++j)
          if (Counts(j))
            w[j] = ratio[q] * rows[q][j] * leaf[j];
      }
      PutAdjointRow(op.x, q, w);
    }
    EndAdjoint(op.x);
    Compute adjoint[KMAX] = {};
#pragma unroll
    for (unsigned j = 0; j < KMAX; ++j) {
      if (Counts(j)) {
        Compute column = Compute(0);
#pragma unroll
        for (int p = 0; p < KMAX; ++p)
          if (Counts(p))
            column = fma(ratio[p], rows[p][j], column);
        adjoint[j] = leaf[j] * column;
      }
    }
    if (live) {
      StoreRow<KMAX>(node_out + ix.Io(op.y & kMask) * K, K, adjoint);
      KeepMarginal(op.y, adjoint);
    }
  }

  __device__ __forceinline__ void CompressReverse(std::uint32_t i) const {
    const uint4 op = a.compress[i];
    const Compute *output_adjoint = static_cast<const Compute *>(a.comp_mu) + ix.Comp(i) * KK;
    Compute middle[KMAX];
    int unused = 0;
    Node(op.y, op.w, middle, unused);
    Compute left[KMAX][KMAX];
    Compute ratio[KMAX][KMAX];
#pragma unroll
    for (int q = 0; q < KMAX; ++q) {
      PathRow(op.x, q, left[q]);
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        ratio[q][j] = Compute(0);
    }
#pragma unroll
    for (unsigned mid = 0; mid < KMAX; ++mid) {
      if (mid < K) {
        Compute right[KMAX];
        PathRow(op.z, mid, right);
#pragma unroll
        for (int q = 0; q < KMAX; ++q) {
          if (Counts(q)) {
            const Compute weight = left[q][mid] * middle[mid];
#pragma unroll
            for (unsigned j = 0; j < KMAX; ++j)
              if (Counts(j))
                ratio[q][j] = fma(weight, right[j], ratio[q][j]);
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < KMAX; ++q) {
      Compute adjoint[KMAX];
      if (q < static_cast<int>(K)) {
        LoadRow<KMAX>(output_adjoint + q * K, K, adjoint);
      } else {
#pragma unroll
        for (unsigned j = 0; j < KMAX; ++j)
          adjoint[j] = Compute(0);
      }
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        ratio[q][j] = Counts(q) && Counts(j) && ratio[q][j] > Compute(0)
                          ? adjoint[j] / ratio[q][j]
                          : Compute(0);
    }
    Compute rights[KMAX][KMAX];
#pragma unroll
    for (unsigned mid = 0; mid < KMAX; ++mid)
      PathRow(op.z, mid, rights[mid]);
    BeginMatrix();
#pragma unroll
    for (int q = 0; q < KMAX; ++q) {
      Compute left_adjoint[KMAX];
#pragma unroll
      for (unsigned mid = 0; mid < KMAX; ++mid) {
        left_adjoint[mid] = Compute(0);
        if (mid < K && Counts(q)) {
          Compute dot = Compute(0);
#pragma unroll
          for (unsigned j = 0; j < KMAX; ++j)
            if (Counts(j))
              dot = fma(rights[mid][j], ratio[q][j], dot);
          left_adjoint[mid] = left[q][mid] * middle[mid] * dot;
        }
      }
      PutAdjointRow(op.x, q, left_adjoint);
    }
    EndAdjoint(op.x);
    BeginMatrix();
    Compute middle_adjoint[KMAX];
#pragma unroll
    for (unsigned mid = 0; mid < KMAX; ++mid) {
      Compute right_adjoint[KMAX] = {};
      Compute total = Compute(0);
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j) {
        if (Counts(mid) && Counts(j)) {
          Compute acc = Compute(0);
#pragma unroll
          for (int p = 0; p < KMAX; ++p)
            if (Counts(p))
              acc = fma(left[p][mid], ratio[p][j], acc);
          right_adjoint[j] = rights[mid][j] * middle[mid] * acc;
          total += right_adjoint[j];
        }
      }
      middle_adjoint[mid] = total;
      PutAdjointRow(op.z, mid, right_adjoint);
    }
    EndAdjoint(op.z);
    if (live) {
      StoreRow<KMAX>(static_cast<Scalar *>(a.node_out) + ix.Io(op.y & kMask) * K, K,
                     middle_adjoint);
      KeepMarginal(op.y, middle_adjoint);
    }
  }
};

// Tail rounds of one tree per team of kTeam threads (kPhaseTailForward /
// kPhaseTailReverse): a warp or a block, whose threads take the operations of
// a step in turn, with a barrier (which also orders their global-memory
// accesses) between steps. With many trees a warp each fills the chip; up to
// kTailBlockTrees a block each does, and a step of a large tree takes a
// quarter of the passes. The line is what the chip (152 SMs) holds of the kind's
// blocks at its registers (58 to 66, reverse 80 to 92; FP64 100 to 104 and 140);
// beyond it some blocks wait for the others' whole chains. Warps -> blocks:
// marginals of 304 (456, 608) trees of 999 nodes, K = 4, FP64 -10 (-6, +4) %, of
// 456 (760, 1,000) of 127 nodes, K = 2, FP32 +4 (0, +7) %, of 608 (760) of 999 -7
// (0) %; of 4,096 trees, K = 4, 1,739 -> 1,795 us.
template <typename Compute, int kKind>
inline constexpr std::uint32_t kTailBlockTrees =
    152 * (kKind == kPhaseTailForward ? (sizeof(Compute) == 4 ? 7 : 4)
                                      : (sizeof(Compute) == 4 ? 5 : 3));

// Starts moving `count` 16-byte records from `p` into L2 (a hint).
__device__ __forceinline__ void PrefetchRecords(const void *p, std::uint32_t count) {
  if (count != 0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(count * 16u)
                 : "memory");
}

template <typename Scalar, typename Compute, bool kReverse, int kTeam>
__device__ __forceinline__ void TailTree(const PhaseOps<Scalar, Compute, ForestIndex> &ops,
                                         const PhaseArgs &a, std::uint32_t item) {
  const unsigned lane = threadIdx.x % kTeam;
  const auto sync = [] {
    if constexpr (kTeam == 32)
      __syncwarp();
    else
      __syncthreads();
  };
  const uint4 tree = a.tail_items[item];
  // The walk below is a chain of dependent loads per round; first bring
  // every tail round's records of this tree into L2 (lane e: round e).
  for (std::uint32_t e = lane; e < tree.z; e += kTeam) {
    const uint4 round = a.tail_rounds[tree.y + e];
    const uint2 rakes = a.tail_rakes[tree.y + e];
    PrefetchRecords(a.gathers + round.x, round.y);
    PrefetchRecords(a.compress + round.z, round.w);
    PrefetchRecords(a.rakes + rakes.x, rakes.y);
  }
  for (std::uint32_t e = 0; e < tree.z; ++e) {
    const std::uint32_t at = tree.y + (kReverse ? tree.z - 1 - e : e);
    const uint4 round = a.tail_rounds[at];
    if constexpr (!kReverse) {
      for (std::uint32_t i = lane; i < round.y; i += kTeam)
        ops.Gather(round.x + i);
      sync();
      for (std::uint32_t i = lane; i < round.w; i += kTeam)
        ops.Compress(round.z + i);
      sync();
    } else {
      for (std::uint32_t i = lane; i < round.w; i += kTeam)
        ops.CompressReverse(round.z + i);
      sync();
      const uint2 rakes = a.tail_rakes[at];
      for (std::uint32_t i = lane; i < rakes.y; i += kTeam)
        ops.RakeReverse(rakes.x + i);
      sync();
    }
  }
}

// Kinds that store matrices: whole warps run them.
template <int kKind>
inline constexpr bool kStoresMatrices =
    kKind == kPhaseCompress || kKind == kPhaseRakeReverse || kKind == kPhaseCompressReverse;

template <typename Scalar, typename Compute, class Index, int kKind>
__device__ __forceinline__ void RunOp(const PhaseArgs &args, const Index &index,
                                      std::uint32_t i, std::uint32_t value, bool live) {
  constexpr bool kTogether =
      kStoresMatrices<kKind> && sizeof(Scalar) == 4 && sizeof(Compute) == 4;
  __shared__ __align__(16) float tiles[kTogether ? kPhaseThreads / 32 * kMatrixTile : 1];
  const PhaseOps<Scalar, Compute, Index, kTogether> ops(
      args, index, live, kTogether ? tiles + threadIdx.x / 32 * kMatrixTile : nullptr);
  if constexpr (kKind == kPhaseGather)
    ops.Gather(i);
  else if constexpr (kKind == kPhaseCompress)
    ops.Compress(i);
  else if constexpr (kKind == kPhaseFinish)
    ops.Finish(i, value);
  else if constexpr (kKind == kPhaseRakeReverse)
    ops.RakeReverse(i);
  else if constexpr (kKind == kPhaseCompressReverse)
    ops.CompressReverse(i);
}

// Minimum resident blocks per SM (a register cap) of the kind that would
// otherwise take a few registers too many for one more block.
template <typename Scalar, typename Compute, int kKind, bool kBatch>
inline constexpr int kPhaseMinBlocks =
    kKind == kPhaseCompressReverse && sizeof(Compute) == 4 ? (kBatch ? 6 : 7) : 0;

// Forest layout: thread t runs operation offset + t (finish: instance), or
// team w of kTeam threads the tail of tree offset + w.
template <typename Scalar, typename Compute, int kKind, int kTeam = 1>
__global__ void
__launch_bounds__(kPhaseThreads, kPhaseMinBlocks<Scalar, Compute, kKind, false>)
    PhaseKernel(PhaseArgs args) {
  if constexpr (kKind == kPhaseTailForward || kKind == kPhaseTailReverse) {
    const std::uint32_t w = blockIdx.x * (kPhaseThreads / kTeam) + threadIdx.x / kTeam;
    if (w >= args.count)
      return;
    const PhaseOps<Scalar, Compute, ForestIndex> ops(args, ForestIndex{});
    TailTree<Scalar, Compute, kKind == kPhaseTailReverse, kTeam>(ops, args, args.offset + w);
  } else {
    const std::uint32_t t = blockIdx.x * kPhaseThreads + threadIdx.x;
    if ((kStoresMatrices<kKind> ? t & ~31u : t) >= args.count)
      return;
    const bool live = t < args.count; // a lane past the end repeats the last operation
    const std::uint32_t i = args.offset + (live ? t : args.count - 1);
    RunOp<Scalar, Compute, ForestIndex, kKind>(args, ForestIndex{}, i, i, live);
  }
}

// Shared-topology layout: thread t runs operation offset + t / items of
// batch item first_item + t % items (finish: the root record for that item).
template <typename Scalar, typename Compute, int kKind>
__global__ void __launch_bounds__(kPhaseThreads, kPhaseMinBlocks<Scalar, Compute, kKind, true>)
    BatchPhaseKernel(PhaseArgs args) {
  // Below 2^31 in all (the record index limit).
  const std::uint32_t total = args.count * args.items;
  std::uint32_t t = blockIdx.x * kPhaseThreads + threadIdx.x;
  if ((kStoresMatrices<kKind> ? t & ~31u : t) >= total)
    return;
  const bool live = t < total;
  t = live ? t : total - 1;
  BatchIndex index;
  index.item = args.first_item + t % args.items;
  index.stride = args.item_stride;
  index.nodes = args.item_nodes;
  index.edges = args.item_edges;
  const std::uint32_t i = args.offset + t / args.items;
  RunOp<Scalar, Compute, BatchIndex, kKind>(args, index, i, index.item, live);
}

} // namespace thmm

#endif // THMM_PHASE_ENGINE_CUH_
