// Phase kernels of the level-synchronous schedule (phase.h) for 4 < K <= 32
// states: one lane group of G = 8, 16 or 32 lanes per operation, the
// operation's K x K matrices in shared memory, products in register tiles.
//
// Each operation performs exactly the floating-point operations of the
// lane-group (G > 1) branch of LinearEngine (engine.cuh), every sum in the
// same order, so the phase and per-tree schedules agree bit for bit; as in the
// K <= 4 phase kernels only the bookkeeping of the power-of-two exponents
// differs (carried per stored object here, summed per team there; both are
// exact integer sums). Which lane forms which element is free, and that is
// where the time went: with lane r holding row r, a K = 20 product took 100
// broadcast loads and 20 rows of register traffic per lane, 20 of 32 lanes
// worked, and the edge adjoints left by 4-byte stores 80 bytes apart.
//
// What bounds them now: shared-memory loads and multiply-adds, then DRAM.
//   * A matrix arrives by asynchronous 16-byte copies (cp.async) in the
//     caller's row-major order: coalesced, no registers held while in flight.
//   * Lane (ti, tj) of the group owns TR x 4 elements of a product and reads
//     16-byte quads: TR + 4 of them per TR x 4 x 4 multiply-adds. At K = 20,
//     25 lanes own 4 x 4 tiles and a product takes 40 loads and 320
//     multiply-adds per lane.
//   * Row pitches P with P / 4 odd make the quads of consecutive rows fall on
//     different banks; a lane's rows are RG apart for the same reason.
//   * Adjoints are formed in place in shared memory and leave in 16-byte
//     coalesced stores.
// Measured on one GB300, rows per lane -> tiles: one reverse compression
// launch list of 256 recursive trees x 5000 nodes at K = 20 3.24 -> 0.79 ms
// (some 6,900 -> 1,500 warp instructions each), compressions 1.03 -> 0.28 ms,
// rake adjoints 1.68 -> 0.71 ms (5.4 TB/s), gathers 0.91 -> 0.61 ms; that
// marginal step 6.65 -> 2.23 ms. The batch API, 500 items on a 399-node tree
// at K = 20, 1.62 -> 0.40 ms (the per-tree engine before).
//
// Both layouts of phase_engine.cuh: a forest (every tree's records, one item)
// and the batch API's shared topology (one tree's records, stored objects
// item-minor, the groups of a warp on consecutive items of one operation). No
// tail kinds: every round runs grid-wide.
#ifndef THMM_PHASE_GROUPS_CUH_
#define THMM_PHASE_GROUPS_CUH_

#include <cstdint>
#include <cuda_runtime.h>

#include "engine.cuh"
#include "phase.h"

namespace thmm {

constexpr int kGroupPhaseThreads = 128;

// Tile shape for padded state count KMAX (a multiple of 4): KMAX / 4 column
// quads times RG row groups of TR rows fit the G lanes.
template <int KMAX> struct GroupTile {
  static constexpr int G = GroupLanes<KMAX>();
  static constexpr int CQ = KMAX / 4;
  static constexpr int TR = KMAX <= 8 ? 2 : KMAX <= 20 ? 4 : 8;
  static constexpr int RG = (KMAX + TR - 1) / TR;
  static constexpr int kRows = RG * TR;
  static constexpr int P = (kRows / 4) % 2 == 1 ? kRows : kRows + 4;
  static constexpr int kMatrix = kRows * P; // elements of one matrix buffer
  static_assert(RG * CQ <= G && G >= KMAX, "tiles and rows fit the group");
};

// Elements of shared memory per lane group.
template <int KMAX, int kKind>
inline constexpr int kGroupPhaseElements =
    kKind == kPhaseGather            ? 2 * (GroupTile<KMAX>::kMatrix + KMAX)
    : kKind == kPhaseRakeReverse     ? GroupTile<KMAX>::kMatrix + 2 * KMAX
    : kKind == kPhaseCompress        ? 2 * GroupTile<KMAX>::kMatrix + KMAX
    : kKind == kPhaseCompressReverse ? 4 * GroupTile<KMAX>::kMatrix + KMAX
                                     : 0;

// Four consecutive values at a 16-byte boundary.
template <typename T> __device__ __forceinline__ void Load4(const T *p, T (&out)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    out[0] = v.x, out[1] = v.y, out[2] = v.z, out[3] = v.w;
  } else {
    const double2 v = reinterpret_cast<const double2 *>(p)[0];
    const double2 w = reinterpret_cast<const double2 *>(p)[1];
    out[0] = v.x, out[1] = v.y, out[2] = w.x, out[3] = w.y;
  }
}
template <bool kStreaming = false, typename D, typename T>
__device__ __forceinline__ void Store4(D *p, const T (&in)[4]) {
  if constexpr (sizeof(D) == 4) {
    const float4 v = make_float4(static_cast<float>(in[0]), static_cast<float>(in[1]),
                                 static_cast<float>(in[2]), static_cast<float>(in[3]));
    if constexpr (kStreaming)
      __stcs(reinterpret_cast<float4 *>(p), v);
    else
      *reinterpret_cast<float4 *>(p) = v;
  } else {
    const double2 v = make_double2(static_cast<double>(in[0]), static_cast<double>(in[1]));
    const double2 w = make_double2(static_cast<double>(in[2]), static_cast<double>(in[3]));
    if constexpr (kStreaming) {
      __stcs(reinterpret_cast<double2 *>(p), v);
      __stcs(reinterpret_cast<double2 *>(p) + 1, w);
    } else {
      reinterpret_cast<double2 *>(p)[0] = v;
      reinterpret_cast<double2 *>(p)[1] = w;
    }
  }
}

// Asynchronous global -> shared copies of 4, 8 or 16 bytes; of 16 past L1 unless
// the source is shared.
template <int kBytes, bool kShared = false>
__device__ __forceinline__ void CopyAsync(void *dst, const void *src) {
  const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  if constexpr (kBytes == 16 && !kShared)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(at), "l"(src), "n"(kBytes)
                 : "memory");
}
__device__ __forceinline__ void CopyCommit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int kPending> __device__ __forceinline__ void CopyWait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// Variants. In single precision K == KMAX has one for each layout, so that the
// compiler folds the bounds and the strides, and the general one has K < KMAX; in
// double the general one is the only one.
enum GroupForm : int { kGeneralForm = 0, kForestForm = 1, kBatchForm = 2 };

template <typename Scalar, typename Compute, int KMAX, int kForm> struct GroupPhaseOps {
  static constexpr bool kExact = kForm != kGeneralForm;
  using Tile = GroupTile<KMAX>;
  static constexpr int G = Tile::G, CQ = Tile::CQ, TR = Tile::TR, RG = Tile::RG, P = Tile::P;
  const PhaseArgs &a;
  unsigned K;
  unsigned KK;
  unsigned inverse;   // i / K = i * inverse >> 16 for i < K * K (K <= 32)
  std::size_t item;   // batch item (0 for a forest)
  std::size_t stride; // items per stored object (1 for a forest)
  unsigned lane;      // lane within the group
  unsigned mask;      // the group's lanes of the warp
  unsigned ti, tj;    // this lane's tile (ti < RG for lanes that own one)
  Compute *smem;      // the group's shared memory

  __device__ __forceinline__ GroupPhaseOps(const PhaseArgs &args, std::uint32_t batch_item,
                                           Compute *group_smem)
      : a(args), K(kExact ? KMAX : args.states), KK(K * K), inverse(65536u / K + 1u),
        item(batch_item), stride(args.item_stride), lane(threadIdx.x % G),
        mask(G == 32 ? kFull : ((1u << (G & 31)) - 1u) << (threadIdx.x % 32 / G * G)),
        ti(lane / CQ), tj(lane % CQ), smem(group_smem) {}

  // K == KMAX: rows of whole 16-byte quads.
  __device__ __forceinline__ bool Whole() const {
    return kExact || (sizeof(Compute) == 8 && K == KMAX);
  }
  __device__ __forceinline__ std::size_t Store(std::uint32_t object) const {
    return object * stride + item;
  }
  __device__ __forceinline__ std::size_t Io(std::uint32_t node) const {
    return item * a.item_nodes + node;
  }
  __device__ __forceinline__ Compute *NodeAt(std::uint32_t node) const {
    return static_cast<Compute *>(a.nodes) + Store(node) * K;
  }
  __device__ __forceinline__ Scalar *NodeOutAt(std::uint32_t node) const {
    return static_cast<Scalar *>(a.node_out) + Io(node) * K;
  }
  __device__ __forceinline__ Compute *CompAt(std::uint32_t tape) const {
    return static_cast<Compute *>(a.comps) + Store(tape) * KK;
  }
  __device__ __forceinline__ Compute *CompMuAt(std::uint32_t tape) const {
    return static_cast<Compute *>(a.comp_mu) + Store(tape) * KK;
  }
  __device__ __forceinline__ const Scalar *EdgeAt(std::uint32_t edge) const {
    return static_cast<const Scalar *>(a.edge_in) + static_cast<std::size_t>(edge) * KK;
  }

  // Element j < K of `node`'s input factor: dense row, or the reference's
  // categorical (root ? root_potential : 1) * emission[observation]
  // (src/gpu_backend_impl.inc:326-382), as Context::InputNode.
  __device__ __forceinline__ Scalar Input(std::uint32_t node, std::uint32_t obs, bool root,
                                          unsigned j) const {
    if (!a.categorical)
      return static_cast<const Scalar *>(a.node_in)[Io(node) * K + j];
    const Scalar *root_potential = static_cast<const Scalar *>(a.root_potential);
    if (obs == kNone)
      return root ? root_potential[j] : Scalar(1);
    const unsigned category = a.observations[Store(obs)];
    if (category >= a.categories)
      return Scalar(0);
    const Scalar emitted = static_cast<const Scalar *>(a.emission)[category * K + j];
    return root ? root_potential[j] * emitted : emitted;
  }
  // Element `lane` of a rake leaf or compression middle (0 past K): the
  // stored value (adding its exponent to `e`) or the input factor.
  __device__ __forceinline__ Compute Node(std::uint32_t ref, std::uint32_t obs, int &e) const {
    if (ref & kFlag) {
      e += a.node_exp[Store(ref & kMask)];
      return lane < K ? NodeAt(ref & kMask)[lane] : Compute(0);
    }
    return lane < K ? static_cast<Compute>(Input(ref, obs, false, lane)) : Compute(0);
  }
  __device__ __forceinline__ int PathExp(std::uint32_t ref) const {
    return (ref & kFlag) ? a.comp_exp[Store(ref & kMask)] : 0;
  }
  __device__ __forceinline__ static int Exponent(Compute m) {
    return m > Compute(0) ? Pow2Exponent(m) : 0;
  }
  __device__ __forceinline__ Compute Max(Compute v) const {
#pragma unroll
    for (int offset = G / 2; offset > 0; offset >>= 1) {
      const Compute other = __shfl_xor_sync(mask, v, offset, G);
      v = v < other ? other : v;
    }
    return v;
  }

  // ------------------------------------------------ matrices and shared memory
  // Zero padding of a matrix buffer whose K is below KMAX (the copies write
  // rows and columns below K only).
  __device__ __forceinline__ void ClearPadding(Compute *m) const {
    if (!Whole())
      for (unsigned i = lane; i < Tile::kMatrix; i += G)
        m[i] = Compute(0);
  }
  // Starts copying a K x K matrix into `m` (pitch P); complete after
  // CopyCommit, CopyWait and a group barrier.
  template <bool kShared, typename T>
  __device__ __forceinline__ void StageWhole(const T *src, Compute *m) const {
    constexpr int kQuads = KMAX * CQ;
#pragma unroll
    for (int first = 0; first < kQuads; first += G) {
      const unsigned q = first + lane;
      if (kQuads % G == 0 || q < kQuads) {
        Compute *dst = m + (q / CQ) * P + 4 * (q % CQ);
        if constexpr (sizeof(T) == sizeof(Compute)) {
#pragma unroll
          for (unsigned part = 0; part < sizeof(T) / 4; ++part)
            CopyAsync<16, kShared>(dst + part * 2, src + 4 * q + part * 2);
        } else {
          T in[4];
          Load4(src + 4 * q, in);
          const Compute out[4] = {static_cast<Compute>(in[0]), static_cast<Compute>(in[1]),
                                  static_cast<Compute>(in[2]), static_cast<Compute>(in[3])};
          Store4(dst, out);
        }
      }
    }
  }
  // The same for K < KMAX, element by element. Each place is found by itself and
  // eight are under way at a time: a gather's rakes are a chain, and a division,
  // dependent places and (for inputs of another width) one load after the other were
  // a quarter of its link (log Z of a star of 998 leaves, K = 7, 922 -> 700 us a call,
  // with double inputs 1,772 -> 1,335).
  template <typename T>
  __device__ __forceinline__ void StagePadded(const T *src, Compute *m) const {
    constexpr int kSteps = (KMAX * KMAX + G - 1) / G;
#pragma unroll 8
    for (int step = 0; step < kSteps; ++step) {
      const unsigned i = lane + step * G;
      if (i < KK) {
        Compute *dst = m + i + (i * inverse >> 16) * (P - K); // row r at r * P
        if constexpr (sizeof(T) == sizeof(Compute))
          CopyAsync<sizeof(T)>(dst, src + i);
        else
          *dst = static_cast<Compute>(src[i]);
      }
    }
  }
  template <bool kShared, typename T>
  __device__ __forceinline__ void StageFrom(const T *src, Compute *m) const {
    if (Whole())
      StageWhole<kShared>(src, m);
    else
      StagePadded(src, m);
  }
  // An edge of the batch layout comes through L1: every group of an SM reads the
  // same few, and past L1 all SMs queue for the same lines of L2 (the one gather
  // launch of 8,192 items of 3 nodes at K = 8 51.6 -> 5.3 us). A forest's edges are
  // read once, and L1 only delays them (256 trees of 5,000 nodes, K = 20, 2,123 ->
  // 2,159 us).
  __device__ __forceinline__ void Stage(std::uint32_t ref, Compute *m) const {
    // Edges of another width are converted, through registers.
    constexpr bool kSame = sizeof(Scalar) == sizeof(Compute);
    if (ref & kFlag)
      StageFrom<false>(static_cast<const Compute *>(CompAt(ref & kMask)), m);
    else if (kSame && (kForm == kBatchForm || (kForm == kGeneralForm && Whole() && a.batch != 0)))
      StageFrom<true>(EdgeAt(ref), m);
    else
      StageFrom<false>(EdgeAt(ref), m);
  }
  // Writes the K x K matrix in `m` out, transformed element by element
  // (value, row, column).
  template <bool kStreaming, typename T, class Map>
  __device__ __forceinline__ void Drain(const Compute *m, T *dst, Map map) const {
    if (Whole()) {
      constexpr int kQuads = KMAX * CQ;
#pragma unroll
      for (int first = 0; first < kQuads; first += G) {
        const unsigned q = first + lane;
        if (kQuads % G == 0 || q < kQuads) {
          const unsigned r = q / CQ, c = 4 * (q % CQ);
          Compute v[4];
          Load4(m + r * P + c, v);
          map(v, r, c);
          Store4<kStreaming>(dst + 4 * q, v);
        }
      }
    } else {
      unsigned r = lane / K, c = lane % K;
      const unsigned step_r = G / K, step_c = G % K;
      for (unsigned i = lane; i < KK; i += G) {
        Compute v[1] = {m[r * P + c]};
        map(v, r, c);
        if constexpr (kStreaming)
          __stcs(dst + i, static_cast<T>(v[0]));
        else
          dst[i] = static_cast<T>(v[0]);
        r += step_r;
        c += step_c;
        if (c >= K) {
          c -= K;
          ++r;
        }
      }
    }
  }
  // The adjoint of path `ref` (a compressed path's stays, an edge's is the
  // caller's marginal).
  template <class Map>
  __device__ __forceinline__ void DrainAdjoint(std::uint32_t ref, const Compute *m,
                                               Map map) const {
    if (ref & kFlag)
      Drain<false>(m, CompMuAt(ref & kMask), map);
    else
      Drain<true>(m,
                  static_cast<Scalar *>(a.edge_out) +
                      (item * a.item_edges + ref) * static_cast<std::size_t>(KK),
                  map);
  }

  // Row `lane` of `m` times `x`, terms in order.
  __device__ __forceinline__ Compute RowDot(const Compute *m, const Compute *x) const {
    Compute dot = Compute(0);
    const Compute *row = m + (lane < KMAX ? lane : 0u) * P;
#pragma unroll
    for (unsigned j = 0; j < KMAX; j += 4) {
      if (j < K) {
        Compute u[4], v[4];
        Load4(row + j, u);
        Load4(x + j, v);
#pragma unroll
        for (int d = 0; d < 4; ++d)
          dot = fma(u[d], v[d], dot);
      }
    }
    return dot;
  }

  // ---------------------------------------------------------- forward
  // Rakes of gather i absorbed into its parent (LinearEngine::AbsorbRake):
  // lane r holds element r of the parent's value. The next rake's matrix and
  // leaf are on their way while this one is worked on.
  __device__ __forceinline__ void Gather(std::uint32_t i) const {
    const uint4 op = a.gathers[i];
    const std::uint32_t node = op.x & kMask;
    const std::uint32_t count = op.w & kCountMask;
    // Two buffers of a matrix and a leaf vector each.
    const auto matrix = [&](unsigned at) { return smem + at * Tile::kMatrix; };
    const auto leaf = [&](unsigned at) { return smem + 2 * Tile::kMatrix + at * KMAX; };
    uint4 rake = a.rakes[op.z];
    ClearPadding(matrix(0));
    ClearPadding(matrix(1));
    __syncwarp(mask);
    int next_exp = PathExp(rake.x);
    Stage(rake.x, matrix(0));
    CopyCommit();
    Compute next_leaf = Node(rake.y, rake.z, next_exp);
    if (count > 1)
      rake = a.rakes[op.z + 1];
    Compute v = Compute(0);
    int e = 0;
    if (op.x & kFlag) {
      if (lane < K)
        v = static_cast<Compute>(Input(node, op.y, (op.w & kRootBit) != 0, lane));
    } else {
      if (lane < K)
        v = NodeAt(node)[lane];
      e = a.node_exp[Store(node)];
    }
    for (std::uint32_t k = 0; k < count; ++k) {
      const unsigned at = k & 1u;
      if (lane < KMAX)
        leaf(at)[lane] = next_leaf;
      e += next_exp;
      if (k + 1 < count) {
        next_exp = PathExp(rake.x);
        Stage(rake.x, matrix(at ^ 1u));
        CopyCommit();
        next_leaf = Node(rake.y, rake.z, next_exp);
        if (k + 2 < count)
          rake = a.rakes[op.z + k + 2];
        CopyWait<1>();
      } else {
        CopyWait<0>();
      }
      __syncwarp(mask);
      Compute dot = RowDot(matrix(at), leaf(at));
      if (lane >= K)
        dot = Compute(0);
      const int s1 = Exponent(Max(dot));
      const Compute value = v * ScalePow2(dot, -s1);
      const int s2 = Exponent(Max(value)); // also: every lane is done with matrix(at)
      v = ScalePow2(value, -s2);
      e += s1 + s2;
    }
    if (lane < K)
      NodeAt(node)[lane] = v;
    if (lane == 0)
      a.node_exp[Store(node)] = e;
  }

  // acc[q][c] += sum over d of A[ti + RG q][d] * B[d][4 tj + c].
  __device__ __forceinline__ void Product(const Compute *A, const Compute *B,
                                          Compute (&acc)[TR][4]) const {
    const Compute *rows = A + (ti < RG ? ti : 0u) * P;
    const Compute *columns = B + 4 * tj;
#pragma unroll
    for (unsigned d0 = 0; d0 < KMAX; d0 += 4) {
      if (d0 < K) {
        Compute u[TR][4];
#pragma unroll
        for (int q = 0; q < TR; ++q)
          Load4(rows + q * RG * P + d0, u[q]);
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          Compute w[4];
          Load4(columns + (d0 + d) * P, w);
#pragma unroll
          for (int q = 0; q < TR; ++q)
#pragma unroll
            for (int c = 0; c < 4; ++c)
              acc[q][c] = fma(u[q][d], w[c], acc[q][c]);
        }
      }
    }
  }

  // The weights left[r][m] * middle[m] of a compression, from `left` into
  // `out` (which may be `left`).
  __device__ __forceinline__ void Weigh(const Compute *left, const Compute *middle,
                                        Compute *out) const {
    constexpr int kQuads = KMAX * CQ;
#pragma unroll
    for (int first = 0; first < kQuads; first += G) {
      const unsigned q = first + lane;
      if (kQuads % G == 0 || q < kQuads) {
        const unsigned at = (q / CQ) * P + 4 * (q % CQ);
        Compute v[4], w[4];
        Load4(left + at, v);
        Load4(middle + 4 * (q % CQ), w);
#pragma unroll
        for (int d = 0; d < 4; ++d)
          v[d] = v[d] * w[d];
        Store4(out + at, v);
      }
    }
  }

  // Compressed path i = left * diag(middle) * right.
  __device__ __forceinline__ void Compress(std::uint32_t i) const {
    const uint4 op = a.compress[i];
    Compute *left = smem, *right = smem + Tile::kMatrix, *middle = smem + 2 * Tile::kMatrix;
    ClearPadding(left);
    ClearPadding(right);
    __syncwarp(mask);
    Stage(op.x, left);
    Stage(op.z, right);
    CopyCommit();
    int e = PathExp(op.x) + PathExp(op.z);
    const Compute own = Node(op.y, op.w, e);
    if (lane < KMAX)
      middle[lane] = own;
    CopyWait<0>();
    __syncwarp(mask);
    Weigh(left, middle, left);
    __syncwarp(mask);
    Compute out[TR][4];
#pragma unroll
    for (int q = 0; q < TR; ++q)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        out[q][c] = Compute(0);
    Product(left, right, out);
    Compute m = Compute(0);
#pragma unroll
    for (int q = 0; q < TR; ++q)
      if (ti < RG && ti + q * RG < K)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          m = m < out[q][c] ? out[q][c] : m; // columns past K are zero
    const int s = Exponent(Max(m));
    Compute *dst = CompAt(i);
    if (ti < RG) {
#pragma unroll
      for (int q = 0; q < TR; ++q) {
        const unsigned r = ti + q * RG;
        if (r < K) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            out[q][c] = ScalePow2(out[q][c], -s);
          if (Whole()) {
            Store4(dst + r * KMAX + 4 * tj, out[q]);
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (4 * tj + c < K)
                dst[r * K + 4 * tj + c] = out[q][c];
          }
        }
      }
    }
    if (lane == 0)
      a.comp_exp[Store(i)] = e + s;
  }

  // log Z = ln 2 * (root exponent) + log(sum(root)), as LinearEngine::Run: root
  // record i, result of instance `value`. With marginals to come a group per
  // instance: every lane forms the sum, lane j divides for state j (FP64 divisions
  // one after the other in one thread took most of the launch's 14 us at K = 20).
  // Without them a thread per instance: the FP64 logarithm once and not per lane
  // (log Z of 5,000 trees of 3 nodes at K = 20, 159 -> 137 us a call).
  __device__ __forceinline__ void Finish(std::uint32_t i, std::uint32_t value) const {
    const uint2 rec = a.roots[i];
    const std::uint32_t node = rec.x & kMask;
    Compute root[KMAX];
    long long total = 0;
    if (rec.x & kFlag) {
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        root[j] = j < K ? NodeAt(node)[j] : Compute(0);
      total = a.node_exp[Store(node)];
    } else {
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        root[j] = j < K ? static_cast<Compute>(Input(node, rec.y, true, j)) : Compute(0);
    }
    double sum = 0.0;
    for (unsigned j = 0; j < KMAX; ++j)
      sum += static_cast<double>(root[j]);
    const double log_z = !(sum > 0.0)
                             ? -INFINITY
                             : fma(static_cast<double>(total), 0.6931471805599453094, log(sum));
    if (lane == 0 || !a.reverse)
      static_cast<Scalar *>(a.values)[value] = static_cast<Scalar>(a.raw ? exp(log_z) : log_z);
    if (a.reverse && lane < K) {
      const double own = static_cast<double>(Select(root, lane));
      NodeOutAt(node)[lane] = static_cast<Scalar>(log_z > -INFINITY ? own / sum : 0.0);
    }
  }

  // ---------------------------------------------------------- adjoint
  __device__ __forceinline__ void RakeReverse(std::uint32_t i) const {
    const uint4 op = a.rakes[i];
    Compute *matrix = smem, *leaf = smem + Tile::kMatrix, *ratio = leaf + KMAX;
    ClearPadding(matrix);
    __syncwarp(mask);
    Stage(op.x, matrix);
    CopyCommit();
    int unused = 0;
    const Compute own = Node(op.y, op.z, unused);
    const Compute parent_adjoint =
        lane < K ? static_cast<Compute>(NodeOutAt(op.w)[lane]) : Compute(0);
    if (lane < KMAX)
      leaf[lane] = own;
    CopyWait<0>();
    __syncwarp(mask);
    const Compute unnormalised = RowDot(matrix, leaf);
    if (lane < KMAX)
      ratio[lane] = lane < K && unnormalised > Compute(0) ? parent_adjoint / unnormalised
                                                          : Compute(0);
    __syncwarp(mask);
    // Edge adjoint: ratio[r] * path[r][c] * leaf[c].
    DrainAdjoint(op.x, matrix, [&](auto &v, unsigned r, unsigned c) {
      const Compute ratio_r = ratio[r];
#pragma unroll
      for (unsigned d = 0; d < sizeof(v) / sizeof(v[0]); ++d)
        v[d] = ratio_r * v[d] * leaf[c + d];
    });
    // Leaf adjoint: leaf[j] * sum_p ratio_p * path[p][j].
    Compute column = Compute(0);
    const Compute *down = matrix + (lane < KMAX ? lane : 0u);
#pragma unroll
    for (unsigned p = 0; p < KMAX; p += 4) {
      if (p < K) {
        Compute u[4];
        Load4(ratio + p, u);
#pragma unroll
        for (int d = 0; d < 4; ++d)
          column = fma(u[d], down[(p + d) * P], column);
      }
    }
    if (lane < K)
      NodeOutAt(op.y & kMask)[lane] = static_cast<Scalar>(own * column);
  }

  // Adjoint of compression i.
  __device__ __forceinline__ void CompressReverse(std::uint32_t i) const {
    const uint4 op = a.compress[i];
    Compute *left = smem, *right = left + Tile::kMatrix, *weight = right + Tile::kMatrix,
            *ratio = weight + Tile::kMatrix, *middle = ratio + Tile::kMatrix;
    ClearPadding(left);
    ClearPadding(right);
    ClearPadding(ratio);
    __syncwarp(mask);
    Stage(op.x, left);
    Stage(op.z, right);
    CopyCommit();
    // The output's adjoint, in this lane's product tile.
    const Compute *output_adjoint = CompMuAt(i);
    Compute adjoint[TR][4];
#pragma unroll
    for (int q = 0; q < TR; ++q) {
      const unsigned r = ti + q * RG;
      if (Whole() && ti < RG && (RG * TR == KMAX || r < K)) {
        Load4(output_adjoint + r * KMAX + 4 * tj, adjoint[q]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          adjoint[q][c] = ti < RG && r < K && 4 * tj + c < K
                              ? output_adjoint[r * K + 4 * tj + c]
                              : Compute(0);
      }
    }
    int unused = 0;
    const Compute own = Node(op.y, op.w, unused);
    if (lane < KMAX)
      middle[lane] = own;
    CopyWait<0>();
    __syncwarp(mask);
    Weigh(left, middle, weight);
    __syncwarp(mask);
    // Unnormalised output, recomputed with the forward's operation order, and
    // ratio = adjoint / output.
    Compute acc[TR][4];
#pragma unroll
    for (int q = 0; q < TR; ++q)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        acc[q][c] = Compute(0);
    Product(weight, right, acc);
#pragma unroll
    for (int q = 0; q < TR; ++q) {
      const unsigned r = ti + q * RG;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        acc[q][c] = acc[q][c] > Compute(0) ? adjoint[q][c] / acc[q][c] : Compute(0);
      if (ti < RG && r < K)
        Store4(ratio + r * P + 4 * tj, acc[q]);
    }
    __syncwarp(mask);
    // Left adjoint: left[r][m] middle[m] sum_j right[m][j] ratio[r][j], this
    // lane's elements r = ti + RG q, m = tj + CQ c, in place of the weights.
#pragma unroll
    for (int q = 0; q < TR; ++q)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        acc[q][c] = Compute(0);
    {
      const Compute *rows = ratio + (ti < RG ? ti : 0u) * P;
      const Compute *columns = right + tj * P;
#pragma unroll
      for (unsigned d0 = 0; d0 < KMAX; d0 += 4) {
        if (d0 < K) {
          Compute u[TR][4];
#pragma unroll
          for (int q = 0; q < TR; ++q)
            Load4(rows + q * RG * P + d0, u[q]);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            Compute w[4];
            Load4(columns + c * CQ * P + d0, w);
#pragma unroll
            for (int q = 0; q < TR; ++q)
#pragma unroll
              for (int d = 0; d < 4; ++d)
                acc[q][c] = fma(w[d], u[q][d], acc[q][c]);
          }
        }
      }
    }
    if (ti < RG) {
#pragma unroll
      for (int q = 0; q < TR; ++q) {
        const unsigned r = ti + q * RG;
        if (RG * TR == KMAX || r < KMAX)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            Compute *w = weight + r * P + tj + CQ * c;
            *w = *w * acc[q][c];
          }
      }
    }
    // Right adjoint: right[m][j] middle[m] sum_p left[p][m] ratio[p][j], this
    // lane's elements m = TR ti + q, j = 4 tj + c, in place of the right factor.
#pragma unroll
    for (int q = 0; q < TR; ++q)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        acc[q][c] = Compute(0);
    {
      const unsigned m0 = TR * (ti < RG ? ti : 0u);
#pragma unroll 4
      for (unsigned p = 0; p < K; ++p) {
        Compute u[TR], w[4];
        if constexpr (TR >= 4) {
#pragma unroll
          for (int part = 0; part < TR; part += 4) {
            Compute four[4];
            Load4(left + p * P + m0 + part, four);
#pragma unroll
            for (int d = 0; d < 4; ++d)
              u[part + d] = four[d];
          }
        } else {
#pragma unroll
          for (int q = 0; q < TR; ++q)
            u[q] = left[p * P + m0 + q];
        }
        Load4(ratio + p * P + 4 * tj, w);
#pragma unroll
        for (int q = 0; q < TR; ++q)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            acc[q][c] = fma(u[q], w[c], acc[q][c]);
      }
      __syncwarp(mask); // every lane is done with right, and weight is written
      if (ti < RG) {
#pragma unroll
        for (int q = 0; q < TR; ++q) {
          const unsigned m = m0 + q;
          if (RG * TR == KMAX || m < KMAX) {
            Compute v[4];
            Load4(right + m * P + 4 * tj, v);
            const Compute middle_m = middle[m];
#pragma unroll
            for (int c = 0; c < 4; ++c)
              v[c] = v[c] * middle_m * acc[q][c];
            Store4(right + m * P + 4 * tj, v);
          }
        }
      }
    }
    const auto same = [](auto &, unsigned, unsigned) {};
    DrainAdjoint(op.x, weight, same);
    __syncwarp(mask);
    DrainAdjoint(op.z, right, same);
    // Middle adjoint: the right adjoint's row sums.
    if (lane < K) {
      Compute total = Compute(0);
#pragma unroll
      for (unsigned j = 0; j < KMAX; j += 4) {
        if (j < K) {
          Compute v[4];
          Load4(right + lane * P + j, v);
#pragma unroll
          for (int d = 0; d < 4; ++d)
            total += v[d];
        }
      }
      NodeOutAt(op.y & kMask)[lane] = static_cast<Scalar>(total);
    }
  }
};

// Minimum resident blocks per SM (a register cap of 65536 / (128 n) per
// thread), chosen so that no FP32 variant spills.
template <int KMAX, bool kWide> constexpr int GroupPhaseMinBlocks(int kind) {
  if (kWide)
    return KMAX <= 16 ? 3 : 2;
  return kind == kPhaseCompressReverse ? (KMAX <= 8 ? 6 : KMAX <= 20 ? 5 : 3)
                                       : (KMAX <= 20 ? 8 : 5);
}

// One kind of one round: lane group g of the grid runs operation offset + g /
// items of item first_item + g % items (finish: the root record).
template <typename Scalar, typename Compute, int KMAX, int kKind, int kForm>
__global__ void __launch_bounds__(kGroupPhaseThreads,
                                  GroupPhaseMinBlocks<KMAX, sizeof(Compute) == 8>(kKind))
    GroupPhaseKernel(PhaseArgs args) {
  using Ops = GroupPhaseOps<Scalar, Compute, KMAX, kForm>;
  constexpr int G = Ops::G;
  constexpr int kElements = kGroupPhaseElements<KMAX, kKind>;
  extern __shared__ __align__(16) unsigned char group_smem[];
  const std::uint64_t t =
      static_cast<std::uint64_t>(blockIdx.x) * kGroupPhaseThreads + threadIdx.x;
  const bool alone = kKind == kPhaseFinish && !args.reverse; // a thread per instance
  // Below 2^31 (the record index limit).
  const auto g = static_cast<std::uint32_t>(alone ? t : t / G);
  if (g >= args.count * args.items)
    return;
  std::uint32_t op = g, item = 0;
  if (args.batch) {
    op = g / args.items;
    item = args.first_item + g % args.items;
  }
  const std::uint32_t i = args.offset + op;
  const Ops ops(args, item,
                reinterpret_cast<Compute *>(group_smem) + threadIdx.x / G * kElements);
  if constexpr (kKind == kPhaseFinish)
    ops.Finish(i, args.batch ? item : i);
  else if constexpr (kKind == kPhaseGather)
    ops.Gather(i);
  else if constexpr (kKind == kPhaseCompress)
    ops.Compress(i);
  else if constexpr (kKind == kPhaseRakeReverse)
    ops.RakeReverse(i);
  else if constexpr (kKind == kPhaseCompressReverse)
    ops.CompressReverse(i);
}

} // namespace thmm

#endif // THMM_PHASE_GROUPS_CUH_
