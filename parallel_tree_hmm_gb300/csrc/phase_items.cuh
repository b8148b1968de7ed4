// Rakes of the batch API's first round for 4 < K <= 32 states in single
// precision: one batch item per lane (phase_groups.cuh has the other rounds).
//
// Every path of the first round is an input edge, which all items share, so 32
// items of one operation read the same matrix. The lane-group form spends some
// 270 warp instructions per rake and item, of which 20 are multiply-adds: it
// stages the shared matrix and reduces over its lanes anew for every item. Here
// lane l holds the vectors of item l, a warp stages the matrix once for its 32
// items (a gather's next one by cp.async while this one is worked on), all
// lanes read the same quad at once, and maxima and exponents are a thread's own.
// At K = 20 a gather of two rakes takes 45 instead of 540 warp instructions per
// item. Compressed paths differ from item to item, so later rounds, which read
// them, stay with the lane groups.
// What bounds them then: a warp's own chain, and the edge marginals, which leave
// through shared memory so that a warp writes runs of several rows of one item's
// matrix and not 16 bytes in 32 places.
//
// Measured on one GB300, 500 items of a 399-node tree at K = 20, lane groups ->
// these kernels: first round's gathers 53 -> 12 us, its rake adjoints 74 -> 46
// us (2.7 TB/s, mostly written); the marginals 370 -> 311 us a step.
//
// Each operation performs the floating-point operations of the lane-group form
// in the same order (products along a row in ascending columns, column sums in
// ascending rows, maxima in any order), so the bits are the same.
#ifndef THMM_PHASE_ITEMS_CUH_
#define THMM_PHASE_ITEMS_CUH_

#include "phase_groups.cuh"

namespace thmm {

constexpr int kItemPhaseThreads = 128;

// Rows of an edge marginal that a warp collects before it writes them.
template <int KMAX> inline constexpr int kItemRows = KMAX <= 8 ? 4 : KMAX <= 28 ? 2 : 1;
// A lane's rows in shared memory; an odd number of quads, so that the 16-byte
// stores of consecutive lanes fall on different banks.
template <int KMAX> inline constexpr int kItemPitch = kItemRows<KMAX> * KMAX + 4;
// Shared memory of a warp: two paths (gather), or a path and the lanes' rows.
template <int KMAX, int kKind>
inline constexpr int kItemElements =
    KMAX * KMAX + (kKind == kPhaseGather ? KMAX * KMAX : 32 * kItemPitch<KMAX>);

template <typename Scalar, int KMAX, bool kExact> struct ItemPhaseOps {
  static constexpr int kRows = kItemRows<KMAX>;
  static constexpr int kPitch = kItemPitch<KMAX>;
  static_assert(kPitch / 4 % 2 == 1 && KMAX % 4 == 0, "bank-conflict-free rows");
  const PhaseArgs &a;
  unsigned K, KK;
  unsigned lane;
  std::size_t item;  // this lane's batch item
  std::size_t first; // the warp's
  unsigned items;    // the warp's live items (the other lanes repeat the last)
  float *paths;      // the warp's staged paths, KMAX * KMAX floats each
  float *tile;       // the warp's 32 * kPitch floats (adjoint)

  __device__ __forceinline__ ItemPhaseOps(const PhaseArgs &args, std::uint32_t first_item,
                                          unsigned live_items, float *warp_smem)
      : a(args), K(kExact ? KMAX : args.states), KK(K * K), lane(threadIdx.x & 31u),
        item(first_item + (lane < live_items ? lane : live_items - 1)), first(first_item),
        items(live_items), paths(warp_smem), tile(warp_smem + KMAX * KMAX) {}

  __device__ __forceinline__ std::size_t Store(std::uint32_t object) const {
    return object * a.item_stride + item;
  }

  // K values at p, as floats (zeros past K). Rows of K == KMAX values are whole
  // aligned quads.
  template <typename T>
  __device__ __forceinline__ void Load(const T *p, float (&out)[KMAX]) const {
    if constexpr (kExact) {
#pragma unroll
      for (int j = 0; j < KMAX; j += 4) {
        T v[4];
        Load4(p + j, v);
#pragma unroll
        for (int d = 0; d < 4; ++d)
          out[j + d] = static_cast<float>(v[d]);
      }
    } else {
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        out[j] = j < K ? static_cast<float>(p[j]) : 0.0f;
    }
  }

  // Input factor of `node`, as GroupPhaseOps::Input.
  __device__ __forceinline__ void Input(std::uint32_t node, std::uint32_t obs, bool root,
                                        float (&out)[KMAX]) const {
    if (!a.categorical) {
      Load(static_cast<const Scalar *>(a.node_in) + (item * a.item_nodes + node) * K, out);
      return;
    }
    const Scalar *root_potential = static_cast<const Scalar *>(a.root_potential);
    const unsigned category = obs != kNone ? a.observations[Store(obs)] : 0u;
    const Scalar *emission = static_cast<const Scalar *>(a.emission) + category * K;
#pragma unroll
    for (unsigned j = 0; j < KMAX; ++j) {
      Scalar value = j < K ? Scalar(1) : Scalar(0);
      if (j < K && obs != kNone)
        value = category < a.categories ? emission[j] : Scalar(0);
      if (j < K && root && (obs == kNone || category < a.categories))
        value = obs == kNone ? root_potential[j] : root_potential[j] * value;
      out[j] = static_cast<float>(value);
    }
  }
  // The value of a rake leaf (adding its exponent to `e`).
  __device__ __forceinline__ void Node(std::uint32_t ref, std::uint32_t obs, float (&out)[KMAX],
                                       int &e) const {
    if (ref & kFlag) {
      const std::size_t at = Store(ref & kMask);
      e += a.node_exp[at];
      Load(static_cast<const float *>(a.nodes) + at * K, out);
    } else {
      Input(ref, obs, false, out);
    }
  }
  __device__ __forceinline__ const Scalar *EdgeAt(std::uint32_t edge) const {
    return static_cast<const Scalar *>(a.edge_in) + static_cast<std::size_t>(edge) * KK;
  }
  // Starts copying a path, rows KMAX apart; there after CopyCommit, CopyWait and
  // __syncwarp. Zero columns past K come from Clear.
  __device__ __forceinline__ void Stage(std::uint32_t edge, float *dst) const {
    const Scalar *src = EdgeAt(edge);
    if constexpr (kExact) {
      constexpr unsigned kQuads = KMAX * KMAX / 4;
#pragma unroll
      for (unsigned at = 0; at < kQuads; at += 32) {
        const unsigned q = at + lane;
        if (kQuads % 32 == 0 || q < kQuads) {
          if constexpr (sizeof(Scalar) == 4) {
            CopyAsync<16, true>(dst + 4 * q, src + 4 * q);
          } else {
            Scalar in[4];
            Load4(src + 4 * q, in);
            const float out[4] = {static_cast<float>(in[0]), static_cast<float>(in[1]),
                                  static_cast<float>(in[2]), static_cast<float>(in[3])};
            Store4(dst + 4 * q, out);
          }
        }
      }
    } else {
      unsigned r = lane / K, c = lane % K;
      const unsigned step_r = 32 / K, step_c = 32 % K;
      for (unsigned i = lane; i < KK; i += 32) {
        if constexpr (sizeof(Scalar) == 4)
          CopyAsync<4>(dst + r * KMAX + c, src + i);
        else
          dst[r * KMAX + c] = static_cast<float>(src[i]);
        r += step_r;
        c += step_c;
        if (c >= K) {
          c -= K;
          ++r;
        }
      }
    }
    CopyCommit();
  }
  __device__ __forceinline__ void Clear(float *dst, unsigned count) const {
    if constexpr (!kExact) {
      for (unsigned i = lane; i < count; i += 32)
        dst[i] = 0.0f;
      __syncwarp();
    }
  }
  __device__ __forceinline__ static void Row(const float *p, float (&out)[KMAX]) {
#pragma unroll
    for (int j = 0; j < KMAX; j += 4) {
      const float4 v = *reinterpret_cast<const float4 *>(p + j);
      out[j] = v.x, out[j + 1] = v.y, out[j + 2] = v.z, out[j + 3] = v.w;
    }
  }
  __device__ __forceinline__ static int Exponent(const float (&v)[KMAX]) {
    float m = v[0];
#pragma unroll
    for (int j = 1; j < KMAX; ++j)
      m = m < v[j] ? v[j] : m;
    return m > 0.0f ? Pow2Exponent(m) : 0;
  }
  __device__ __forceinline__ static void Scale(float (&v)[KMAX], int s) {
    if (s >= -126 && s <= 127) {
      const float factor = __uint_as_float(static_cast<unsigned>(127 + s) << 23);
#pragma unroll
      for (int j = 0; j < KMAX; ++j)
        v[j] = v[j] * factor;
    } else {
#pragma unroll
      for (int j = 0; j < KMAX; ++j)
        v[j] = ldexpf(v[j], s);
    }
  }
  __device__ __forceinline__ static float Dot(const float (&row)[KMAX], const float (&x)[KMAX]) {
    float dot = 0.0f;
#pragma unroll
    for (int j = 0; j < KMAX; ++j)
      dot = fmaf(row[j], x[j], dot);
    return dot;
  }

  __device__ __forceinline__ void Gather(std::uint32_t i) const {
    const uint4 op = a.gathers[i];
    const std::uint32_t node = op.x & kMask;
    const std::uint32_t count = op.w & kCountMask;
    float v[KMAX];
    int e = 0;
    uint4 rake = a.rakes[op.z];
    Clear(paths, 2 * KMAX * KMAX);
    Stage(rake.x, paths);
    if (op.x & kFlag)
      Input(node, op.y, (op.w & kRootBit) != 0, v);
    else
      Node(node | kFlag, kNone, v, e);
#pragma unroll 1
    for (std::uint32_t k = 0; k < count; ++k) {
      const float *path = paths + (k & 1u) * (KMAX * KMAX);
      float leaf[KMAX], message[KMAX];
      Node(rake.y, rake.z, leaf, e);
      if (k + 1 < count) {
        rake = a.rakes[op.z + k + 1];
        Stage(rake.x, paths + (~k & 1u) * (KMAX * KMAX));
        CopyWait<1>();
      } else {
        CopyWait<0>();
      }
      __syncwarp();
#pragma unroll
      for (unsigned r = 0; r < KMAX; ++r) {
        message[r] = 0.0f;
        if (r < K) {
          float row[KMAX];
          Row(path + r * KMAX, row);
          message[r] = Dot(row, leaf);
        }
      }
      __syncwarp(); // every lane is done with `path`
      int s = Exponent(message);
      e += s;
      Scale(message, -s);
#pragma unroll
      for (int j = 0; j < KMAX; ++j)
        v[j] = v[j] * message[j];
      s = Exponent(v);
      e += s;
      Scale(v, -s);
    }
    if (lane < items) {
      const std::size_t at = Store(node);
      float *out = static_cast<float *>(a.nodes) + at * K;
      if constexpr (kExact) {
#pragma unroll
        for (int j = 0; j < KMAX; j += 4)
          *reinterpret_cast<float4 *>(out + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      } else {
#pragma unroll
        for (unsigned j = 0; j < KMAX; ++j)
          if (j < K)
            out[j] = v[j];
      }
      a.node_exp[at] = e;
    }
  }

  // The rake adjoints have K == KMAX.
  // Puts `row` at element `at` of this lane's part of the tile.
  __device__ __forceinline__ void Put(unsigned at, const float (&row)[KMAX]) const {
    float *dst = tile + lane * kPitch + at;
#pragma unroll
    for (int j = 0; j < KMAX; j += 4)
      *reinterpret_cast<float4 *>(dst + j) =
          make_float4(row[j], row[j + 1], row[j + 2], row[j + 3]);
  }
  // Writes `rows` <= kCount rows of every live lane's part to `out`, `pitch`
  // elements from item to item.
  template <int kCount>
  __device__ __forceinline__ void Flush(Scalar *out, std::size_t pitch, unsigned rows) const {
    constexpr unsigned kQuads = kCount * KMAX / 4; // of an item
    __syncwarp();
#pragma unroll 2 // all of them hold kQuads addresses and spill
    for (unsigned b = 0; b < kQuads; ++b) {
      const unsigned q = b * 32 + lane, at = q / kQuads, quad = q % kQuads;
      if (at < items && 4 * quad < rows * KMAX) {
        float v[4];
        Load4(tile + at * kPitch + 4 * quad, v);
        Store4<true>(out + at * pitch + 4 * quad, v);
      }
    }
    __syncwarp();
  }

  __device__ __forceinline__ void RakeReverse(std::uint32_t i) const {
    const uint4 op = a.rakes[i];
    Clear(paths, KMAX * KMAX);
    Stage(op.x, paths);
    Scalar *node_out = static_cast<Scalar *>(a.node_out);
    const Scalar *parent = node_out + (item * a.item_nodes + op.w) * K;
    Scalar *out = static_cast<Scalar *>(a.edge_out) +
                  (first * a.item_edges + op.x) * static_cast<std::size_t>(KK);
    const std::size_t pitch = a.item_edges * static_cast<std::size_t>(KK);
    float leaf[KMAX], column[KMAX];
    int unused = 0;
    Node(op.y, op.z, leaf, unused);
#pragma unroll
    for (int j = 0; j < KMAX; ++j)
      column[j] = 0.0f;
    float next = static_cast<float>(parent[0]);
    CopyWait<0>();
    __syncwarp();
#pragma unroll 1
    for (unsigned r0 = 0; r0 < K; r0 += kRows) {
#pragma unroll 1
      for (unsigned q = 0; q < kRows; ++q) {
        const unsigned r = r0 + q;
        if (r < K) {
          const float adjoint = next;
          if (r + 1 < K)
            next = static_cast<float>(parent[r + 1]);
          float row[KMAX];
          Row(paths + r * KMAX, row);
          const float unnormalised = Dot(row, leaf);
          const float ratio = unnormalised > 0.0f ? adjoint / unnormalised : 0.0f;
#pragma unroll
          for (int j = 0; j < KMAX; ++j) {
            column[j] = fmaf(ratio, row[j], column[j]);
            row[j] = ratio * row[j] * leaf[j];
          }
          Put(q * K, row);
        }
      }
      Flush<kRows>(out + r0 * K, pitch, K - r0 < kRows ? K - r0 : kRows);
    }
#pragma unroll
    for (int j = 0; j < KMAX; ++j)
      column[j] = leaf[j] * column[j];
    Put(0, column);
    Flush<1>(node_out + (first * a.item_nodes + (op.y & kMask)) * K, a.item_nodes * K, 1);
  }
};

// Warp w runs operation offset + w / tiles of 32 batch items.
template <typename Scalar, int KMAX, int kKind, bool kExact>
__global__ void __launch_bounds__(kItemPhaseThreads, KMAX > 20                   ? 2
                                                     : kKind == kPhaseGather ? 4
                                                                             : 5)
    ItemPhaseKernel(PhaseArgs args) {
  static_assert(kExact || kKind == kPhaseGather, "rake adjoints: whole quads");
  constexpr int kWarps = kItemPhaseThreads / 32;
  constexpr int kElements = kItemElements<KMAX, kKind>;
  __shared__ __align__(16) float smem[kWarps * kElements];
  const std::uint32_t w = blockIdx.x * kWarps + threadIdx.x / 32;
  const std::uint32_t per_op = (args.items + 31) / 32;
  const std::uint32_t op = w / per_op, from = w % per_op * 32;
  if (op >= args.count)
    return;
  const ItemPhaseOps<Scalar, KMAX, kExact> ops(
      args, args.first_item + from, args.items - from < 32 ? args.items - from : 32u,
      smem + threadIdx.x / 32 * kElements);
  if constexpr (kKind == kPhaseGather)
    ops.Gather(args.offset + op);
  else
    ops.RakeReverse(args.offset + op);
}

} // namespace thmm

#endif // THMM_PHASE_ITEMS_CUH_
