// Phase kernels of MAP reconstruction and posterior sampling (K <= 32) on the
// level-synchronous schedule (phase.h): every round of every tree in one
// grid-wide launch per operation kind, the last rounds in one CTA per tree.
//
// Arithmetic. Each operation performs the floating-point operations of
// MaxEngine and SampleEngine (engine.cuh) in the same order, so the discrete
// outputs agree bit for bit. The per-tree engines run a round's rakes,
// pairwise branch combinations and absorptions as separate steps; here one
// gather does all three for one parent. Its rakes are stored in branch order
// and the plan combines branch i with branch i + s for i a multiple of 2s,
// s = 1, 2, 4, ..., which is the order of a binary counter: after branch k,
// merge once per trailing one bit of k; at the end, merge the remaining
// partial sums from the newest to the oldest.
//
// The rakes of a gather are independent up to those sums. A group takes a few of
// them one after the other; more than kWideGather of a grid-wide round get a block
// of their own. A tail's block, which is short of operations and not of threads,
// forms all messages of a round before the sums. One star at K = 4, MAP, a group
// -> a block: 100 leaves 287 -> 52 us a call, 10,000 leaves 23.7 -> 0.15 ms (the
// per-tree engine 74 and 420 us).
//
// What bounds them. A factor enters through a logarithm of some 45
// instructions, and sampling adds an exponential per term, so at K = 8 the
// kernels are bound by instruction issue and not by DRAM (a 256-byte edge
// matrix costs 64 logarithms). Hence the split: a group of G lanes
// (G = 8, 16 or 32, the power of two >= K) runs one operation, lane r takes
// row r, and every logarithm is taken once: a leaf's by lane j and passed
// around by shuffles, a right factor's by row into a shared-memory tile. The
// per-tree engines took the right factor's K^2 logarithms once per lane.
// K <= 4 has one thread per operation and K^2 <= 16 logarithms of its own.
// Measured on one GB300, per-tree engines -> these kernels: MAP of 320
// Galton-Watson trees (8.2 M nodes, K = 8) 7.57 -> 1.21 ms, sampling of the
// same trees 11.4 -> 1.94 ms, a host-to-host MAP call on 48 uneven trees
// (76 k nodes, K = 8) 2.35 -> 0.26 ms.
#ifndef THMM_PHASE_LOG_CUH_
#define THMM_PHASE_LOG_CUH_

#include <cstdint>
#include <cuda_runtime.h>

#include "engine.cuh"
#include "phase.h"

namespace thmm {

constexpr int kLogPhaseThreads = 128;

// Shared-memory tile of one lane group: the right factor's logarithms, KMAX
// rows of KMAX, padded by 8 values so that the groups of a warp read
// different banks.
template <int KMAX> inline constexpr int kLogTile = KMAX * KMAX + 8;

// Logarithms and exponentials four at a time, without branches: a branch per
// element would put each some 20 to 30 instructions in a block of its own.
// Elements outside the range of the short forms (subnormal or infinite
// factors; exponents between -104 and -87) send the four to the general
// functions, which give the same bits inside the range.
__device__ __forceinline__ void PotentialLogs(float (&v)[4]) {
  float out[4];
  bool rare = false;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const unsigned bits = __float_as_uint(v[j]);
    out[j] = v[j] > 0.0f ? thmm_logf_normal(bits, 0) : NegInf<float>();
    rare = rare || (v[j] > 0.0f && bits - 0x00800000u >= 0x7f000000u);
  }
  if (rare) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      out[j] = PotentialLog(v[j]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    v[j] = out[j];
}
__device__ __forceinline__ void PotentialLogs(double (&v)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
    v[j] = PotentialLog(v[j]);
}

// sum + exp(x[0]) + ... + exp(x[3]), in that order, for x <= 0 (or NaN, which
// the short form passes on).
__device__ __forceinline__ float AddExps(float sum, const float (&x)[4]) {
  float e[4];
  if (fminf(fminf(x[0], x[1]), fminf(x[2], x[3])) >= -87.0f) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      e[j] = thmm_expf_short(x[j]);
  } else {
    // Zero factors: -inf. Between -104 and -87 the general function.
    bool rare = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      e[j] = x[j] < -103.972084f ? 0.0f : thmm_expf_short(x[j]);
      rare = rare || (x[j] < -87.0f && !(x[j] < -103.972084f));
    }
    if (rare) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        e[j] = thmm_expf(x[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    sum = sum + e[j];
  return sum;
}
__device__ __forceinline__ double AddExps(double sum, const double (&x)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
    sum = sum + thmm_exp(x[j]);
  return sum;
}

// LogSumExp (src/inference.cc:100-110) over terms[0..K), -inf from K on (which
// changes neither the maximum nor, adding zeros, the sum).
template <typename T, int KMAX>
__device__ __forceinline__ T PaddedLogSumExp(const T (&terms)[KMAX], unsigned K) {
  T maximum = NegInf<T>();
#pragma unroll
  for (unsigned j = 0; j < KMAX; ++j)
    maximum = sizeof(T) == 4 ? static_cast<T>(fmaxf(maximum, terms[j])) // NaN: ignored too
                             : maximum < terms[j] ? terms[j] : maximum;
  if (!isfinite(maximum))
    return maximum;
  T sum = T(0);
#pragma unroll
  for (unsigned q = 0; q < KMAX; q += 4) {
    if (q < K) {
      const T x[4] = {terms[q] - maximum, terms[q + 1] - maximum, terms[q + 2] - maximum,
                      terms[q + 3] - maximum};
      sum = AddExps(sum, x);
    }
  }
  return maximum + PortableLog(sum);
}

// kExact: K == KMAX, so that the compiler folds the bounds and the strides.
template <typename T, int KMAX, bool kSample, bool kExact> struct LogPhaseOps {
  static constexpr int G = GroupLanes<KMAX>();
  static constexpr int ROWS = (KMAX + G - 1) / G; // rows per lane: KMAX or 1
  static constexpr unsigned kLevels = 5;          // a gather's partial sums in registers
  const PhaseArgs &a;
  unsigned K;
  unsigned KK;
  std::size_t item;   // batch item (0 for a forest)
  std::size_t stride; // items per stored object (1 for a forest)
  unsigned lane;      // lane within the group
  unsigned mask;      // the group's lanes of the warp
  T *tile;            // the group's shared-memory tile (G > 1)

  __device__ __forceinline__ LogPhaseOps(const PhaseArgs &args, std::uint32_t batch_item,
                                         T *group_tile)
      : a(args), K(kExact ? KMAX : args.states), KK(K * K), item(batch_item),
        stride(args.item_stride), lane(threadIdx.x % G),
        mask(G == 32 ? kFull : ((1u << (G & 31)) - 1u) << (threadIdx.x % 32 / G * G)),
        tile(group_tile) {}

  // Where objects live: stored values are item-minor, the caller's arrays
  // item-major (phase_engine.cuh's two index maps, with stride 1 and item 0
  // for a forest).
  __device__ __forceinline__ std::size_t Store(std::uint32_t object) const {
    return object * stride + item;
  }
  __device__ __forceinline__ std::size_t Io(std::uint32_t node) const {
    return item * a.item_nodes + node;
  }

  // Factor j of input node `node` in the input precision, as
  // Context::InputNode.
  __device__ __forceinline__ T InputElement(std::uint32_t node, std::uint32_t obs, bool root,
                                            unsigned j) const {
    if (!a.categorical)
      return static_cast<const T *>(a.node_in)[Io(node) * K + j];
    const T *root_potential = static_cast<const T *>(a.root_potential);
    if (obs == kNone)
      return root ? root_potential[j] : T(1);
    const unsigned category = a.observations[Store(obs)];
    if (category >= a.categories)
      return T(0);
    const T emitted = static_cast<const T *>(a.emission)[category * K + j];
    return root ? root_potential[j] * emitted : emitted;
  }

  // Log value of a node (every lane the whole vector, -inf past K).
  __device__ __forceinline__ void NodeVector(std::uint32_t ref, std::uint32_t obs, bool root,
                                             T (&out)[KMAX]) const {
    if (G == 1 || (ref & kFlag)) {
      NodeVectorAlone(ref, obs, root, out);
    } else {
      const T own =
          lane < K ? PotentialLog(InputElement(ref, obs, root, lane)) : NegInf<T>();
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        out[j] = __shfl_sync(mask, own, j, G);
    }
  }
  // The same, by one thread alone.
  __device__ __forceinline__ void NodeVectorAlone(std::uint32_t ref, std::uint32_t obs,
                                                  bool root, T (&out)[KMAX]) const {
    if (ref & kFlag) {
      Row(static_cast<const T *>(a.nodes) + Store(ref & kMask) * K, NegInf<T>(), out);
    } else {
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        out[j] = j < K ? InputElement(ref, obs, root, j) : T(0);
      Logs(out);
    }
  }

  // K values from p, `pad` past K, in 16-byte loads where every row starts on
  // a 16-byte boundary.
  __device__ __forceinline__ void Row(const T *p, T pad, T (&out)[KMAX]) const {
    constexpr unsigned kPer = 16 / sizeof(T);
    if (K % kPer == 0) {
#pragma unroll
      for (unsigned q = 0; q < KMAX / kPer; ++q) {
        if (q * kPer < K) {
          const uint4 raw = reinterpret_cast<const uint4 *>(p)[q];
          T values[kPer];
          memcpy(values, &raw, 16);
#pragma unroll
          for (unsigned j = 0; j < kPer; ++j)
            out[q * kPer + j] = values[j];
        } else {
#pragma unroll
          for (unsigned j = 0; j < kPer; ++j)
            out[q * kPer + j] = pad;
        }
      }
    } else {
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        out[j] = j < K ? p[j] : pad;
    }
  }
  // Logarithms in place (of factors, 0 past K: -inf there).
  __device__ __forceinline__ void Logs(T (&v)[KMAX]) const {
#pragma unroll
    for (unsigned q = 0; q < KMAX; q += 4) {
      if (q < K) {
        T four[4] = {v[q], v[q + 1], v[q + 2], v[q + 3]};
        PotentialLogs(four);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[q + j] = four[j];
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[q + j] = NegInf<T>();
      }
    }
  }
  // Log row r of a path, -inf past K.
  __device__ __forceinline__ void PathRow(std::uint32_t ref, unsigned r, T (&out)[KMAX]) const {
    if (ref & kFlag) {
      Row(static_cast<const T *>(a.comps) + Store(ref & kMask) * KK + r * K, NegInf<T>(), out);
    } else {
      Row(static_cast<const T *>(a.edge_in) + static_cast<std::size_t>(ref) * KK + r * K, T(0),
          out);
      Logs(out);
    }
  }
  // Log column j of a path, -inf past K.
  __device__ __forceinline__ void PathColumn(std::uint32_t ref, unsigned j,
                                             T (&out)[KMAX]) const {
    const bool stored = (ref & kFlag) != 0;
    const T *p = stored ? static_cast<const T *>(a.comps) + Store(ref & kMask) * KK
                        : static_cast<const T *>(a.edge_in) + static_cast<std::size_t>(ref) * KK;
#pragma unroll
    for (unsigned m = 0; m < KMAX; ++m)
      out[m] = m < K ? p[m * K + j] : stored ? NegInf<T>() : T(0);
    if (!stored)
      Logs(out);
  }

  // ---------------------------------------------------------- forward
  // Message of one rake at row r (src/inference.cc:576-594, 259-277).
  __device__ __forceinline__ T Message(std::uint32_t rake, const uint4 &op, unsigned r,
                                       const T (&leaf)[KMAX]) const {
    T row[KMAX];
    PathRow(op.x, r, row);
    if constexpr (kSample) {
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        row[j] = row[j] + leaf[j];
      return PaddedLogSumExp<T, KMAX>(row, K);
    } else {
      T best = row[0] + leaf[0];
      unsigned choice = 0;
#pragma unroll
      for (unsigned j = 1; j < KMAX; ++j) { // terms past K are -inf and never win
        const T term = row[j] + leaf[j];
        if (term > best) {
          best = term;
          choice = j;
        }
      }
      a.rake_choices[Store(rake) * K + r] = static_cast<std::uint8_t>(choice);
      return best;
    }
  }

  // Element r of a branch's scratch vector.
  __device__ __forceinline__ T *BranchAt(std::uint32_t rake, unsigned r) const {
    return static_cast<T *>(a.branches) + Store(rake) * K + r;
  }
  __device__ __forceinline__ T Branch(std::uint32_t rake, unsigned r) const {
    return r < K ? *BranchAt(rake, r) : T(0);
  }

  // Rake `rake` alone: its message into the branch's scratch vector.
  __device__ __forceinline__ void Rake(std::uint32_t rake) const {
    const uint4 op = a.rakes[rake];
    T leaf[KMAX];
    NodeVector(op.y, op.z, false, leaf);
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      const unsigned r = lane + q * G;
      if (r < K)
        *BranchAt(rake, r) = Message(rake, op, r, leaf);
    }
  }

  // The node value that gather `op` adds its branches to, element r.
  __device__ __forceinline__ T Previous(const uint4 &op, unsigned r) const {
    const std::uint32_t node = op.x & kMask;
    return (op.x & kFlag) ? PotentialLog(InputElement(node, op.y, (op.w & kRootBit) != 0, r))
                          : static_cast<const T *>(a.nodes)[Store(node) * K + r];
  }

  // Branch combinations and absorption of gather `op`, whose messages lie in the
  // branches' scratch, by the whole block of kThreads threads.
  template <int kThreads> __device__ __forceinline__ void CombineByBlock(const uint4 &op) const {
    const std::uint32_t count = op.w & kCountMask;
    for (std::uint32_t s = 1; s < count; s *= 2) {
      const std::size_t pairs = (static_cast<std::size_t>(count) + s - 1) / (2 * s);
      for (std::size_t e = threadIdx.x; e < pairs * K; e += kThreads) {
        const auto b = op.z + static_cast<std::uint32_t>(e / K) * 2 * s;
        const unsigned r = static_cast<unsigned>(e % K);
        *BranchAt(b, r) = *BranchAt(b, r) + *BranchAt(b + s, r);
      }
      __syncthreads();
    }
    for (unsigned r = threadIdx.x; r < K; r += kThreads)
      static_cast<T *>(a.nodes)[Store(op.x & kMask) * K + r] = Previous(op, r) + *BranchAt(op.z, r);
  }

  // Gather `op` by the whole block: a rake per group at a time, unless the
  // messages are ready.
  template <int kThreads> __device__ __forceinline__ void GatherByBlock(const uint4 &op) const {
    const std::uint32_t count = op.w & kCountMask;
    if (a.ready == 0) {
      for (std::uint32_t k = threadIdx.x / G; k < count; k += kThreads / G)
        Rake(op.z + k);
      __syncthreads();
    }
    CombineByBlock<kThreads>(op);
  }

  // Rakes (kReady: their messages lie in the branches' scratch), branch
  // combinations and absorption of gather `op` by one group.
  template <bool kReady> __device__ __forceinline__ void Gather(const uint4 &op) const {
    const std::uint32_t node = op.x & kMask;
    const std::uint32_t count = op.w & kCountMask;
    // Binary counter of partial sums: the low levels in registers, the others
    // (fan-in of 32 and more) in the scratch of the gather's own branches,
    // which has an entry per rake and so one per level (that rake's message has
    // been added by then).
    T partial[kLevels][ROWS];
    for (std::uint32_t k = 0; k < count; ++k) {
      T value[ROWS];
      if constexpr (kReady) {
#pragma unroll
        for (int q = 0; q < ROWS; ++q)
          value[q] = Branch(op.z + k, lane + q * G);
      } else {
        const uint4 rake = a.rakes[op.z + k];
        T leaf[KMAX];
        NodeVector(rake.y, rake.z, false, leaf);
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
          const unsigned r = lane + q * G;
          value[q] = r < K ? Message(op.z + k, rake, r, leaf) : T(0);
        }
      }
      bool carry = true;
#pragma unroll
      for (unsigned level = 0; level < kLevels; ++level) {
        if (carry) {
          carry = (k >> level) & 1u;
#pragma unroll
          for (int q = 0; q < ROWS; ++q) {
            if (carry)
              value[q] = partial[level][q] + value[q];
            else
              partial[level][q] = value[q];
          }
        }
      }
      if (carry) {
        unsigned level = kLevels;
        for (; (k >> level) & 1u; ++level)
#pragma unroll
          for (int q = 0; q < ROWS; ++q)
            value[q] = Branch(op.z + level, lane + q * G) + value[q];
#pragma unroll
        for (int q = 0; q < ROWS; ++q)
          if (lane + q * G < K)
            *BranchAt(op.z + level, lane + q * G) = value[q];
      }
    }
    T sum[ROWS];
    bool first = true;
#pragma unroll
    for (unsigned level = 0; level < kLevels; ++level) {
      if ((count >> level) & 1u) {
#pragma unroll
        for (int q = 0; q < ROWS; ++q)
          sum[q] = first ? partial[level][q] : partial[level][q] + sum[q];
        first = false;
      }
    }
    for (unsigned level = kLevels; (count >> level) != 0; ++level) {
      if ((count >> level) & 1u) {
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
          const T high = Branch(op.z + level, lane + q * G);
          sum[q] = first ? high : high + sum[q];
        }
        first = false;
      }
    }
    T *dst = static_cast<T *>(a.nodes) + Store(node) * K;
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      const unsigned r = lane + q * G;
      if (r < K)
        dst[r] = Previous(op, r) + sum[q];
    }
  }

  // Compressed path i (src/inference.cc:614-639, 297-324).
  __device__ __forceinline__ void Compress(std::uint32_t i) const {
    const uint4 op = a.compress[i];
    T middle[KMAX];
    NodeVector(op.y, op.w, false, middle);
    T rights[G == 1 ? KMAX : 1][KMAX]; // G = 1: the right factor in registers
    if constexpr (G == 1) {
#pragma unroll
      for (unsigned m = 0; m < KMAX; ++m)
        if (m < K)
          PathRow(op.z, m, rights[m]);
    } else {
      __syncwarp(mask); // the group's previous operation is done with the tile
      if (lane < KMAX) {
        T right[KMAX];
        if (lane < K) {
          PathRow(op.z, lane, right);
        } else {
#pragma unroll
          for (unsigned j = 0; j < KMAX; ++j)
            right[j] = NegInf<T>();
        }
#pragma unroll
        for (unsigned j = 0; j < KMAX; ++j)
          tile[kSample ? j * KMAX + lane : lane * KMAX + j] = right[j];
      }
      __syncwarp(mask);
    }
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      const unsigned r = lane + q * G;
      if (r >= K)
        continue;
      T head[KMAX];
      PathRow(op.x, r, head);
#pragma unroll
      for (unsigned m = 0; m < KMAX; ++m)
        head[m] = head[m] + middle[m];
      T *dst = static_cast<T *>(a.comps) + Store(i) * KK + r * K;
      if constexpr (kSample) {
        T out[KMAX];
        if constexpr (G == 1) {
#pragma unroll
          for (unsigned j = 0; j < KMAX; ++j) {
            if (j < K) {
              T terms[KMAX];
#pragma unroll
              for (unsigned m = 0; m < KMAX; ++m)
                terms[m] = m < K ? head[m] + rights[m][j] : NegInf<T>();
              out[j] = PaddedLogSumExp<T, KMAX>(terms, K);
            }
          }
          StoreRow<KMAX>(dst, K, out);
        } else {
          for (unsigned j = 0; j < K; ++j) {
            T terms[KMAX];
#pragma unroll
            for (unsigned m = 0; m < KMAX; ++m)
              terms[m] = head[m] + tile[j * KMAX + m];
            dst[j] = PaddedLogSumExp<T, KMAX>(terms, K);
          }
        }
      } else {
        T best[KMAX];
        unsigned choice[KMAX];
#pragma unroll
        for (unsigned j = 0; j < KMAX; ++j) {
          best[j] = head[0] + (G == 1 ? rights[0][j] : tile[j]);
          choice[j] = 0;
        }
#pragma unroll
        for (unsigned m = 1; m < KMAX; ++m) {
          if (m < K) {
#pragma unroll
            for (unsigned j = 0; j < KMAX; ++j) {
              const T term = head[m] + (G == 1 ? rights[G == 1 ? m : 0][j] : tile[m * KMAX + j]);
              if (term > best[j]) {
                best[j] = term;
                choice[j] = m;
              }
            }
          }
        }
        if constexpr (KMAX == 4 || KMAX >= 16) {
          StoreRow<KMAX>(dst, K, best);
        } else {
          if (K == KMAX && sizeof(T) == 4) {
#pragma unroll
            for (unsigned q4 = 0; q4 < KMAX / 4; ++q4)
              reinterpret_cast<float4 *>(dst)[q4] = make_float4(
                  best[4 * q4], best[4 * q4 + 1], best[4 * q4 + 2], best[4 * q4 + 3]);
          } else {
            StoreRow<KMAX>(dst, K, best);
          }
        }
        std::uint8_t *choices = a.comp_choices + Store(i) * KK + r * K;
        if (K % 4 == 0) { // rows of choices start on 4-byte boundaries
#pragma unroll
          for (unsigned q4 = 0; q4 < KMAX / 4; ++q4)
            if (4 * q4 < K)
              reinterpret_cast<std::uint32_t *>(choices)[q4] =
                  choice[4 * q4] | choice[4 * q4 + 1] << 8 | choice[4 * q4 + 2] << 16 |
                  choice[4 * q4 + 3] << 24;
        } else {
#pragma unroll
          for (unsigned j = 0; j < KMAX; ++j)
            if (j < K)
              choices[j] = static_cast<std::uint8_t>(choice[j]);
        }
      }
    }
  }

  // ---------------------------------------------------------- top-down
  __device__ __forceinline__ unsigned Draw(const T (&terms)[KMAX], T normalizer,
                                           std::uint32_t node) const {
    const T uniform = static_cast<const T *>(a.uniforms)[Io(node)];
    if (!(uniform >= T(0) && uniform < T(1)))
      atomicOr(a.error, kErrorInvalidUniform);
    const unsigned choice = SampleLogWeights<T, KMAX>(terms, K, normalizer, uniform);
    if (choice >= K) {
      atomicOr(a.error, kErrorEmptyConditional);
      return 0;
    }
    return choice;
  }

  // FinishRoot (src/inference.cc:641-649, 326-361): root record i, result of
  // instance `value`.
  __device__ __forceinline__ void Root(std::uint32_t i, std::uint32_t value) const {
    const uint2 rec = a.roots[i];
    const std::uint32_t node = rec.x & kMask;
    T terms[KMAX];
    NodeVectorAlone(rec.x, rec.y, true, terms);
    unsigned choice = 0;
    T result;
    if constexpr (kSample) {
      result = PaddedLogSumExp<T, KMAX>(terms, K);
      if (isfinite(result))
        choice = Draw(terms, result, node);
    } else {
      result = terms[0];
#pragma unroll
      for (unsigned j = 1; j < KMAX; ++j) {
        if (terms[j] > result) {
          result = terms[j];
          choice = j;
        }
      }
    }
    static_cast<T *>(a.values)[value] = result;
    a.states_out[Io(node)] = choice;
  }

  // ExpandRakes / ExpandCompressions (src/inference.cc:651-667, 363-412), one
  // thread per operation: a sampled state needs one row of the rake's matrix
  // (one row and one column of a compression's), a MAP state one stored byte.
  __device__ __forceinline__ void ExpandRake(std::uint32_t i) const {
    const uint4 op = a.rakes[i];
    const std::uint32_t leaf_node = op.y & kMask;
    const unsigned parent_state = a.states_out[Io(op.w)];
    if constexpr (kSample) {
      T leaf[KMAX], terms[KMAX];
      NodeVectorAlone(op.y, op.z, false, leaf);
      PathRow(op.x, parent_state, terms);
#pragma unroll
      for (unsigned j = 0; j < KMAX; ++j)
        terms[j] = terms[j] + leaf[j];
      const T normalizer = PaddedLogSumExp<T, KMAX>(terms, K);
      a.states_out[Io(leaf_node)] = Draw(terms, normalizer, leaf_node);
    } else {
      a.states_out[Io(leaf_node)] = a.rake_choices[Store(i) * K + parent_state];
    }
  }
  __device__ __forceinline__ void ExpandCompress(std::uint32_t i) const {
    const uint4 op = a.compress[i];
    const uint2 end = a.ends[i];
    const std::uint32_t middle_node = op.y & kMask;
    const unsigned parent_state = a.states_out[Io(end.x)];
    const unsigned child_state = a.states_out[Io(end.y)];
    if constexpr (kSample) {
      T middle[KMAX], terms[KMAX], right[KMAX];
      NodeVectorAlone(op.y, op.w, false, middle);
      PathRow(op.x, parent_state, terms);
      PathColumn(op.z, child_state, right);
#pragma unroll
      for (unsigned m = 0; m < KMAX; ++m)
        terms[m] = terms[m] + middle[m] + right[m];
      const T normalizer = PaddedLogSumExp<T, KMAX>(terms, K);
      a.states_out[Io(middle_node)] = Draw(terms, normalizer, middle_node);
    } else {
      a.states_out[Io(middle_node)] =
          a.comp_choices[Store(i) * KK + parent_state * K + child_state];
    }
  }
};

// One kind of one round over args.count operations of args.items items:
// group (top-down kinds and roots: thread) t runs operation offset + t /
// items of item first_item + t % items, so the groups of a warp read one
// record and one edge matrix of a batch together. The tail kind runs the
// last rounds, the root and the last rounds' top-down steps of one tree per
// CTA, with a CTA barrier between steps.
// A tail block's passes over a step are dependent trips to memory, so where
// every block has an SM of its own it gets as many threads as the registers
// allow: 48 uneven trees, MAP at K = 8, 278 us a call with 128 threads, 256 us
// with 512; 320 trees 1.30 ms with 128, 1.34 ms with 512.
template <typename T, int KMAX>
inline constexpr int kLogTailThreads = sizeof(T) == 4 && KMAX <= 8    ? 512
                                       : sizeof(T) == 4 && KMAX <= 20 ? 256
                                                                      : kLogPhaseThreads;
constexpr std::uint64_t kLogTailBlocks = 152; // SMs

// Kinds that run a lane group per operation.
template <int kKind>
inline constexpr bool kLogGroups = kKind == kPhaseGather || kKind == kPhaseCompress ||
                                   kKind == kPhaseRake || kKind == kPhaseReadyGather;

// Fan-in above which a tail's block forms a gather's sums together; its messages
// lie in scratch already.
constexpr std::uint32_t kWideCombine = 32;

template <typename T, int KMAX, bool kSample, int kKind, int kThreads, bool kExact>
__global__ void __launch_bounds__(kThreads, kThreads > kLogPhaseThreads      ? 1
                                            : kThreads < kLogPhaseThreads ? 12
                                            : KMAX <= 8 && sizeof(T) == 4 ? 4
                                            : KMAX <= 4                   ? 3
                                                                          : 2)
    LogPhaseKernel(PhaseArgs args) {
  using Ops = LogPhaseOps<T, KMAX, kSample, kExact>;
  constexpr int G = Ops::G;
  constexpr bool kTile = G > 1 && (kKind == kPhaseCompress || kKind == kPhaseTailForward);
  __shared__ __align__(16) T tiles[kTile ? (kThreads / G) * kLogTile<KMAX> : 1];
  T *tile = kTile ? tiles + threadIdx.x / G * kLogTile<KMAX> : nullptr;
  if constexpr (kKind == kPhaseTailForward) {
    const uint4 tree = args.tail_items[args.batch ? 0u : args.offset + blockIdx.x];
    const std::uint32_t item = args.batch ? args.first_item + blockIdx.x : 0u;
    const Ops ops(args, item, tile);
    const unsigned group = threadIdx.x / G;
    for (std::uint32_t e = 0; e < tree.z; ++e) {
      const uint4 round = args.tail_rounds[tree.y + e];
      const uint2 rakes = args.tail_rakes[tree.y + e];
      for (std::uint32_t i = group; i < rakes.y; i += kThreads / G)
        ops.Rake(rakes.x + i);
      __syncthreads();
      bool wide = false;
      for (std::uint32_t i = group; i < round.y; i += kThreads / G) {
        const uint4 op = args.gathers[round.x + i];
        if ((op.w & kCountMask) > kWideCombine)
          wide = true;
        else
          ops.template Gather<true>(op);
      }
      if (__syncthreads_or(wide)) {
        for (std::uint32_t i = 0; i < round.y; ++i) {
          const uint4 op = args.gathers[round.x + i];
          if ((op.w & kCountMask) > kWideCombine)
            ops.template CombineByBlock<kThreads>(op);
        }
        __syncthreads();
      }
      if (round.w != 0) {
        for (std::uint32_t i = group; i < round.w; i += kThreads / G)
          ops.Compress(round.z + i);
        __syncthreads();
      }
    }
    if (threadIdx.x == 0)
      ops.Root(tree.x, args.batch ? item : tree.x);
    __syncthreads();
    for (std::uint32_t e = tree.z; e-- > 0;) {
      const uint4 round = args.tail_rounds[tree.y + e];
      if (round.w != 0) {
        for (std::uint32_t i = threadIdx.x; i < round.w; i += kThreads)
          ops.ExpandCompress(round.z + i);
        __syncthreads();
      }
      const uint2 rakes = args.tail_rakes[tree.y + e];
      for (std::uint32_t i = threadIdx.x; i < rakes.y; i += kThreads)
        ops.ExpandRake(rakes.x + i);
      __syncthreads();
    }
  } else if constexpr (kKind == kPhaseWideGather) {
    const std::uint32_t op = args.batch ? blockIdx.x / args.items : blockIdx.x;
    const Ops ops(args, args.batch ? args.first_item + blockIdx.x % args.items : 0u, tile);
    ops.template GatherByBlock<kThreads>(args.gathers[args.wide[args.offset + op]]);
  } else {
    constexpr bool kGroups = kLogGroups<kKind>;
    const std::uint32_t t =
        kGroups ? static_cast<std::uint32_t>(
                      (static_cast<std::uint64_t>(blockIdx.x) * kThreads + threadIdx.x) / G)
                : blockIdx.x * kThreads + threadIdx.x;
    if (t >= args.count * args.items) // below 2^31 (the record index limit)
      return;
    std::uint32_t op = t, item = 0;
    if (args.batch) {
      op = t / args.items;
      item = args.first_item + t % args.items;
    }
    const Ops ops(args, item, tile);
    if constexpr (kKind == kPhaseGather || kKind == kPhaseReadyGather) {
      const uint4 gather = args.gathers[args.offset + op];
      if ((gather.w & kCountMask) <= kWideGather)
        ops.template Gather<kKind == kPhaseReadyGather>(gather);
    } else if constexpr (kKind == kPhaseRake)
      ops.Rake(args.offset + op);
    else if constexpr (kKind == kPhaseCompress)
      ops.Compress(args.offset + op);
    else if constexpr (kKind == kPhaseFinish)
      ops.Root(args.offset + op, args.batch ? item : args.offset + op);
    else if constexpr (kKind == kPhaseRakeReverse)
      ops.ExpandRake(args.offset + op);
    else if constexpr (kKind == kPhaseCompressReverse)
      ops.ExpandCompress(args.offset + op);
  }
}

// ------------------------------------------------------------- launching
template <typename T, int KMAX, bool kSample, int kKind>
cudaError_t LaunchLogKind(const PhaseArgs &args, LaunchStream stream, int *blocks_per_sm) {
  constexpr bool kGroups = kLogGroups<kKind>;
  constexpr bool kNarrow = kKind == kPhaseTailForward && KMAX == 4 && sizeof(T) == 4;
  if constexpr (kNarrow) {
    if (blocks_per_sm != nullptr && args.narrow)
      return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          blocks_per_sm, LogPhaseKernel<T, KMAX, kSample, kKind, 32, false>, 32, 0);
  }
  if (blocks_per_sm != nullptr)
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        blocks_per_sm, LogPhaseKernel<T, KMAX, kSample, kKind, kLogPhaseThreads, false>,
        kLogPhaseThreads, 0);
  std::uint64_t grid;
  if (kKind == kPhaseTailForward) {
    grid = args.batch ? args.items : args.count;
  } else if (kKind == kPhaseWideGather) {
    grid = static_cast<std::uint64_t>(args.count) * args.items;
  } else {
    const std::uint64_t threads = static_cast<std::uint64_t>(args.count) * args.items *
                                  (kGroups ? GroupLanes<KMAX>() : 1);
    grid = (threads + kLogPhaseThreads - 1) / kLogPhaseThreads;
  }
  if (grid == 0)
    return cudaSuccess;
  if (grid > 0x7fffffffull)
    return cudaErrorInvalidConfiguration;
  if constexpr (kNarrow) {
    if (args.narrow)
      return LaunchOn(stream, LogPhaseKernel<T, KMAX, kSample, kKind, 32, false>,
                      static_cast<unsigned>(grid), 32, 0, args);
  }
  if constexpr (kKind == kPhaseTailForward) {
    constexpr int kWide = kLogTailThreads<T, KMAX>;
    if (grid <= kLogTailBlocks) {
      return LaunchOn(stream, LogPhaseKernel<T, KMAX, kSample, kKind, kWide, false>,
                      static_cast<unsigned>(grid), kWide, 0, args);
    }
  }
  // Folded bounds, K = 8 in single precision: MAP of the Galton-Watson forest
  // 1,296 -> 1,222 us, sampling 2,069 -> 1,950 us. Double is bound by its
  // pipe, and K = 32 is not folded: it adds a fifth to the build for one size.
  if constexpr ((kKind == kPhaseGather || kKind == kPhaseCompress) && sizeof(T) == 4 &&
                KMAX <= 20) {
    if (args.states == KMAX) {
      return LaunchOn(stream, LogPhaseKernel<T, KMAX, kSample, kKind, kLogPhaseThreads, true>,
                      static_cast<unsigned>(grid), kLogPhaseThreads, 0, args);
    }
  }
  return LaunchOn(stream, LogPhaseKernel<T, KMAX, kSample, kKind, kLogPhaseThreads, false>,
                  static_cast<unsigned>(grid), kLogPhaseThreads, 0, args);
}

template <typename T, int KMAX, bool kSample>
cudaError_t LaunchLogStates(int kind, const PhaseArgs &args, LaunchStream stream, int *blocks_per_sm) {
  switch (kind) {
  case kPhaseGather:
    return LaunchLogKind<T, KMAX, kSample, kPhaseGather>(args, stream, blocks_per_sm);
  case kPhaseCompress:
    return LaunchLogKind<T, KMAX, kSample, kPhaseCompress>(args, stream, blocks_per_sm);
  case kPhaseFinish:
    return LaunchLogKind<T, KMAX, kSample, kPhaseFinish>(args, stream, blocks_per_sm);
  case kPhaseRakeReverse:
    return LaunchLogKind<T, KMAX, kSample, kPhaseRakeReverse>(args, stream, blocks_per_sm);
  case kPhaseCompressReverse:
    return LaunchLogKind<T, KMAX, kSample, kPhaseCompressReverse>(args, stream, blocks_per_sm);
  case kPhaseTailForward:
    return LaunchLogKind<T, KMAX, kSample, kPhaseTailForward>(args, stream, blocks_per_sm);
  case kPhaseWideGather:
    return LaunchLogKind<T, KMAX, kSample, kPhaseWideGather>(args, stream, blocks_per_sm);
  case kPhaseRake:
    return LaunchLogKind<T, KMAX, kSample, kPhaseRake>(args, stream, blocks_per_sm);
  case kPhaseReadyGather:
    return LaunchLogKind<T, KMAX, kSample, kPhaseReadyGather>(args, stream, blocks_per_sm);
  default:
    return cudaErrorInvalidValue;
  }
}

// Padded state counts: the group sizes, and 20 beside 32 in single
// precision, where the terms past K cost registers and additions (at K = 20,
// 2.6x the terms of a compression); terms past K are skipped by K, so every
// padding gives the same bits.
template <typename T, bool kSample>
cudaError_t LaunchLog(int kind, const PhaseArgs &args, LaunchStream stream, int *blocks_per_sm) {
  if (args.states <= 4)
    return LaunchLogStates<T, 4, kSample>(kind, args, stream, blocks_per_sm);
  if (args.states <= 8)
    return LaunchLogStates<T, 8, kSample>(kind, args, stream, blocks_per_sm);
  if (args.states <= 16)
    return LaunchLogStates<T, 16, kSample>(kind, args, stream, blocks_per_sm);
  if constexpr (sizeof(T) == 4) {
    if (args.states <= 20)
      return LaunchLogStates<T, 20, kSample>(kind, args, stream, blocks_per_sm);
  }
  return args.states <= 32 ? LaunchLogStates<T, 32, kSample>(kind, args, stream, blocks_per_sm)
                           : cudaErrorInvalidValue;
}

} // namespace thmm

#endif // THMM_PHASE_LOG_CUH_
