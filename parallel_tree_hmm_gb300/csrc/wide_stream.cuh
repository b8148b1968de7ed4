// Compressions and their adjoints for 32 < K <= 128, K a multiple of 4: the
// tensor-core phase kinds (wide_phase.cuh) as a pipeline of depth-64 steps fed
// by asynchronous copies.
//
// What bounded the kernels these replace (they stay for the other K, whose rows
// have no 16-byte quads): at K = 64 one reverse compression read 64 KB, wrote
// 32 KB and took 22 us of a CTA's time in ten rounds of global loads, each
// waited for before its values were staged; the tensor pipe was 12 % busy, DRAM
// 30 %, and two thirds of a warp's time went to those loads. At K = 128 the
// adjoint ratio was formed twice from column-wise 4-byte loads.
//
// The pipeline. An operation is a sequence of steps, each one depth chunk of 64
// of one product: load, convert and store the operands, tcgen05.mma, wait. The
// matrices of step s + 1 (or of the next operation's first step) come into
// shared memory by cp.async while step s's products run and during the
// epilogue. What the load/store unit does in one go is a quarter warp's 128
// bytes, so every access is dealt out for quarter warps:
//   * global reads and writes: eight consecutive quads of a row (eight rows at a
//     time took 4,500 of 7,500 wavefronts per reverse compression at K = 64 and
//     bound the kernel);
//   * raw and epilogue tiles in shared memory: quads swizzled by row, so that
//     rows and columns both are read without bank conflicts;
//   * direct operands (rows as stored): 8 rows x 4 quads per warp; transposed
//     ones: 4 rows x 8 quads, where four lanes transpose their 4 x 4 block by
//     shuffles and each stores one quad of a column.
// At K_P = 64 the adjoint ratio is formed once and kept in registers for both
// products. All loads of a stage are issued before its stores, with no branch
// between them.
// Measured on one GB300: marginals of 64 path-heavy trees x 2000 nodes, K = 64,
// 6.82 -> 4.52 ms; 64 x 500 nodes, K = 128, 9.13 -> 5.17 ms (DRAM at 3.0 to 3.7
// TB/s in the large launches, the tensor pipe 17 to 21 % busy). What is left is
// latency: two CTAs (one at K_P = 128) take turns at barriers, products and
// tensor-memory reads.
#ifndef THMM_WIDE_STREAM_CUH_
#define THMM_WIDE_STREAM_CUH_

#include <cstdint>
#include <cuda_runtime.h>

#include "phase.h"
#include "wide_phase.cuh"

namespace thmm {
namespace wide {

// Shared memory of a CTA: the operands (PhaseLayout), raw tiles of up to three
// matrices' step quads, the middle vectors of this and the next
// operation. Two CTAs per SM at KP = 64, one at 128.
template <int KP, bool kReverse> struct StreamLayout {
  using L = PhaseLayout<KP>;
  static constexpr unsigned kThreads = L::kThreads;
  static constexpr unsigned kQuads = KP * (kChunk / 4) / kThreads; // a thread's, per step
  static_assert(kQuads == 4, "quads per thread and step");
  static constexpr unsigned kSlotBytes = kQuads * kThreads * 16;
  static constexpr unsigned kSlotsAt = 4 * L::kPart;
  static constexpr unsigned kMiddleAt = kSlotsAt + (kReverse ? 3 : 2) * kSlotBytes;
  static constexpr unsigned kBytes = kMiddleAt + 2 * KP * 4;
  static constexpr int kResident = KP == 64 ? 2 : 1;
  // With 1 KB of reserved and at most 512 bytes of static shared memory each.
  static_assert(kResident * (kBytes + 1024 + 512) <= 228 * 1024, "resident CTAs");
  // A further CTA would wait on a TMEM allocation.
  static_assert((kResident + 1) * kBytes > 228 * 1024 || (kResident + 1) * L::kColumns <= 512,
                "TMEM columns");
};

// kExact: K == KP, so that the compiler folds the bounds and the strides.
template <int KP, bool kReverse, bool kBf16, bool kExact> struct StreamOps {
  using L = PhaseLayout<KP>;
  using S = StreamLayout<KP, kReverse>;
  static constexpr unsigned T = S::kThreads, kWarps = T / 32;
  static constexpr unsigned kChunks = KP / kChunk;
  static constexpr unsigned kSteps = (kReverse ? 2 : 1) * kChunks;
  // The reverse's ratio stays in registers between its two products.
  static constexpr bool kKeepRatio = kReverse && kChunks == 1;
  static constexpr unsigned kParts = T / 128; // threads per TMEM lane
  // Epilogue blocks of 4 rows x 8 quads, dealt to the warps round robin: kWalk
  // per warp.
  static constexpr unsigned kWalk = (KP / 4) * (KP / 32) / kWarps;

  // An operation's matrices and exponents.
  struct Op {
    uint4 record;
    const float *left, *right, *mu, *stored;
    int inputs; // exponent of the unnormalised product's inputs
    int own;    // exponent of the stored compressed path (reverse)
    float middle; // this thread's element of the middle vector
  };

  const PhaseArgs &a;
  PhaseShared &sh;
  unsigned char *smem;
  std::uint32_t tmem;
  std::uint32_t &phase;
  bool &ok;
  unsigned K, KK, warp, lane;

  __device__ StreamOps(const PhaseArgs &args, PhaseShared &shared, unsigned char *dynamic_smem,
                       std::uint32_t tmem_base, std::uint32_t &mma_phase, bool &status)
      : a(args), sh(shared), smem(dynamic_smem), tmem(tmem_base), phase(mma_phase), ok(status),
        K(kExact ? KP : args.states), KK(K * K), warp(threadIdx.x / 32),
        lane(threadIdx.x & 31u) {}

  __device__ __forceinline__ const float *PathPtr(std::uint32_t ref) const {
    return (ref & kFlag) ? static_cast<const float *>(a.comps) +
                               static_cast<std::size_t>(ref & kMask) * KK
                         : static_cast<const float *>(a.edge_in) +
                               static_cast<std::size_t>(ref) * KK;
  }
  __device__ __forceinline__ int PathExp(std::uint32_t ref) const {
    return (ref & kFlag) ? a.comp_exp[ref & kMask] : 0;
  }
  __device__ __forceinline__ float *AdjointOf(std::uint32_t ref) const {
    return (ref & kFlag) ? static_cast<float *>(a.comp_mu) +
                               static_cast<std::size_t>(ref & kMask) * KK
                         : static_cast<float *>(a.edge_out) + static_cast<std::size_t>(ref) * KK;
  }
  __device__ __forceinline__ float *MiddleAt(unsigned parity) const {
    return reinterpret_cast<float *>(smem + S::kMiddleAt) + parity * KP;
  }

  // Pointers of operation i; its scalars follow by Scalars.
  __device__ __forceinline__ void Find(Op &op, std::uint32_t i) const {
    op.record = a.compress[i];
    op.left = PathPtr(op.record.x);
    op.right = PathPtr(op.record.z);
    op.mu = static_cast<const float *>(a.comp_mu) + static_cast<std::size_t>(i) * KK;
    op.stored = static_cast<const float *>(a.comps) + static_cast<std::size_t>(i) * KK;
  }
  __device__ __forceinline__ void Scalars(Op &op, std::uint32_t i) const {
    const std::uint32_t ref = op.record.y, obs = op.record.w, node = ref & kMask;
    const unsigned j = threadIdx.x;
    op.inputs = PathExp(op.record.x) + PathExp(op.record.z);
    op.own = kReverse ? a.comp_exp[i] : 0;
    op.middle = 0.0f;
    if (ref & kFlag) {
      op.inputs += a.node_exp[node];
      if (j < K)
        op.middle = static_cast<const float *>(a.nodes)[static_cast<std::size_t>(node) * K + j];
    } else if (j < K) { // input factor, as WideOps::Input
      if (!a.categorical) {
        op.middle = static_cast<const float *>(a.node_in)[static_cast<std::size_t>(node) * K + j];
      } else if (obs == kNone) {
        op.middle = 1.0f;
      } else {
        const unsigned category = a.observations[obs];
        op.middle = category < a.categories
                        ? static_cast<const float *>(a.emission)[category * K + j]
                        : 0.0f;
      }
    }
  }

  // --------------------------------------------------------------- quad maps
  // Quad b of this thread; the column is the same for every b, and rows are a
  // constant apart.
  struct Spot {
    unsigned row, quad;
  };
  // Operand conversion in a direct chunk: 8 rows x 4 quads per warp.
  __device__ __forceinline__ Spot Direct(unsigned b) const {
    return {warp / 4 * 8 + (lane & 7u) + b * (kWarps * 2), warp % 4 * 4 + (lane >> 3)};
  }
  // In a transposed chunk (rows: depths, quads: columns): 4 rows x 8 quads.
  __device__ __forceinline__ Spot Across(unsigned b) const {
    return {warp / (KP / 32) * 4 + (lane & 3u) + b * 16, warp % (KP / 32) * 8 + (lane >> 2)};
  }
  // Global accesses, 4 rows x 8 quads per warp with a row per quarter warp: of
  // a direct chunk (KP rows of 16 quads) and of whole rows (KP / 4 quads).
  __device__ __forceinline__ Spot ChunkRun(unsigned b) const {
    return {warp / 2 * 4 + (lane >> 3) + b * (kWarps * 2), warp % 2 * 8 + (lane & 7u)};
  }
  __device__ __forceinline__ Spot RowRun(unsigned b) const {
    return {warp / (KP / 32) * 4 + (lane >> 3) + b * 16, warp % (KP / 32) * 8 + (lane & 7u)};
  }
  static_assert(kWarps * 128 / KP == 16, "rows between quads");

  // Raw tiles: quad q of row r at q ^ (r % 8) in a direct tile, at
  // q ^ 2 (r % 4) in an across tile, for the quarter warps that read them.
  __device__ __forceinline__ float4 *Raw(unsigned tile) const {
    return reinterpret_cast<float4 *>(smem + S::kSlotsAt + tile * S::kSlotBytes);
  }
  static __device__ __forceinline__ unsigned DirectAt(const Spot &s) {
    return s.row * (kChunk / 4) + (s.quad ^ (s.row & 7u));
  }
  static __device__ __forceinline__ unsigned AcrossAt(const Spot &s) {
    return s.row * (KP / 4) + (s.quad ^ (2 * (s.row & 3u)));
  }
  // Copies a quad, or zeroes (from where nothing is read) if it is not `valid`.
  __device__ __forceinline__ void Copy(void *dst, const float *base, unsigned at,
                                       bool valid) const {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(umma::SmemAddress(dst)),
                 "l"(base + (valid ? at : 0u)), "r"(valid ? 16u : 0u)
                 : "memory");
  }
  // Chunk d0 of a row-major matrix into a raw tile: columns [d0, d0 + 64), or
  // (across) rows [d0, d0 + 64); zero past K.
  __device__ __forceinline__ void FetchDirect(unsigned tile, const float *p, unsigned d0) const {
#pragma unroll
    for (unsigned b = 0; b < 4; ++b) {
      const Spot s = ChunkRun(b);
      Copy(Raw(tile) + DirectAt(s), p, s.row * K + d0 + 4 * s.quad,
           s.row < K && d0 + 4 * s.quad < K);
    }
  }
  __device__ __forceinline__ void FetchAcross(unsigned tile, const float *p, unsigned d0) const {
#pragma unroll
    for (unsigned b = 0; b < 4; ++b) {
      const Spot s = RowRun(b);
      Copy(Raw(tile) + AcrossAt(s), p, (d0 + s.row) * K + 4 * s.quad,
           d0 + s.row < K && 4 * s.quad < K);
    }
  }
  // Starts the copies of one step (one group of copies).
  __device__ __forceinline__ void Fetch(const Op &op, unsigned step) const {
    if constexpr (!kReverse) {
      FetchDirect(0, op.left, step * kChunk);
      FetchAcross(1, op.right, step * kChunk);
    } else if (step < kChunks) {
      if constexpr (kKeepRatio) {
        FetchAcross(0, op.mu, 0);
        FetchAcross(1, op.stored, 0);
      } else {
        FetchDirect(0, op.mu, step * kChunk);
        FetchDirect(1, op.stored, step * kChunk);
      }
      FetchDirect(2, op.right, step * kChunk);
    } else if constexpr (kKeepRatio) {
      FetchAcross(0, op.left, 0);
    } else {
      const unsigned d0 = (step - kChunks) * kChunk;
      FetchAcross(0, op.mu, d0);
      FetchAcross(1, op.stored, d0);
      FetchAcross(2, op.left, d0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // -------------------------------------------------------------- operands
  __device__ __forceinline__ void PutX(unsigned r, unsigned d, float4 v) const {
    Put4<kBf16>(smem + L::kXh, smem + L::kXl, r, d, v);
  }
  __device__ __forceinline__ void PutY(unsigned r, unsigned d, float4 v) const {
    Put4<kBf16>(smem + L::kYh, smem + L::kYl, r, d, v);
  }
  // The 4 x 4 block of lanes 4k .. 4k + 3 (lane: row), transposed.
  __device__ __forceinline__ float4 Transposed(float4 v) const {
    const bool odd = lane & 1u, high = lane & 2u;
    float s0 = odd ? v.x : v.y, s1 = odd ? v.z : v.w;
    s0 = __shfl_xor_sync(kFull, s0, 1);
    s1 = __shfl_xor_sync(kFull, s1, 1);
    if (odd)
      v.x = s0, v.z = s1;
    else
      v.y = s0, v.w = s1;
    s0 = high ? v.x : v.z, s1 = high ? v.y : v.w;
    s0 = __shfl_xor_sync(kFull, s0, 2);
    s1 = __shfl_xor_sync(kFull, s1, 2);
    if (high)
      v.x = s0, v.y = s1;
    else
      v.z = s0, v.w = s1;
    return v;
  }
  static __device__ __forceinline__ float4 Zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
  // This thread's quads of a raw tile.
  __device__ __forceinline__ void TakeDirect(unsigned tile, float4 (&v)[4]) const {
#pragma unroll
    for (unsigned b = 0; b < 4; ++b)
      v[b] = Raw(tile)[DirectAt(Direct(b))];
  }
  __device__ __forceinline__ void TakeAcross(unsigned tile, float4 (&v)[4]) const {
#pragma unroll
    for (unsigned b = 0; b < 4; ++b)
      v[b] = Raw(tile)[AcrossAt(Across(b))];
  }
  // Stores direct quads as operand rows. Rows past K hold zeros that no result
  // in use depends on.
  template <bool kX> __device__ __forceinline__ void PutDirect(const float4 (&v)[4]) const {
#pragma unroll
    for (unsigned b = 0; b < 4; ++b) {
      const Spot s = Direct(b);
      if constexpr (kX)
        PutX(s.row, 4 * s.quad, v[b]);
      else
        PutY(s.row, 4 * s.quad, v[b]);
    }
  }
  // Stores across quads (rows: depths) as quads of operand rows.
  template <bool kX> __device__ __forceinline__ void PutAcross(const float4 (&v)[4]) const {
    float4 t[4];
#pragma unroll
    for (unsigned b = 0; b < 4; ++b)
      t[b] = Transposed(v[b]);
#pragma unroll
    for (unsigned b = 0; b < 4; ++b) {
      const Spot s = Across(b);
      const unsigned r = 4 * s.quad + (lane & 3u), d = s.row & ~3u;
      if constexpr (kX)
        PutX(r, d, t[b]);
      else
        PutY(r, d, t[b]);
    }
  }
  // mu / (stored * 2^shift), as Ratio; one branch for the four quads.
  __device__ __forceinline__ void Ratios(const Op &op, const float4 (&m)[4], const float4 (&s)[4],
                                         float4 (&out)[4]) const {
    const Ratio ratio(op.own - op.inputs);
    if (ratio.exact) {
      const auto one = [&](float mu, float stored) {
        const float q = __fdividef(mu, stored) * ratio.factor;
        return stored > 0.0f ? q : 0.0f;
      };
#pragma unroll
      for (unsigned b = 0; b < 4; ++b)
        out[b] = make_float4(one(m[b].x, s[b].x), one(m[b].y, s[b].y), one(m[b].z, s[b].z),
                             one(m[b].w, s[b].w));
    } else {
#pragma unroll
      for (unsigned b = 0; b < 4; ++b)
        out[b] = make_float4(ratio(m[b].x, s[b].x), ratio(m[b].y, s[b].y),
                             ratio(m[b].z, s[b].z), ratio(m[b].w, s[b].w));
    }
  }

  // Converts a step's raw tiles (once every thread's copies have arrived) into
  // the operands.
  __device__ __forceinline__ void Stage(const Op &op, unsigned step, const float *middle,
                                        float4 (&kept)[4]) const {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float4 u[4], v[4];
    if constexpr (!kReverse) {
      TakeDirect(0, u);
      TakeAcross(1, v);
      const float4 w =
          *reinterpret_cast<const float4 *>(middle + step * kChunk + 4 * Direct(0).quad);
#pragma unroll
      for (unsigned b = 0; b < 4; ++b)
        u[b] = make_float4(u[b].x * w.x, u[b].y * w.y, u[b].z * w.z, u[b].w * w.w);
      PutDirect<true>(u);
      PutAcross<false>(v);
    } else if (step < kChunks) {
      if constexpr (kKeepRatio) {
        TakeAcross(0, u);
        TakeAcross(1, v);
      } else {
        TakeDirect(0, u);
        TakeDirect(1, v);
      }
      Ratios(op, u, v, kept);
      TakeDirect(2, u);
      if constexpr (kKeepRatio) {
#pragma unroll
        for (unsigned b = 0; b < 4; ++b) {
          const Spot s = Across(b);
          PutX(s.row, 4 * s.quad, kept[b]);
        }
      } else {
        PutDirect<true>(kept);
      }
      PutDirect<false>(u);
    } else if constexpr (kKeepRatio) {
      TakeAcross(0, u);
      PutAcross<false>(kept);
      PutAcross<true>(u);
    } else {
      TakeAcross(0, u);
      TakeAcross(1, v);
      Ratios(op, u, v, kept);
      TakeAcross(2, u);
      PutAcross<false>(kept);
      PutAcross<true>(u);
    }
  }

  // ------------------------------------------------------------- epilogues
  // Tiles of KP x KP floats in the operand buffers; quad q of row r sits at
  // q ^ (r % 8), so that eight rows' quads fall on different banks.
  __device__ __forceinline__ float4 *TileQuad(unsigned tile, unsigned r, unsigned q) const {
    return reinterpret_cast<float4 *>(smem) + (tile * KP + r) * (KP / 4) + (q ^ (r & 7u));
  }
  __device__ __forceinline__ void TileRow(unsigned tile, unsigned r, unsigned c,
                                          const float (&row)[32]) const {
#pragma unroll
    for (unsigned q = 0; q < 8; ++q)
      if (c + 4 * q < K)
        *TileQuad(tile, r, c / 4 + q) =
            make_float4(row[4 * q], row[4 * q + 1], row[4 * q + 2], row[4 * q + 3]);
  }

  __device__ __forceinline__ void FinishForward(std::uint32_t i, const Op &op) const {
    const unsigned row = threadIdx.x % 128, c = threadIdx.x / 128 * 32;
    const std::uint32_t lane_base = tmem + ((row & ~31u) << 16);
    float values[32];
    SplitSum32<KP>(lane_base, c, values, kBf16);
    float m = 0.0f;
#pragma unroll
    for (unsigned q = 0; q < 32; ++q)
      if (row < K && c + q < K)
        m = m < values[q] ? values[q] : m;
    const int s = ExponentOf(CtaMax<T>(m, sh));
    if (row < K) {
#pragma unroll
      for (unsigned q = 0; q < 32; ++q)
        values[q] = ScalePow2(values[q], -s);
      TileRow(0, row, c, values);
    }
    __syncthreads();
    float *out = static_cast<float *>(a.comps) + static_cast<std::size_t>(i) * KK;
#pragma unroll
    for (unsigned b = 0; b < kWalk; ++b) {
      const Spot at = RowRun(b);
      if (at.row < K && 4 * at.quad < K)
        *reinterpret_cast<float4 *>(out + at.row * K + 4 * at.quad) =
            *TileQuad(0, at.row, at.quad);
    }
    if (threadIdx.x == 0)
      a.comp_exp[i] = op.inputs + s;
  }

  // Quads of the left and right matrices that the epilogue multiplies: the
  // first kAtOnce of the walk are loaded before the last products are waited
  // for.
  static constexpr unsigned kAtOnce = 4;
  __device__ __forceinline__ void LoadPair(const Op &op, unsigned b0, float4 (&l)[kAtOnce],
                                           float4 (&r)[kAtOnce]) const {
#pragma unroll
    for (unsigned b = 0; b < kAtOnce; ++b) {
      const Spot at = RowRun(b0 + b);
      const bool valid = at.row < K && 4 * at.quad < K;
      const unsigned offset = valid ? at.row * K + 4 * at.quad : 0u;
      l[b] = *reinterpret_cast<const float4 *>(op.left + offset);
      r[b] = *reinterpret_cast<const float4 *>(op.right + offset);
    }
  }

  // Left adjoint left[r][m] middle[m] P1[r][m], right adjoint right[m][c]
  // middle[m] P2[m][c], middle adjoint the row sums of the latter.
  __device__ __forceinline__ void FinishReverse(const Op &op, const float *middle,
                                                float4 (&l)[kAtOnce],
                                                float4 (&r)[kAtOnce]) const {
    const unsigned row = threadIdx.x % 128, c = threadIdx.x / 128 * 32;
    const std::uint32_t lane_base = tmem + ((row & ~31u) << 16);
#pragma unroll
    for (unsigned tile = 0; tile < 2; ++tile) {
      float values[32];
      umma::Load32(lane_base + tile * KP + c, values);
      if (row < K)
        TileRow(tile, row, c, values);
    }
    float *left_out = AdjointOf(op.record.x);
    float *right_out = AdjointOf(op.record.z);
    __syncthreads();
#pragma unroll
    for (unsigned b0 = 0; b0 < kWalk; b0 += kAtOnce) {
      if (b0 != 0)
        LoadPair(op, b0, l, r);
      float4 p1[kAtOnce], p2[kAtOnce];
      float partial[kAtOnce];
#pragma unroll
      for (unsigned b = 0; b < kAtOnce; ++b) {
        const Spot at = RowRun(b0 + b); // rows past K: within the tiles
        p1[b] = *TileQuad(0, at.row, at.quad);
        p2[b] = *TileQuad(1, at.row, at.quad);
      }
      const float4 w = *reinterpret_cast<const float4 *>(middle + 4 * RowRun(0).quad);
#pragma unroll
      for (unsigned b = 0; b < kAtOnce; ++b) {
        const Spot at = RowRun(b0 + b);
        const float mr = middle[at.row];
        p1[b] = make_float4(l[b].x * w.x * p1[b].x, l[b].y * w.y * p1[b].y,
                            l[b].z * w.z * p1[b].z, l[b].w * w.w * p1[b].w);
        p2[b] = make_float4(r[b].x * mr * p2[b].x, r[b].y * mr * p2[b].y, r[b].z * mr * p2[b].z,
                            r[b].w * mr * p2[b].w);
        const bool valid = at.row < K && 4 * at.quad < K;
        partial[b] = valid ? (p2[b].x + p2[b].y) + (p2[b].z + p2[b].w) : 0.0f;
        if (valid) {
          *reinterpret_cast<float4 *>(left_out + at.row * K + 4 * at.quad) = p1[b];
          *reinterpret_cast<float4 *>(right_out + at.row * K + 4 * at.quad) = p2[b];
        }
      }
      // The row's sum over this block's 32 columns, where the block's first
      // quad (the quarter warp's first lane's) was.
#pragma unroll
      for (unsigned offset = 1; offset < 8; offset *= 2)
#pragma unroll
        for (unsigned b = 0; b < kAtOnce; ++b)
          partial[b] += __shfl_xor_sync(kFull, partial[b], offset);
      if ((lane & 7u) == 0) {
#pragma unroll
        for (unsigned b = 0; b < kAtOnce; ++b) {
          const Spot at = RowRun(b0 + b);
          TileQuad(1, at.row, at.quad)->x = partial[b];
        }
      }
    }
    __syncthreads();
    const unsigned j = threadIdx.x;
    if (j < K) {
      float total = 0.0f;
      for (unsigned q = 0; 4 * q < K; q += 8)
        total += TileQuad(1, j, q)->x;
      static_cast<float *>(a.node_out)[static_cast<std::size_t>(op.record.y & kMask) * K + j] =
          total;
    }
  }

  // Operations first, first + stride, ... below `count` of this launch.
  __device__ __forceinline__ void Run(std::uint32_t first, std::uint32_t stride) const {
    Op op, next;
    Find(op, a.offset + first);
    Fetch(op, 0);
    Scalars(op, a.offset + first);
    if (threadIdx.x < KP)
      MiddleAt(0)[threadIdx.x] = op.middle;
    unsigned parity = 0;
    for (std::uint32_t t = first; t < a.count; t += stride, parity ^= 1u) {
      const std::uint32_t i = a.offset + t;
      const bool more = t + stride < a.count;
      if (more)
        Find(next, i + stride);
      const float *middle = MiddleAt(parity);
      float4 kept[4], l[kAtOnce], r[kAtOnce];
#pragma unroll
      for (unsigned step = 0; step < kSteps; ++step) {
        Stage(op, step, middle, kept);
        if constexpr (!kReverse)
          IssueChunk<KP, true>(smem, sh, tmem, step, kBf16);
        else
          IssueChunk<KP, false>(smem, sh, tmem + step / kChunks * KP, step % kChunks, kBf16);
        // Every thread has read the raw tiles (IssueChunk's barrier).
        if (step + 1 < kSteps)
          Fetch(op, step + 1);
        else if (more)
          Fetch(next, 0);
        if (step + 1 == kSteps) {
          if constexpr (kReverse)
            LoadPair(op, 0, l, r);
          if (more)
            Scalars(next, i + stride);
        }
        ok = WaitChunk(sh, phase) && ok;
      }
      if (more && threadIdx.x < KP)
        MiddleAt(parity ^ 1u)[threadIdx.x] = next.middle;
      if constexpr (kReverse)
        FinishReverse(op, middle, l, r);
      else
        FinishForward(i, op);
      // The tiles are read before the next operands are stored (Stage's
      // barrier), the accumulators before the next products (IssueChunk's).
      if (more)
        op = next;
    }
  }
};

// The compress kinds for K a multiple of 4: a persistent grid, CTA b taking
// operations b, b + grid, ...
template <int KP, bool kReverse, bool kBf16, bool kExact>
__global__ void __launch_bounds__(PhaseLayout<KP>::kThreads,
                                  StreamLayout<KP, kReverse>::kResident)
    WideStreamKernel(PhaseArgs args) {
  using L = PhaseLayout<KP>;
  // (Aligned to 128 bytes only: 1024 would cost a KB that two CTAs do not have.)
  extern __shared__ __align__(128) unsigned char stream_smem[];
  __shared__ PhaseShared sh;
  std::uint32_t phase = 0;
  bool ok = true;
  if (threadIdx.x == 0)
    umma::BarrierInit(&sh.barrier);
  if (threadIdx.x < 32)
    umma::Allocate(&sh.tmem, L::kColumns);
  umma::FenceBeforeSync();
  __syncthreads();
  umma::FenceAfterSync();
  {
    const StreamOps<KP, kReverse, kBf16, kExact> ops(args, sh, stream_smem, sh.tmem, phase, ok);
    if (blockIdx.x < args.count)
      ops.Run(blockIdx.x, gridDim.x);
  }
  if (!ok && threadIdx.x == 0)
    atomicOr(args.error, kErrorTensorTimeout);
  umma::FenceBeforeSync();
  __syncthreads();
  umma::FenceAfterSync();
  if (threadIdx.x < 32)
    umma::Deallocate(sh.tmem, L::kColumns);
}

} // namespace wide
} // namespace thmm

#endif // THMM_WIDE_STREAM_CUH_
