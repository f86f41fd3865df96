// FlashAttention forward for few query rows (decode and short prompts against a long key/value cache), sm_100a.
//
// What bounds it is reading K and V once.  The general kernel (fa_fwd_sm100.cuh) gives every query head its own 256-row
// block, so with one new token per sequence 255 of 256 rows are padding, a grouped-query cache is read once per QUERY head
// (from L2, but through the same per-tile chain) and a block walks all keys alone.  Here
//   - the query heads that share a key/value head are packed into one 128-row tile (row = head * Sq + position; one TMA box
//     of Sq x heads rows), so a K/V tile is loaded and multiplied once for all of them;
//   - the key tiles of all (batch, kv head) items form ONE list of T = items * nkv tiles that is cut into `pipes` equal
//     runs.  A run may start or end inside an item: such a segment leaves fp32 partial results (O / l and the base-2 LSE)
//     in the workspace and fa_split_combine_kernel merges them; a segment that covers its item writes the output itself;
//   - a CTA carries two independent pipelines (softmax warpgroup, MMA warp, TMA warp, K/V ring and 256 TMEM columns each),
//     so one pipeline's softmax -> MMA chain (~3000 cycles a tile) runs under the other's, and together they stay ahead of
//     the ~2700 cycles a 64 KB tile takes at an SM's share of the HBM rate.
//
// B16 Hq64 Hkv8 D128 bf16, one row, 6001 keys: 547 us with the general kernel (0.72 TB/s of K and V), 71 us here (5.5 TB/s);
// B8 Hq32 Hkv8, 16 rows, 4096 keys: 111 -> 37 us; B64 Hq32 Hkv32, one row, 512 keys: 112 -> 89 us (6.0 TB/s); B1 H8, 128
// rows, 4096 keys: 57 -> 21 us; a prompt of 120 rows on itself: 7.4 us either way.
#pragma once

#include "fa_fwd_sm100.cuh"
#include "fa_split_plan.h"

namespace hb {

static_assert(kFaSplitTile == kTileM && kFaSplitTile == kTileN, "the plan and the kernel cut the same tiles");
constexpr int kSplitThreads = 384;  // 2 softmax warpgroups, 2 MMA warps, 2 TMA warps
enum FaSplitRole : uint32_t { kRoleSplitSoftmax = 6, kRoleSplitMma = 7, kRoleSplitTma = 8, kRoleSplitDrain = 9 };

struct alignas(64) FaSplitParams {
  CUtensorMap tm_q, tm_k, tm_v;
  void* o;
  float* lse;       // optional
  float* part_o;    // [2 * pipes][rows][D] fp32, O / l of a partial segment
  float* part_lse;  // [2 * pipes][rows] base-2 LSE of a partial segment (-inf: no visible key)
  uint32_t* status;
  long long o_sb, o_sh, o_ss;
  int B, Hq, Hkv, Sq, Skv;
  int group;     // Hq / Hkv
  int causal;
  FaSplitPlan plan;
  float scale_log2;
};

// RC: rows the shared-memory Q tile holds (64 or 128)
template <typename T, int D, int RC>
struct FaSplitSmem {
  static constexpr int kQBytes = RC * D * 2;
  static constexpr int kTileBytes = kTileN * D * 2;
  // as many K/V tiles per pipeline as fit in 227 KB next to the Q tiles
  static constexpr int kStages = D == 128 ? (RC == 64 ? 3 : 2) : 6;
  alignas(1024) uint8_t q[2][kQBytes];
  // The Q operand has M = 128 rows whatever RC is: with RC = 64 the tensor core also reads the 64 rows behind (pipeline 0) or
  // in front of (pipeline 1) the tile, always inside this struct.  Those rows only feed rows of S and O that nobody reads.
  alignas(1024) uint8_t kv[2][kStages][kTileBytes];
  uint64_t q_full[2], q_empty[2];
  uint64_t kv_full[2][kStages], kv_empty[2][kStages];
  uint64_t s_full[2], p_full[2], o_full[2];
  uint64_t drain[2];
  uint32_t tmem_base;
  uint32_t abort_flag;
};

struct FaSegment {
  int item, b, hq0, hkv;
  int heads;   // live query heads of the row tile
  int j0, j1;  // key tiles [j0, j1)
};

__device__ __forceinline__ void fa_split_item(const FaSplitParams& p, int item, FaSegment& g) {
  g.item = item;
  const int hg = item % p.plan.hgroups, bk = item / p.plan.hgroups;
  g.b = bk / p.Hkv;
  g.hkv = bk - g.b * p.Hkv;
  g.hq0 = g.hkv * p.group + hg * p.plan.hb;
  g.heads = min(p.plan.hb, p.group - hg * p.plan.hb);
}
__device__ __forceinline__ FaSegment fa_split_segment(const FaSplitParams& p, long long t, long long end) {
  FaSegment g;
  int item;
  fa_split_segment(p.plan, t, end, item, g.j0, g.j1);
  fa_split_item(p, item, g);
  return g;
}

// Rows of pipeline 1 that fit 64 rows sit on TMEM lanes 64.. (its Q operand starts 64 rows before its tile): a decode call
// has one live warp per pipeline, and lanes 0 of both would put the two on the same sub-partition and its exponential unit.
template <int RC>
__device__ __forceinline__ constexpr int fa_split_row0(int i) {
  return RC == 64 ? 64 * i : 0;
}

// End of a segment: O / l of the thread's row (its lane of O at tO) to the output, or as a partial result.
template <typename T, int D>
__device__ __forceinline__ void fa_split_store_segment(const FaSplitParams& p, const FaSegment& g, uint32_t tO, int w, bool first, int row,
                                                       int head, int pos, float m, float l) {
  const bool whole = g.j0 == 0 && g.j1 == p.plan.nkv;
  const bool live = row < p.plan.rows && head < g.heads;
  const float inv_l = (l > 0.f) ? (1.0f / l) : 0.f;
  const float lse2 = (l > 0.f) ? (m * p.scale_log2 + fast_log2(l)) : -INFINITY;
  const long long slot = 2ll * w + (first ? 0 : 1);
  T* orow = static_cast<T*>(p.o) + g.b * p.o_sb + (g.hq0 + head) * p.o_sh + static_cast<long long>(pos) * p.o_ss;
  float* prow = p.part_o + (slot * p.plan.rows + row) * D;
#pragma unroll
  for (int c = 0; c < D / 32; ++c) {
    uint32_t r[32];
    __syncwarp();
    tmem_ld32(tO + c * 32, r);
    tmem_wait_ld();
    if (live && whole) {
#pragma unroll
      for (int e = 0; e < 32; e += 8) {
        uint4 o;
        o.x = Pack2<T>::pack(__uint_as_float(r[e]) * inv_l, __uint_as_float(r[e + 1]) * inv_l);
        o.y = Pack2<T>::pack(__uint_as_float(r[e + 2]) * inv_l, __uint_as_float(r[e + 3]) * inv_l);
        o.z = Pack2<T>::pack(__uint_as_float(r[e + 4]) * inv_l, __uint_as_float(r[e + 5]) * inv_l);
        o.w = Pack2<T>::pack(__uint_as_float(r[e + 6]) * inv_l, __uint_as_float(r[e + 7]) * inv_l);
        *reinterpret_cast<uint4*>(orow + c * 32 + e) = o;
      }
    } else if (live) {
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        *reinterpret_cast<float4*>(prow + c * 32 + e) =
            make_float4(__uint_as_float(r[e]) * inv_l, __uint_as_float(r[e + 1]) * inv_l, __uint_as_float(r[e + 2]) * inv_l,
                        __uint_as_float(r[e + 3]) * inv_l);
      }
    }
  }
  if (live && whole) {
    if (p.lse != nullptr)
      p.lse[(static_cast<long long>(g.b) * p.Hq + g.hq0 + head) * p.Sq + pos] = lse2 * 0.6931471805599453f;
  } else if (live) {
    p.part_lse[slot * p.plan.rows + row] = lse2;
  }
}

// The softmax of calls with at most 8 NH rows (NH 1 or 2), decode above all.  With a thread a row, one warp turned 128 columns over for
// a handful of live lanes: 1500 cycles of the 2500 to 2900 that a step of such a pipeline took, which with 64-wide heads (32 KB a step)
// is slower than HBM.  Here a row lies on the four lanes of a quad, 32 columns each: a quarter of the exponentials (half, with 9 to 16
// rows), two shuffles for the maximum, the sum put together at the end of the segment.
// us a thread a row -> a quad a row: D 64 B54 H12 393 keys 26.0 -> 21.1, B2 H32 Sq 2 15777 keys 55.0 -> 50.9, B25 Hq32 Hkv8 2189 keys
// 29.5 -> 27.0, B32 H4 559 keys 12.3 -> 9.6; D 128 B62 H16 Sq 3 442 keys 48.0 -> 44.7, B13 Hq32 Hkv4 6060 keys 36.6 -> 35.5, B14 H1 Sq 8 146
// keys 7.5 -> 6.2, B16 Hq64 Hkv8 6001 keys 70.2 -> 69.3.
template <typename T, int D, int NH, int RC>
__device__ __forceinline__ void fa_split_softmax_few(const FaSplitParams& p, FaSplitSmem<T, D, RC>& s, const AbortCtx& ctx, uint32_t tmem,
                                                     int i, int w) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const uint32_t tS = tmem + lane_off + static_cast<uint32_t>(i * 256), tO = tS + 128;
  const int c = lane & 3, lane_head = lane / p.Sq;
  const float scale_log2 = p.scale_log2;
  const int past = p.Skv - p.Sq;
  uint32_t s_phase = 0, o_phase = 0;
  int row[NH], pos[NH];
#pragma unroll
  for (int h = 0; h < NH; ++h) {
    row[h] = (lane >> 2) + 8 * h;
    pos[h] = row[h] % p.Sq;
  }
  // the value of the lane's own row, for whole rows on lanes
  auto of_row = [&](const float (&x)[NH]) {
    float y = __shfl_sync(0xffffffffu, x[0], (lane & 7) * 4);
    if constexpr (NH == 2) {
      const float z = __shfl_sync(0xffffffffu, x[1], (lane & 7) * 4);
      if (lane & 8) y = z;
    }
    return y;
  };

  const long long end = fa_split_begin(p.plan, w + 1);
  bool first = true;
  for (long long t = fa_split_begin(p.plan, w); t < end; first = false) {
    const FaSegment g = fa_split_segment(p, t, end);
    t += g.j1 - g.j0;
    float m[NH], l[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      m[h] = -INFINITY;
      l[h] = 0.f;
    }

    for (int j = g.j0; j < g.j1; ++j) {
      if (!mbar_wait_warp(&s.s_full[i], s_phase, ctx, kRoleSplitSoftmax)) return;
      s_phase ^= 1;
      tc_fence_after();
      uint32_t r[64], pk[32];
      tmem_ld_16x128cols(tS, r);
      tmem_wait_ld();
      const int col0 = j * kTileN;
      const bool need_mask = col0 + kTileN > p.Skv || (p.causal && col0 + kTileN - 1 > past);
      float alpha[NH];
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        if (need_mask) {
          int lim = p.Skv - 1 - col0;
          if (p.causal) lim = min(lim, past + pos[h] - col0);
          lim -= 2 * c;
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            uint32_t* x = &r[4 * q + 2 * h];
            x[0] = 8 * q <= lim ? x[0] : 0xff800000u;  // -inf
            x[1] = 8 * q + 1 <= lim ? x[1] : 0xff800000u;
          }
        }
        float mx[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) mx[q] = fmaxf(__uint_as_float(r[4 * q + 2 * h]), __uint_as_float(r[4 * q + 2 * h + 1]));
#pragma unroll
        for (int q = 4; q < 16; ++q)
          mx[q & 3] = max3(mx[q & 3], __uint_as_float(r[4 * q + 2 * h]), __uint_as_float(r[4 * q + 2 * h + 1]));
        float row_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        row_max = fmaxf(row_max, __shfl_xor_sync(0xffffffffu, row_max, 1));
        row_max = fmaxf(row_max, __shfl_xor_sync(0xffffffffu, row_max, 2));

        // the same rule as the general kernel: a maximum that grew by less than 2^8 is not adopted
        const float m_cand = fmaxf(m[h], row_max);
        const float diff = (m[h] - m_cand) * scale_log2;
        const bool adopt = row[h] < p.plan.rows && diff < -FaTraits<T>::kRescaleThreshold;  // padding rows never ask for a rescale
        alpha[h] = adopt ? fast_exp2(diff) : 1.f;
        m[h] = adopt ? m_cand : m[h];
        const float m_scaled = (m[h] == -INFINITY) ? 0.f : m[h] * scale_log2;

        const uint64_t sc2 = pack_f32x2(scale_log2, scale_log2), nm2 = pack_f32x2(-m_scaled, -m_scaled);
        uint64_t sa = pack_f32x2(0.f, 0.f), sb = sa;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const uint64_t x =
              fma_f32x2(pack_f32x2(__uint_as_float(r[4 * q + 2 * h]), __uint_as_float(r[4 * q + 2 * h + 1])), sc2, nm2);
          float a, b;
          unpack_f32x2(x, a, b);
          a = fast_exp2(a);
          b = fast_exp2(b);
          if (q & 1) sb = add_f32x2(sb, pack_f32x2(a, b));
          else sa = add_f32x2(sa, pack_f32x2(a, b));
          pk[2 * q + h] = Pack2<T>::pack(a, b);
          if (NH == 1) pk[2 * q + 1] = 0u;
        }
        float sum0, sum1, sum2, sum3;
        unpack_f32x2(sa, sum0, sum1);
        unpack_f32x2(sb, sum2, sum3);
        l[h] = l[h] * alpha[h] + ((sum0 + sum1) + (sum2 + sum3));  // of this lane's columns
      }
      tmem_st_16x64cols(tS, pk);
      // O is rescaled a row a lane: S(j) was committed behind PV(j - 1), so that product is complete, and PV(j) is only issued after
      // this warp's arrival on p_full
      bool moved = alpha[0] != 1.f;
      if constexpr (NH == 2) moved = moved || alpha[1] != 1.f;
      if (j > g.j0 && __any_sync(0xffffffffu, moved)) {
        const float a = of_row(alpha);
#pragma unroll
        for (int q = 0; q < D / 32; ++q) {
          uint32_t o[32];
          tmem_ld32(tO + q * 32, o);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * a);
          tmem_st32(tO + q * 32, o);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.p_full[i]);
    }

    if (!mbar_wait_warp(&s.o_full[i], o_phase, ctx, kRoleSplitSoftmax)) return;
    o_phase ^= 1;
    tc_fence_after();
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
      l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
    }
    const float m_row = of_row(m), l_row = of_row(l);
    fa_split_store_segment<T, D>(p, g, tO, w, first, lane, lane_head, lane - lane_head * p.Sq, m_row, l_row);
    // the next segment's first product overwrites O: it waits for this warp's next arrival on p_full
    tc_fence_before();
    __syncwarp();
  }
}

template <typename T, int D, int RC>
__device__ __forceinline__ void fa_split_softmax_role(const FaSplitParams& p, FaSplitSmem<T, D, RC>& s, const AbortCtx& ctx,
                                                      uint32_t tmem, int i, int w) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = (threadIdx.x & (kTileM - 1)) - fa_split_row0<RC>(i);
  const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const uint32_t tS = tmem + lane_off + static_cast<uint32_t>(i * 256), tO = tS + 128;
  const float scale_log2 = p.scale_log2;
  const int head = row / p.Sq, pos = row - head * p.Sq;
  const int past = p.Skv - p.Sq;
  uint32_t s_phase = 0, o_phase = 0;

  const long long end = fa_split_begin(p.plan, w + 1);
  bool first = true;
  for (long long t = fa_split_begin(p.plan, w); t < end; first = false) {
    const FaSegment g = fa_split_segment(p, t, end);
    t += g.j1 - g.j0;
    float m = -INFINITY, l = 0.f;

    for (int j = g.j0; j < g.j1; ++j) {
      if (!mbar_wait_warp(&s.s_full[i], s_phase, ctx, kRoleSplitSoftmax)) return;
      s_phase ^= 1;
      tc_fence_after();
      uint32_t v[kTileN];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, &v[c * 32]);
      tmem_wait_ld();

      const int col0 = j * kTileN;
      if (col0 + kTileN > p.Skv || (p.causal && col0 + kTileN - 1 > past)) {
        int lim = p.Skv - 1 - col0;
        if (p.causal) lim = min(lim, past + pos - col0);
#pragma unroll
        for (int c = 0; c < kTileN; ++c) v[c] = (c <= lim) ? v[c] : 0xff800000u;  // -inf
      }
      float mx[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) mx[c] = __uint_as_float(v[c]);
#pragma unroll
      for (int c = 4; c < kTileN; c += 8) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (c + 4 < kTileN) mx[e] = max3(mx[e], __uint_as_float(v[c + e]), __uint_as_float(v[c + 4 + e]));
          else mx[e] = fmaxf(mx[e], __uint_as_float(v[c + e]));
        }
      }
      const float row_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));

      // the same rule as the general kernel: a maximum that grew by less than 2^8 is not adopted
      const float m_cand = fmaxf(m, row_max);
      const float diff = (m - m_cand) * scale_log2;
      const bool adopt = row < p.plan.rows && diff < -FaTraits<T>::kRescaleThreshold;  // padding rows never ask for a rescale
      const float alpha = adopt ? fast_exp2(diff) : 1.f;
      m = adopt ? m_cand : m;
      const float m_scaled = (m == -INFINITY) ? 0.f : m * scale_log2;

      const uint64_t sc2 = pack_f32x2(scale_log2, scale_log2), nm2 = pack_f32x2(-m_scaled, -m_scaled);
      uint64_t sa = pack_f32x2(0.f, 0.f), sb = sa;
#pragma unroll
      for (int q = 0; q < kTileN / 32; ++q) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const int c = q * 32 + e;
          const uint64_t x0 = fma_f32x2(pack_f32x2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), sc2, nm2);
          const uint64_t x1 = fma_f32x2(pack_f32x2(__uint_as_float(v[c + 2]), __uint_as_float(v[c + 3])), sc2, nm2);
          float a0, a1, b0, b1;
          unpack_f32x2(x0, a0, a1);
          unpack_f32x2(x1, b0, b1);
          a0 = fast_exp2(a0);
          a1 = fast_exp2(a1);
          b0 = fast_exp2(b0);
          b1 = fast_exp2(b1);
          sa = add_f32x2(sa, pack_f32x2(a0, a1));
          sb = add_f32x2(sb, pack_f32x2(b0, b1));
          pk[e / 2] = Pack2<T>::pack(a0, a1);
          pk[e / 2 + 1] = Pack2<T>::pack(b0, b1);
        }
        tmem_st16(tS + q * 16, pk);
      }
      float sum0, sum1, sum2, sum3;
      unpack_f32x2(sa, sum0, sum1);
      unpack_f32x2(sb, sum2, sum3);
      l = l * alpha + ((sum0 + sum1) + (sum2 + sum3));
      // O is rescaled by the row's own thread, once the scores are out of its registers: S(j) was committed behind PV(j - 1), so that product is complete, and PV(j)
      // is only issued after this thread's arrival on p_full
      if (j > g.j0 && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(tO + c * 32, r);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
          tmem_st32(tO + c * 32, r);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.p_full[i]);
    }

    // end of the segment: O / l to the output, or as a partial result
    if (!mbar_wait_warp(&s.o_full[i], o_phase, ctx, kRoleSplitSoftmax)) return;
    o_phase ^= 1;
    tc_fence_after();
    fa_split_store_segment<T, D>(p, g, tO, w, first, row, head, pos, m, l);
    // the next segment's first product overwrites O: it waits for this thread's next arrival on p_full
    tc_fence_before();
    __syncwarp();
  }
}

template <typename T, int D, int RC>
__device__ __forceinline__ void fa_split_mma_role(const FaSplitParams& p, FaSplitSmem<T, D, RC>& s, const AbortCtx& ctx,
                                                  uint32_t tmem, int i, int w) {
  using Smem = FaSplitSmem<T, D, RC>;
  constexpr uint32_t kFmt = FaTraits<T>::kFormat;
  constexpr uint32_t idesc_qk = make_idesc(kFmt, kTileM, kTileN, 0, 0);
  constexpr uint32_t idesc_pv = make_idesc(kFmt, kTileM, D, 0, 1);
  constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // see fa_mma_role
  constexpr uint32_t kLboK = (16u >> 4) << 16;
  constexpr uint32_t kLboV = (kTileN * 128u >> 4) << 16;
  constexpr uint32_t kTile16 = Smem::kTileBytes >> 4;
  constexpr uint32_t kQSub = RC * 128u >> 4, kKSub = kTileN * 128u >> 4;  // next 64 head_dim columns of Q / K
  auto desc = [](uint32_t lo) -> uint64_t { return (static_cast<uint64_t>(kDescHi) << 32) | lo; };
  const uint32_t q_lo = ((smem_u32(s.q[i]) - static_cast<uint32_t>(fa_split_row0<RC>(i)) * 128u) >> 4) | kLboK;
  const uint32_t kv_lo = smem_u32(s.kv[i][0]) >> 4;
  const uint32_t tS = tmem + static_cast<uint32_t>(i * 256), tO = tS + 128;
  const bool leader = elect_one();
  uint32_t slot = 0, phase = 0, q_phase = 0, p_phase = 0;
  auto advance = [&]() {
    if (++slot == Smem::kStages) {
      slot = 0;
      phase ^= 1;
    }
  };

  const long long end = fa_split_begin(p.plan, w + 1);
  for (long long t = fa_split_begin(p.plan, w); t < end;) {
    const FaSegment g = fa_split_segment(p, t, end);
    t += g.j1 - g.j0;
    if (!mbar_wait_warp(&s.q_full[i], q_phase, ctx, kRoleSplitMma)) return;
    q_phase ^= 1;
    for (int j = g.j0; j <= g.j1; ++j) {
      if (j > g.j0) {  // O += P(j - 1) V(j - 1)
        if (!mbar_wait_warp(&s.kv_full[i][slot], phase, ctx, kRoleSplitMma)) return;
        if (!mbar_wait_warp(&s.p_full[i], p_phase, ctx, kRoleSplitMma)) return;
        p_phase ^= 1;
        tc_fence_after();
        const uint32_t va = (kv_lo + slot * kTile16) | kLboV;
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < kTileN / 16; ++kk)
            umma_ts_f16(tO, tS + static_cast<uint32_t>(kk * 8), desc(va + static_cast<uint32_t>(kk) * (16u * 128u >> 4)), idesc_pv,
                        (kk > 0 || j > g.j0 + 1) ? 1u : 0u);
          umma_commit(&s.kv_empty[i][slot]);
          if (j == g.j1) umma_commit(&s.o_full[i]);
        }
        advance();
      }
      if (j < g.j1) {  // S = Q K(j)
        if (!mbar_wait_warp(&s.kv_full[i][slot], phase, ctx, kRoleSplitMma)) return;
        tc_fence_after();
        const uint32_t ka = (kv_lo + slot * kTile16) | kLboK;
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            umma_ss_f16(tS, desc(q_lo + static_cast<uint32_t>(kk >> 2) * kQSub + static_cast<uint32_t>(kk & 3) * 2u),
                        desc(ka + static_cast<uint32_t>(kk >> 2) * kKSub + static_cast<uint32_t>(kk & 3) * 2u), idesc_qk,
                        kk > 0 ? 1u : 0u);
          umma_commit(&s.s_full[i]);
          umma_commit(&s.kv_empty[i][slot]);
          if (j + 1 == g.j1) umma_commit(&s.q_empty[i]);
        }
        advance();
      }
    }
  }
}

template <typename T, int D, int RC>
__device__ __forceinline__ void fa_split_tma_role(const FaSplitParams& p, FaSplitSmem<T, D, RC>& s, const AbortCtx& ctx, int i,
                                                  int w) {
  using Smem = FaSplitSmem<T, D, RC>;
  uint32_t slot = 0, phase = 1, q_phase = 1;  // "empty" barriers start out free
  const long long end = fa_split_begin(p.plan, w + 1);
  for (long long t = fa_split_begin(p.plan, w); t < end;) {
    const FaSegment g = fa_split_segment(p, t, end);
    t += g.j1 - g.j0;
    auto load_kv = [&](const CUtensorMap* tm, int j) -> bool {
      if (!mbar_wait(&s.kv_empty[i][slot], phase, ctx, kRoleSplitTma)) return false;
      mbar_arrive_expect_tx(&s.kv_full[i][slot], Smem::kTileBytes);
#pragma unroll
      for (int h = 0; h < D / 64; ++h)
        tma_load_4d(s.kv[i][slot] + h * (kTileN * 128), tm, &s.kv_full[i][slot], h * 64, j * kTileN, g.hkv, g.b);
      if (++slot == Smem::kStages) {
        slot = 0;
        phase ^= 1;
      }
      return true;
    };
    if (!mbar_wait(&s.q_empty[i], q_phase, ctx, kRoleSplitTma)) return;
    q_phase ^= 1;
    mbar_arrive_expect_tx(&s.q_full[i], static_cast<uint32_t>(p.plan.rows) * D * 2u);
#pragma unroll
    for (int h = 0; h < D / 64; ++h) tma_load_4d(s.q[i] + h * (RC * 128), &p.tm_q, &s.q_full[i], h * 64, 0, g.hq0, g.b);
    if (!load_kv(&p.tm_k, g.j0)) return;
    for (int j = g.j0; j < g.j1; ++j) {
      if (!load_kv(&p.tm_v, j)) return;
      if (j + 1 < g.j1 && !load_kv(&p.tm_k, j + 1)) return;
    }
  }
}

template <typename T, int D, int RC, int NH>
__device__ __forceinline__ void fa_split_softmax(const FaSplitParams& p, FaSplitSmem<T, D, RC>& s, const AbortCtx& ctx, uint32_t tmem, int i,
                                                 int w) {
  if constexpr (NH > 0) fa_split_softmax_few<T, D, NH, RC>(p, s, ctx, tmem, i, w);
  else fa_split_softmax_role<T, D, RC>(p, s, ctx, tmem, i, w);
}

// NH: 0, or 1 or 2 for at most 8 NH rows (fa_split_softmax_few)
template <typename T, int D, int RC, int NH>
__global__ void __launch_bounds__(kSplitThreads, 1) fa_split_kernel(const __grid_constant__ FaSplitParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  using Smem = FaSplitSmem<T, D, RC>;
  Smem& s = *reinterpret_cast<Smem*>(smem_raw);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  AbortCtx ctx{&s.abort_flag, p.status};
  const int softmax_warps = (p.plan.rows + 31) / 32;  // per pipeline; the others have no live row

  if (threadIdx.x == 0) {
    s.abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s.q_full[i], 1);
      mbar_init(&s.q_empty[i], 1);
      mbar_init(&s.s_full[i], 1);
      mbar_init(&s.p_full[i], softmax_warps);
      mbar_init(&s.o_full[i], 1);
      mbar_init(&s.drain[i], 1);
      for (int k = 0; k < Smem::kStages; ++k) {
        mbar_init(&s.kv_full[i][k], 1);
        mbar_init(&s.kv_empty[i][k], 1);
      }
    }
    fence_mbar_init();
    if ((smem_u32(smem_raw) & 1023u) != 0u) raise_abort(ctx, kStatusSmemMisaligned);
    prefetch_tensormap(&p.tm_q);
    prefetch_tensormap(&p.tm_k);
    prefetch_tensormap(&p.tm_v);
  }
  if (warp == 8) {
    tmem_alloc(&s.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(s.tmem_base);
  const bool run = (s.abort_flag == 0);
  grid_launch_dependents();
  grid_wait();

  // pipelines 0 of all CTAs come first, so a list shorter than 2 * gridDim.x runs is spread over all SMs
  const int i = warp < 8 ? warp >> 2 : (warp & 1);
  const int w = static_cast<int>(blockIdx.x) + i * static_cast<int>(gridDim.x);
  // 384 threads start with 168 registers; the softmax warps hold a row of 128 scores
  static_assert(8 * 32 * 200 + 4 * 32 * 96 <= kSplitThreads * 168, "setmaxnreg budget does not balance");
  if (warp < 8) {
    reg_inc<200>();
    const int first_warp = fa_split_row0<RC>(i) / 32;
    if (run && w < p.plan.pipes && (warp & 3) >= first_warp && (warp & 3) < first_warp + softmax_warps)
      fa_split_softmax<T, D, RC, NH>(p, s, ctx, tmem, i, w);
  } else {
    reg_dec<96>();
    if (run && w < p.plan.pipes && warp < 10) {
      fa_split_mma_role<T, D, RC>(p, s, ctx, tmem, i, w);
      __syncwarp();
      if (s.abort_flag && lane == 0) {
        umma_commit(&s.drain[i]);  // aborting: let the tensor pipe drain before TMEM is released
        mbar_wait(&s.drain[i], 0, ctx, kRoleSplitDrain);
      }
    } else if (run && w < p.plan.pipes && lane == 0) {
      fa_split_tma_role<T, D, RC>(p, s, ctx, i, w);
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Merges the partial segments of an item: one block per (candidate, row), its warps deal the segments out, a lane has D / 32
// columns; weights exp2(lse - max lse).  Items that one pipeline covered are already written.  It is bound by the latency of
// its loads: the block has a warp per four segments (one item over 256 runs: 21.5 us a call with 4 warps, 15.3 with 16).  With
// fewer runs than items the candidates are the boundaries between runs: one block per (item, row) was 155648 blocks for 295 items
// in parts (B38 Hq256 Hkv32, 16 rows, 4096 keys: 564 -> 457 us).  The two forms are two kernels: as one it took 40 registers
// instead of 32, and three blocks of 16 warps on an SM instead of four (B4 H1, 128 rows, 13208 keys: 24.2 -> 27.7 us).
constexpr int kCombineMaxWarps = 16;
template <typename T, int D, bool kBoundaries>
__global__ void __launch_bounds__(kCombineMaxWarps * 32) fa_split_combine_kernel(const __grid_constant__ FaSplitParams p) {
  grid_launch_dependents();
  grid_wait();
  const int candidate = blockIdx.x / p.plan.rows, row = blockIdx.x - candidate * p.plan.rows;
  const int item = kBoundaries ? fa_split_candidate(p.plan, candidate) : candidate;
  if (kBoundaries && item < 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  int w0, w1;
  fa_split_pipes_of(p.plan, item, w0, w1);
  FaSegment g;
  fa_split_item(p, item, g);
  const int head = row / p.Sq, pos = row - head * p.Sq;
  if (w0 == w1 || head >= g.heads) return;
  // only the first pipeline's part can be its second segment
  const int first_slot = fa_split_slot(p.plan, w0, item);
  auto slot_of = [&](int w) -> long long { return w == w0 ? first_slot : 2 * w; };

  float mx = -INFINITY;
  for (int w = w0 + lane; w <= w1; w += 32) mx = fmaxf(mx, p.part_lse[slot_of(w) * p.plan.rows + row]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (mx == -INFINITY) mx = 0.f;  // no visible key at all: every weight is 0

  constexpr int kCols = D / 32;
  float acc[kCols] = {}, sum = 0.f;
#pragma unroll 4
  for (int w = w0 + warp; w <= w1; w += warps) {
    const long long r = slot_of(w) * p.plan.rows + row;
    const float wt = fast_exp2(p.part_lse[r] - mx);
    const float* src = p.part_o + r * D + lane * kCols;
    sum += wt;
    if constexpr (kCols == 4) {
      const float4 x = *reinterpret_cast<const float4*>(src);
      acc[0] += wt * x.x;
      acc[1] += wt * x.y;
      acc[2] += wt * x.z;
      acc[3] += wt * x.w;
    } else {
      const float2 x = *reinterpret_cast<const float2*>(src);
      acc[0] += wt * x.x;
      acc[1] += wt * x.y;
    }
  }
  __shared__ float s_acc[kCombineMaxWarps][D], s_sum[kCombineMaxWarps];
#pragma unroll
  for (int e = 0; e < kCols; ++e) s_acc[warp][lane * kCols + e] = acc[e];
  if (lane == 0) s_sum[warp] = sum;
  __syncthreads();
  if (warp != 0) return;
  sum = 0.f;
  for (int k = 0; k < warps; ++k) sum += s_sum[k];
  const float inv = sum > 0.f ? 1.0f / sum : 0.f;
  uint32_t packed[kCols / 2];
#pragma unroll
  for (int e = 0; e < kCols; e += 2) {
    float a = 0.f, b = 0.f;
    for (int k = 0; k < warps; ++k) {
      a += s_acc[k][lane * kCols + e];
      b += s_acc[k][lane * kCols + e + 1];
    }
    packed[e / 2] = Pack2<T>::pack(a * inv, b * inv);
  }
  T* dst = static_cast<T*>(p.o) + g.b * p.o_sb + (g.hq0 + head) * p.o_sh + static_cast<long long>(pos) * p.o_ss + lane * kCols;
  if constexpr (kCols == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
  else *reinterpret_cast<uint32_t*>(dst) = packed[0];
  if (lane == 0 && p.lse != nullptr)
    p.lse[(static_cast<long long>(g.b) * p.Hq + g.hq0 + head) * p.Sq + pos] =
        (sum > 0.f ? mx + fast_log2(sum) : -INFINITY) * 0.6931471805599453f;
}

}  // namespace hb
