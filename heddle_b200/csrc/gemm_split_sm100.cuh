// tcgen05 GEMM for products whose tiles would leave most of the chip idle (decode steps, short prompts), sm_100a.
//
// What bounds such a product is reading the weights once, and how fast an SM can do that: 128 x 256 tiles of a 24-row
// product are 16 to 86 CTAs on 148 SMs.  Here the tile width is free (16 .. 256 columns) and a cluster of up to 8 CTAs splits
// the K range of one tile: every CTA accumulates its part in TMEM, and the CTAs share out the tile's rows: each row's fp32
// parts go to its owner through distributed shared memory, which adds them in a fixed order (the sum does not depend on
// timing) and applies the epilogue.  No workspace, no second launch.  Loads are plain tiled TMA
// loads; only live rows of A are loaded (the box is M rounded up to 8 rows), which leaves the ring to the weights.
//
// A stage holds one or more 64-wide K slabs, brought by ONE tensor copy per operand (the map's third dimension walks the
// slabs): with one slab per stage a narrow tile took 270 ns a step whatever its width, for two copies, two barriers and four
// MMAs, 20.8 us for a single row of 4096 x 4096.
//
// 256 threads: warp 0 TMA producer, warp 1 MMA issuer, then all warps read the accumulator back and run the epilogue.
#pragma once

#include "gemm_sm100.cuh"

namespace hb {

constexpr int kGemmSplitThreads = 256;
constexpr int kGemmSplitMaxStages = 12;
constexpr int kGemmSplitRing = 221 * 1024;  // operand ring; reused for the fp32 partial tile

struct GemmSplitParams {
  GemmParams g;    // tile_cols = output columns of a tile
  int width;       // accumulator columns of a tile (= tile_cols, twice that for SWIGLU)
  int a_rows;      // rows of the A box (multiple of 8, <= 128)
  int slabs;       // 64-wide K slabs per stage; g.k_steps counts stages
  // 1: the maps are A [64, rows, K / 64, batch] and W [64, rows, parts, K / 64, batch], 0: [K, rows, ..., 1, batch].  A SWIGLU
  // weight has two parts, gate and up: one copy brings both.
  int k_slabs;
  int stages;
  int splits;      // cluster size
  int tmem_cols;   // power of two >= width
};

// With `Tail`, what a K that is not a multiple of 64 leaves behind its whole slabs is the last stage, one slab brought by maps of the
// second kind, which fill it up with zeros.  (A kernel of its own: with the choice at run time the others paid 3 to 4 %.)
// us with one slab per stage for such a K -> with the tail apart: 17 x 5344 x 3056 16.8 -> 11.4, 8 x 1392 x 11616 16.4 -> 11.7, 28 x 7120 x
// 5416 26.6 -> 22.4, 1 x 1360 x 5912 10.9 -> 8.7, 2 x 1120 x 1160 7.1 -> 5.8.
template <bool Tail>
struct GemmSplitArgs : GemmSplitParams {};
template <>
struct GemmSplitArgs<true> : GemmSplitParams {
  int tail_stage;
  int last_slabs;  // whole slabs in the stage in front of it
  CUtensorMap tm_a_tail, tm_w_tail;
};

struct GemmSplitCtrl {
  uint64_t full[kGemmSplitMaxStages], empty[kGemmSplitMaxStages];
  uint64_t acc_full, drain;
  uint32_t tmem_base;
  uint32_t abort_flag;
};
constexpr int kGemmSplitSmemBytes = kGemmSplitRing + static_cast<int>(sizeof(GemmSplitCtrl));

// 16 bytes to the shared memory of a CTA of the cluster (shared::cluster address)
__device__ __forceinline__ void st_cluster_16(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Eight consecutive accumulator columns of one row, summed over the parts in rank order.
__device__ __forceinline__ void gemm_split_sum8(const uint8_t* part0, uint32_t part_bytes, int splits, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(part0), b = *reinterpret_cast<const float4*>(part0 + 16);
  v[0] = a.x;
  v[1] = a.y;
  v[2] = a.z;
  v[3] = a.w;
  v[4] = b.x;
  v[5] = b.y;
  v[6] = b.z;
  v[7] = b.w;
#pragma unroll 4
  for (int r = 1; r < splits; ++r) {
    const uint8_t* q = part0 + static_cast<uint32_t>(r) * part_bytes;
    const float4 x = *reinterpret_cast<const float4*>(q), y = *reinterpret_cast<const float4*>(q + 16);
    v[0] += x.x;
    v[1] += x.y;
    v[2] += x.z;
    v[3] += x.w;
    v[4] += y.x;
    v[5] += y.y;
    v[6] += y.z;
    v[7] += y.w;
  }
}

template <typename T>
__device__ __forceinline__ void gemm_split_scale_bias8(const GemmParams& p, float rs, int bias_col, float (&v)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] *= rs;
  if (p.bias != nullptr) {
    float b[8];
    load_bias8<T>(p, bias_col, b);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] += b[e];
  }
}

template <typename T, int EPI, bool Tail>
__global__ void __launch_bounds__(kGemmSplitThreads, 1) gemm_split_kernel(const __grid_constant__ GemmSplitArgs<Tail> sp) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const GemmParams& p = sp.g;
  const uint32_t a_slab = static_cast<uint32_t>(sp.a_rows) * 128u, b_slab = static_cast<uint32_t>(sp.width) * 128u;
  const uint32_t a_bytes = a_slab * sp.slabs, b_bytes = b_slab * sp.slabs;
  // The A operand has M = 128 rows: with a shorter box the tensor core also reads what lies behind it (the next stages or
  // the B ring, which is at least 16 KB); those rows only feed accumulator rows nobody reads.
  uint8_t* const ring_a = smem_raw;
  uint8_t* const ring_b = ring_a + sp.stages * a_bytes;
  GemmSplitCtrl& s = *reinterpret_cast<GemmSplitCtrl*>(smem_raw + kGemmSplitRing);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = sp.splits;
  const int rank = static_cast<int>(blockIdx.x) % splits, t = static_cast<int>(blockIdx.x) / splits;
  AbortCtx ctx{&s.abort_flag, p.status};

  int m_t, n_t, b;
  gemm_tile_coords(p, t, m_t, n_t, b);
  const int m0 = m_t * kGemmBM, n0 = n_t * p.tile_cols;
  const int k_begin = p.k_steps * rank / splits, k_end = p.k_steps * (rank + 1) / splits;  // at most 2^25 stages, 8 ranks
  // In front of the wait for the predecessor, where the time is free: a 64-bit division and first reads of the parameters, which miss the
  // constant cache, lay 0.7 us between that and the first copies, 0.3 us now.  us back to back, before -> after: 1 x 4096 x 4096 10.2 ->
  // 9.9, 64 x 1024 x 512 4.4 -> 4.1, 1 x 640 x 720 4.9 -> 4.5, batch of 3 67 x 280 x 1392 6.0 -> 5.5.
  computed(m0, n0, b, k_begin, k_end, a_bytes, b_bytes, p.w_kn, sp.k_slabs);

  if (threadIdx.x == 0) {
    s.abort_flag = 0;
    for (int i = 0; i < sp.stages; ++i) {
      mbar_init(&s.full[i], 1);
      mbar_init(&s.empty[i], 1);
    }
    mbar_init(&s.acc_full, 1);
    mbar_init(&s.drain, 1);
    fence_mbar_init();
    if ((smem_u32(smem_raw) & 1023u) != 0u) raise_abort(ctx, kStatusSmemMisaligned);
    prefetch_tensormap(&p.tm_a);
    prefetch_tensormap(&p.tm_w);
    if constexpr (Tail) {
      prefetch_tensormap(&sp.tm_a_tail);
      if (!p.w_kn) prefetch_tensormap(&sp.tm_w_tail);
    }
  }
  if (warp == 1) {
    tmem_alloc(&s.tmem_base, static_cast<uint32_t>(sp.tmem_cols));
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmem_base;
  const bool run = (s.abort_flag == 0);
  grid_launch_dependents();
  grid_wait();

  if (warp == 0) {
    if (run && lane == 0) {
      uint32_t st = 0, phase = 1;
      for (int ks = k_begin; ks < k_end; ++ks) {
        if (!mbar_wait(&s.empty[st], phase, ctx, kGemmRoleTma)) break;
        uint8_t* const sb = ring_b + st * b_bytes;
        if constexpr (Tail) {
          if (ks == sp.tail_stage) {
            const int k0 = p.K / kGemmBK * kGemmBK;
            mbar_arrive_expect_tx(&s.full[st], a_slab + (p.w_kn ? b_bytes : b_slab));
            if (p.w_kn) {  // rows past K are zeros
              for (int i = 0; i < sp.width / 64; ++i)
                tma_load_3d(sb + i * (sp.slabs * kGemmBK * 128), &p.tm_w, &s.full[st], n0 + i * 64, k0, b);
            } else {
              tma_load_5d(sb, &sp.tm_w_tail, &s.full[st], k0, n0, 0, 0, b);
            }
            tma_load_4d(ring_a + st * a_bytes, &sp.tm_a_tail, &s.full[st], k0, m0, 0, b);
            break;
          }
        }
        mbar_arrive_expect_tx(&s.full[st], a_bytes + b_bytes);
        const int kc = sp.k_slabs ? 0 : ks * kGemmBK, slab = sp.k_slabs ? ks * sp.slabs : 0;
        if (p.w_kn) {
          for (int i = 0; i < sp.width / 64; ++i)
            tma_load_3d(sb + i * (sp.slabs * kGemmBK * 128), &p.tm_w, &s.full[st], n0 + i * 64, ks * sp.slabs * kGemmBK, b);
        } else {
          tma_load_5d(sb, &p.tm_w, &s.full[st], kc, n0, 0, slab, b);
        }
        tma_load_4d(ring_a + st * a_bytes, &p.tm_a, &s.full[st], kc, m0, slab, b);
        if (++st == static_cast<uint32_t>(sp.stages)) {
          st = 0;
          phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (run) {
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // see gemm_kernel
      constexpr uint32_t kLbo = (16u >> 4) << 16;
      const uint32_t idesc = make_idesc(Pack2<T>::kFormat, kGemmBM, static_cast<uint32_t>(sp.width), 0, p.w_kn ? 1u : 0u);
      // [K, N] operand: 64-column groups of slabs * 64 k-rows; [N, K] operand: one slab after the other
      const uint32_t b_lbo = p.w_kn ? (static_cast<uint32_t>(sp.slabs) * kGemmBK * 128u >> 4) << 16 : kLbo;
      const uint32_t b_step = p.w_kn ? (16u * 128u >> 4) : 2u;
      const uint32_t b_next = p.w_kn ? (kGemmBK * 128u >> 4) : b_slab >> 4;
      const bool leader = elect_one();
      uint32_t st = 0, phase = 0;
      bool ok = true;
      for (int ks = k_begin; ks < k_end; ++ks) {
        if (!mbar_wait_warp(&s.full[st], phase, ctx, kGemmRoleMma)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a_lo = (smem_u32(ring_a + st * a_bytes) >> 4) | kLbo, b_lo = (smem_u32(ring_b + st * b_bytes) >> 4) | b_lbo;
        if (leader) {
          auto slabs = [&]() -> int {
            // the last stage of whole slabs may hold fewer: with a [K, N] operand the rest of its box are the tail's rows
            if constexpr (Tail) return ks == sp.tail_stage ? 1 : ks == sp.tail_stage - 1 ? sp.last_slabs : sp.slabs;
            else return sp.slabs;
          };
          for (int sl = 0; sl < slabs(); ++sl) {
            const uint32_t a = a_lo + static_cast<uint32_t>(sl) * (a_slab >> 4), w = b_lo + static_cast<uint32_t>(sl) * b_next;
#pragma unroll
            for (int kk = 0; kk < kGemmBK / 16; ++kk) {
              const uint64_t da = (static_cast<uint64_t>(kDescHi) << 32) | (a + kk * 2);
              const uint32_t acc = (ks > k_begin || sl > 0 || kk > 0) ? 1u : 0u;
              umma_ss_f16(tmem, da, (static_cast<uint64_t>(kDescHi) << 32) | (w + kk * b_step), idesc, acc);
            }
          }
          umma_commit(&s.empty[st]);
        }
        if (++st == static_cast<uint32_t>(sp.stages)) {
          st = 0;
          phase ^= 1;
        }
      }
      if (ok && leader) umma_commit(&s.acc_full);
      __syncwarp();
      if (s.abort_flag && lane == 0) {
        umma_commit(&s.drain);
        mbar_wait(&s.drain, 0, ctx, kGemmRoleDrain);
      }
    }
    __syncwarp();
  }

  // ---- exchange: each CTA of the cluster finishes `own` rows of the tile.  Every thread holds one row of its CTA's part and
  // writes it, as fp32, into the shared memory of the row's owner (remote stores are posted; pulling the parts instead put
  // a round trip in front of every group of columns: 3 us for 120 x 96 over three CTAs, 10 us for 120 x 256 over eight).
  // The parts lie over the rings: the first barrier says that every load of the cluster has landed and every MMA is done.
  // Rows are padded by 16 bytes, so a warp's 16-byte writes (one row per thread) touch all banks evenly. ----
  const int rows = min(kGemmBM, p.M - m0);
  const int own = (rows + splits - 1) / splits;
  const uint32_t pitch = static_cast<uint32_t>(sp.width + 4) * 4u, part_bytes = static_cast<uint32_t>(own) * pitch;
  const bool ok = run && mbar_wait_warp(&s.acc_full, 0, ctx, kGemmRoleEpi);
  __syncwarp();
  if (splits > 1) cluster_sync_relaxed();
  else __syncthreads();
  if (ok) {
    tc_fence_after();
    const int quarter = warp & 3, r_tile = quarter * 32 + lane;
    if (quarter * 32 < rows) {
      const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
      const int owner = r_tile / own;
      const uint32_t local = smem_u32(smem_raw) + static_cast<uint32_t>(rank) * part_bytes + static_cast<uint32_t>(r_tile - owner * own) * pitch;
      const bool live = r_tile < rows;
      const uint32_t dst = live ? mapa_u32(local, static_cast<uint32_t>(owner)) : 0;
      for (int c = (warp >> 2) * 32; c < sp.width; c += 64) {  // the last read may pass the tile's width, never tmem_cols
        uint32_t r[32];
        __syncwarp();
        tmem_ld32(taddr + static_cast<uint32_t>(c), r);
        tmem_wait_ld();
        if (live) {
#pragma unroll
          for (int e = 0; e < 32; e += 4)
            if (c + e < sp.width) st_cluster_16(dst + static_cast<uint32_t>(c + e) * 4u, r[e], r[e + 1], r[e + 2], r[e + 3]);
        }
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  if (splits > 1) cluster_sync_all();  // the parts are in place; nothing remote is touched after this
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, static_cast<uint32_t>(sp.tmem_cols));
  }

  // ---- epilogue: groups of eight output columns of this CTA's rows (consecutive threads take consecutive groups) ----
  if (ok) {
    const int half = p.head_dim >> 1;
    const int groups = (EPI == kEpiRope ? p.tile_cols / 2 : p.tile_cols) / 8;  // per row; ROPE handles both halves of a pair
    const int row_lo = rank * own, total = max(0, min(own, rows - row_lo)) * groups;
    int r = static_cast<int>(threadIdx.x) / groups, g = static_cast<int>(threadIdx.x) - r * groups;
    const int dr = kGemmSplitThreads / groups, dg = kGemmSplitThreads - dr * groups;
    for (int idx = static_cast<int>(threadIdx.x); idx < total; idx += kGemmSplitThreads) {
      const int row = m0 + row_lo + r, r_own = r;
      int c = g * 8;  // column inside the tile
      if constexpr (EPI == kEpiRope) c = c / half * p.head_dim + c % half;
      r += dr;
      g += dg;
      if (g >= groups) {
        g -= groups;
        ++r;
      }
      const int col = n0 + c;
      if (col >= p.N_out) continue;
      const float rs = p.row_scale != nullptr ? p.row_scale[(long long)b * p.M + row] : 1.0f;
      const uint8_t* src = smem_raw + static_cast<uint32_t>(r_own) * pitch + static_cast<uint32_t>(c) * 4u;
      float v[8];
      gemm_split_sum8(src, part_bytes, splits, v);
      gemm_split_scale_bias8<T>(p, rs, col, v);
      if constexpr (EPI == kEpiPlain) {
        with_act(p.act, [&](auto act) { apply_act8<decltype(act)::value>(v); });
      } else if constexpr (EPI == kEpiSwiglu) {
        float u[8];
        gemm_split_sum8(src + static_cast<uint32_t>(p.tile_cols) * 4u, part_bytes, splits, u);
        gemm_split_scale_bias8<T>(p, rs, p.w_row2_offset + col, u);
        apply_act8<kActSilu>(v);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] *= u[e];
      } else {
        float x2[8];
        gemm_split_sum8(src + static_cast<uint32_t>(half) * 4u, part_bytes, splits, x2);
        gemm_split_scale_bias8<T>(p, rs, col + half, x2);
        if (col < p.rope_cols) {
          const long long angles = static_cast<long long>(row % p.rope_seq) * half + c % half;
          float cs[8], sn[8];
          load_angles8<T>(p, p.rope_cos, angles, cs);
          load_angles8<T>(p, p.rope_sin, angles, sn);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float xa = v[e], xb = x2[e];
            v[e] = xa * cs[e] - xb * sn[e];
            x2[e] = xb * cs[e] + xa * sn[e];
          }
        }
        store8<T>(p, b, row, col + half, x2);
      }
      store8<T>(p, b, row, col, v);
    }
  }
}

}  // namespace hb
