// hb_gemm_epilogue / hb_rms_rowstat: validation, TMA descriptors and launch.
#include "gemm_split_plan.h"
#include "gemm_split_sm100.cuh"
#include "host_common.h"

#include <algorithm>
#include <cstdlib>
#include <mutex>

namespace hb {

template <typename T, int EPI>
static int launch_gemm(const GemmParams& p, int grid, const DeviceState* st, cudaStream_t stream) {
  if ((int)sizeof(GemmSmem) > st->smem_optin)
    return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: kernel needs %d bytes of shared memory, device offers %d",
                     (int)sizeof(GemmSmem), st->smem_optin);
  auto kernel = gemm_kernel<T, EPI>;
  static bool configured[64] = {};
  if (!configured[st->device & 63]) {
    HB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GemmSmem)));
    configured[st->device & 63] = true;
  }
  HB_CUDA_CHECK(launch_dependent(kernel, grid, kGemmThreads, sizeof(GemmSmem), stream, 0, p));
  return HB_OK;
}

template <typename T, int EPI, bool Residual>
static int launch_gemm_pair(const GemmPairParams<Residual>& p, int grid, const DeviceState* st, cudaStream_t stream) {
  if (kPairSmemBytes > st->smem_optin)
    return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: kernel needs %d bytes of shared memory, device offers %d",
                     kPairSmemBytes, st->smem_optin);
  auto kernel = gemm_pair_kernel<T, EPI, Residual>;
  static bool configured[64] = {};
  if (!configured[st->device & 63]) {
    HB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemBytes));
    configured[st->device & 63] = true;
  }
  HB_CUDA_CHECK(launch_dependent(kernel, grid, kGemmThreads, kPairSmemBytes, stream, 0, p));  // clusters of two (compile-time)
  return HB_OK;
}

template <typename T>
static int dispatch_gemm_pair(int epi_class, const GemmParams& base, const CUtensorMap* residual, int grid, const DeviceState* st,
                              cudaStream_t stream) {
  if (residual != nullptr) {
    GemmPairParams<true> p;
    static_cast<GemmParams&>(p) = base;
    p.tm_res = *residual;
    return launch_gemm_pair<T, kEpiPlain, true>(p, grid, st, stream);
  }
  GemmPairParams<false> p;
  static_cast<GemmParams&>(p) = base;
  switch (epi_class) {
    case kEpiPlain:
      return launch_gemm_pair<T, kEpiPlain, false>(p, grid, st, stream);
    case kEpiSwiglu:
      return launch_gemm_pair<T, kEpiSwiglu, false>(p, grid, st, stream);
    default:
      return launch_gemm_pair<T, kEpiRope, false>(p, grid, st, stream);
  }
}

template <typename T>
static int dispatch_gemm(int epi_class, const GemmParams& p, int grid, const DeviceState* st, cudaStream_t stream) {
  switch (epi_class) {
    case kEpiPlain:
      return launch_gemm<T, kEpiPlain>(p, grid, st, stream);
    case kEpiSwiglu:
      return launch_gemm<T, kEpiSwiglu>(p, grid, st, stream);
    default:
      return launch_gemm<T, kEpiRope>(p, grid, st, stream);
  }
}

// ---- the split-K kernel (gemm_split_plan.h: whether it is the one to run) ----

// CTAs of gemm_split_kernel that run at one time in clusters of 1 .. kMaxSplits, per device (the GPCs of the part do not hold a
// whole number of clusters of every size).  Asked for once; the entries do not change after that.
static const int* gemm_split_slots(const DeviceState* st) {
  static int slots[64][kMaxSplits + 1] = {};
  static std::mutex mutex;
  std::lock_guard<std::mutex> lock(mutex);
  int* const table = slots[st->device & 63];
  for (int splits = 1; splits <= kMaxSplits && table[kMaxSplits] == 0; ++splits) {
    auto kernel = gemm_split_kernel<__nv_bfloat16, kEpiPlain, false>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(splits * st->sm_count));
    cfg.blockDim = dim3(kGemmSplitThreads);
    cfg.dynamicSmemBytes = kGemmSplitSmemBytes;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)splits;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSplitSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters <= 0) {
      (void)cudaGetLastError();
      clusters = st->sm_count / (2 * splits) > 0 ? st->sm_count / (2 * splits) : 1;
    }
    table[splits] = clusters * splits;
  }
  return table;
}

template <typename T, int EPI, bool Tail>
static int launch_gemm_split(const GemmSplitArgs<Tail>& p, int grid, const DeviceState* st, cudaStream_t stream) {
  if (kGemmSplitSmemBytes > st->smem_optin)
    return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: kernel needs %d bytes of shared memory, device offers %d",
                     kGemmSplitSmemBytes, st->smem_optin);
  auto kernel = gemm_split_kernel<T, EPI, Tail>;
  static bool configured[64] = {};
  if (!configured[st->device & 63]) {
    HB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSplitSmemBytes));
    configured[st->device & 63] = true;
  }
  HB_CUDA_CHECK(launch_dependent(kernel, grid, kGemmSplitThreads, kGemmSplitSmemBytes, stream, (unsigned)p.splits, p));
  return HB_OK;
}

template <typename T, bool Tail>
static int dispatch_gemm_split(int epi_class, const GemmSplitArgs<Tail>& p, int grid, const DeviceState* st, cudaStream_t stream) {
  switch (epi_class) {
    case kEpiPlain:
      return launch_gemm_split<T, kEpiPlain, Tail>(p, grid, st, stream);
    case kEpiSwiglu:
      return launch_gemm_split<T, kEpiSwiglu, Tail>(p, grid, st, stream);
    default:
      return launch_gemm_split<T, kEpiRope, Tail>(p, grid, st, stream);
  }
}

static bool aligned16(const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; }

static int gemm_impl(const hb_gemm_args* args) {
  if (args == nullptr) return set_error(HB_ERR_BAD_ARG, "hb_gemm_epilogue: args is NULL");
  hb_gemm_args copy = *args;
  const hb_gemm_args* const a = &copy;
  const bool rope16 = copy.epilogue == HB_EPI_ROPE && (copy.dtype & HB_GEMM_ROPE_TABLES_16) != 0;
  if (rope16) copy.dtype &= ~HB_GEMM_ROPE_TABLES_16;
  if (a->M < 0 || a->N <= 0 || a->K <= 0)
    return set_error(HB_ERR_BAD_ARG, "hb_gemm_epilogue: bad extents M=%d N=%d K=%d", a->M, a->N, a->K);
  if (a->dtype != HB_BF16 && a->dtype != HB_FP16)
    return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: dtype %d not supported (bf16, fp16)", a->dtype);
  if (a->epilogue < HB_EPI_NONE || a->epilogue > HB_EPI_ROPE)
    return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: unknown epilogue %d", a->epilogue);
  int n_out = a->N;
  int epi_class = kEpiPlain;
  if (a->epilogue == HB_EPI_SWIGLU) {
    if (a->N % 2 != 0) return set_error(HB_ERR_BAD_ARG, "hb_gemm_epilogue: SWIGLU needs an even N (stacked [Wg; Wu])");
    n_out = a->N / 2;
    epi_class = kEpiSwiglu;
  } else if (a->epilogue == HB_EPI_ROPE) {
    epi_class = kEpiRope;
    if (a->head_dim != 64 && a->head_dim != 128 && a->head_dim != 256)
      return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: ROPE head_dim %d not supported (64, 128, 256)", a->head_dim);
    if (a->N % a->head_dim != 0 || a->rope_cols % a->head_dim != 0 || a->rope_cols < 0 || a->rope_cols > a->N)
      return set_error(HB_ERR_BAD_ARG, "hb_gemm_epilogue: ROPE needs head_dim | N and head_dim | rope_cols <= N");
    if (a->rope_cos == nullptr || a->rope_sin == nullptr || a->rope_seq <= 0)
      return set_error(HB_ERR_BAD_ARG, "hb_gemm_epilogue: ROPE needs cos/sin tables and rope_seq > 0");
    if ((reinterpret_cast<uintptr_t>(a->rope_cos) & 15) != 0 || (reinterpret_cast<uintptr_t>(a->rope_sin) & 15) != 0)
      return set_error(HB_ERR_ALIGN, "hb_gemm_epilogue: ROPE tables need 16-byte alignment");
  }
  if (a->schedule < HB_GEMM_AUTO || a->schedule > HB_GEMM_SPLIT)
    return set_error(HB_ERR_BAD_ARG, "hb_gemm_epilogue: unknown schedule %d", a->schedule);
  const int batch = a->batch > 0 ? a->batch : 1;
  const bool w_kn = a->w_layout == HB_W_KN;
  if (a->w_layout != HB_W_NK && a->w_layout != HB_W_KN)
    return set_error(HB_ERR_BAD_ARG, "hb_gemm_epilogue: unknown w_layout %d", a->w_layout);
  if (w_kn && epi_class != kEpiPlain)
    return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: SWIGLU / ROPE need the weight in [N, K] layout");
  if (batch > 1 && epi_class == kEpiRope)
    return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: ROPE is not defined for batched products");
  if (a->M == 0) return HB_OK;
  if (a->a == nullptr || a->w == nullptr || a->out == nullptr)
    return set_error(HB_ERR_BAD_ARG, "hb_gemm_epilogue: a, w and out must be non-NULL");
  if ((a->K % 8) || (n_out % 8) || (a->lda % 8) || (a->ldw % 8) || (a->ldo % 8) ||
      (a->residual != nullptr && (a->ldr % 8)))
    return set_error(HB_ERR_ALIGN, "hb_gemm_epilogue: K, N_out and the leading dimensions must be multiples of 8");
  if (a->lda < a->K || a->ldw < (w_kn ? a->N : a->K) || a->ldo < n_out || (a->residual != nullptr && a->ldr < n_out))
    return set_error(HB_ERR_BAD_ARG, "hb_gemm_epilogue: a leading dimension is smaller than its row");
  const long long w_rows = w_kn ? a->K : a->N;
  // batch strides (elements); 0 selects densely packed batches
  const long long a_bs = a->a_batch_stride ? a->a_batch_stride : (long long)a->M * a->lda;
  const long long w_bs = a->w_batch_stride ? a->w_batch_stride : w_rows * a->ldw;
  const long long o_bs = a->o_batch_stride ? a->o_batch_stride : (long long)a->M * a->ldo;
  const long long r_bs = a->r_batch_stride ? a->r_batch_stride : (long long)a->M * a->ldr;
  if (batch > 1 && ((a_bs % 8) || (w_bs % 8) || (o_bs % 8) || (a->residual != nullptr && (r_bs % 8))))
    return set_error(HB_ERR_ALIGN, "hb_gemm_epilogue: batch strides must be multiples of 8 elements");
  if (!aligned16(a->a) || !aligned16(a->w) || !aligned16(a->out) || !aligned16(a->residual) || !aligned16(a->bias))
    return set_error(HB_ERR_ALIGN, "hb_gemm_epilogue: pointers must be 16-byte aligned");

  DeviceState* st = nullptr;
  int rc = get_device_state(&st);
  if (rc != HB_OK) return rc;

  // Which kernel.  The persistent kernels win once their 256-column tiles fill the chip; below that the split-K kernel runs where
  // its estimate is the smaller one (gemm_split_plan.h).
  const int k_steps = (a->K + kGemmBK - 1) / kGemmBK;
  const GemmWide wide = gemm_wide(st->sm_count, a->M, a->N, batch);
  GemmSplitChoice split;
  if (a->schedule == HB_GEMM_SPLIT || (a->schedule == HB_GEMM_AUTO && gemm_split_eligible(wide))) {
    split = gemm_split_choose(gemm_split_slots(st), st->sm_count, epi_class, a->M, n_out, k_steps, a->K % kGemmBK == 0, batch, a->head_dim, w_kn);
    const bool plain = epi_class == kEpiPlain && a->epilogue == HB_EPI_NONE;
    const double bytes = 2.0 * batch * ((double)a->M * a->K + (double)a->N * a->K + (double)a->M * n_out);
    if (a->schedule == HB_GEMM_AUTO && !gemm_split_wins(split, wide, k_steps, plain, bytes)) split = GemmSplitChoice();
  }
  const bool use_split = split.width > 0;

  GemmSplitArgs<true> sp;
  memset(&sp, 0, sizeof(sp));
  GemmParams& p = sp.g;
  const CUtensorMapDataType dt = a->dtype == HB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  bool split_tail = false;
  if (use_split) {
    sp.a_rows = a->M > kGemmBM ? kGemmBM : (a->M + 7) / 8 * 8;
    sp.slabs = split.slabs;
    const bool tail = a->K % kGemmBK != 0;
    sp.k_slabs = tail && sp.slabs == 1 ? 0 : 1;  // stages of one slab need no tail of their own: the plain map fills up
    // `whole`: slabs of 64 along a third dimension; else K as it is
    auto a_map = [&](CUtensorMap* tm, bool whole) {
      const uint32_t box[4] = {(uint32_t)kGemmBK, (uint32_t)sp.a_rows, whole ? (uint32_t)sp.slabs : 1u, 1};
      const uint64_t dims[4] = {whole ? (uint64_t)kGemmBK : (uint64_t)a->K, (uint64_t)a->M, whole ? (uint64_t)(a->K / kGemmBK) : 1, (uint64_t)batch};
      const uint64_t str[3] = {(uint64_t)a->lda * 2, kGemmBK * 2, (uint64_t)a_bs * 2};
      return encode_tensor_map(tm, dt, 4, a->a, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    };
    auto w_map = [&](CUtensorMap* tm, bool whole) {
      const uint32_t parts = epi_class == kEpiSwiglu ? 2 : 1;
      const uint32_t box[5] = {(uint32_t)kGemmBK, (uint32_t)split.width / parts, parts, whole ? (uint32_t)sp.slabs : 1u, 1};
      const uint64_t dims[5] = {whole ? (uint64_t)kGemmBK : (uint64_t)a->K, (uint64_t)n_out, parts, whole ? (uint64_t)(a->K / kGemmBK) : 1, (uint64_t)batch};
      const uint64_t str[4] = {(uint64_t)a->ldw * 2, (uint64_t)n_out * a->ldw * 2, kGemmBK * 2, (uint64_t)w_bs * 2};
      return encode_tensor_map(tm, dt, 5, a->w, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B);  // 35.2 -> 33.5 us for 24 x 22016 x 4096
    };
    rc = a_map(&p.tm_a, sp.k_slabs != 0);
    if (rc != HB_OK) return rc;
    if (w_kn) {
      const uint32_t box[3] = {64, (uint32_t)(sp.slabs * kGemmBK), 1};
      const uint64_t dims[3] = {(uint64_t)a->N, (uint64_t)a->K, (uint64_t)batch};
      const uint64_t str[2] = {(uint64_t)a->ldw * 2, (uint64_t)w_bs * 2};
      rc = encode_tensor_map(&p.tm_w, dt, 3, a->w, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    } else {
      rc = w_map(&p.tm_w, sp.k_slabs != 0);
    }
    if (rc != HB_OK) return rc;
    const GemmSplitStages stages = gemm_split_stages(sp.a_rows, split.width, k_steps, !tail);
    p.k_steps = stages.stages;
    split_tail = tail && sp.k_slabs;
    if (split_tail) {
      sp.tail_stage = stages.stages - 1;
      sp.last_slabs = a->K / kGemmBK - (sp.tail_stage - 1) * sp.slabs;
      rc = a_map(&sp.tm_a_tail, false);
      if (rc == HB_OK && !w_kn) rc = w_map(&sp.tm_w_tail, false);
    }
    if (rc != HB_OK) return rc;
  } else {
    const uint32_t box[3] = {(uint32_t)kGemmBK, 128, 1};
    const uint64_t dims[3] = {(uint64_t)a->K, (uint64_t)a->M, (uint64_t)batch};
    const uint64_t str[2] = {(uint64_t)a->lda * 2, (uint64_t)a_bs * 2};
    rc = encode_tensor_map(&p.tm_a, dt, 3, a->a, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != HB_OK) return rc;
  }
  if (use_split) {
    // maps are in place
  } else if (w_kn) {
    const uint32_t box[3] = {64, (uint32_t)kGemmBK, 1};  // 64 columns (128 bytes) x 64 k-rows
    const uint64_t dims[3] = {(uint64_t)a->N, (uint64_t)a->K, (uint64_t)batch};
    const uint64_t str[2] = {(uint64_t)a->ldw * 2, (uint64_t)w_bs * 2};
    rc = encode_tensor_map(&p.tm_w, dt, 3, a->w, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != HB_OK) return rc;
  } else {
    const uint32_t box[3] = {(uint32_t)kGemmBK, 128, 1};
    const uint64_t dims[3] = {(uint64_t)a->K, (uint64_t)a->N, (uint64_t)batch};
    const uint64_t str[2] = {(uint64_t)a->ldw * 2, (uint64_t)w_bs * 2};
    rc = encode_tensor_map(&p.tm_w, dt, 3, a->w, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != HB_OK) return rc;
  }
  const bool pair = !use_split &&
                    (a->schedule == HB_GEMM_PAIR || (a->schedule == HB_GEMM_AUTO && a->M > kGemmBM && st->sm_count >= 2));
  // A tensor map has strides of 16 bytes to 2^40, forward only: a residual with others (its batches may lie in any order) is read by threads.
  const bool res_strides = a->ldr < (1ll << 39) && (batch == 1 || (r_bs > 0 && r_bs < (1ll << 39)));
  const bool res_tma = pair && epi_class == kEpiPlain && a->residual != nullptr && res_strides;
  CUtensorMap tm_res;
  if (epi_class == kEpiPlain && !use_split) {
    const uint32_t box[3] = {64, (uint32_t)kGemmBM, 1};
    const uint64_t dims[3] = {(uint64_t)n_out, (uint64_t)a->M, (uint64_t)batch};
    const uint64_t str[2] = {(uint64_t)a->ldo * 2, (uint64_t)o_bs * 2};
    rc = encode_tensor_map(&p.tm_out, dt, 3, a->out, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != HB_OK) return rc;
    p.tma_store = 1;
    if (res_tma) {
      const uint64_t res_str[2] = {(uint64_t)a->ldr * 2, (uint64_t)(batch == 1 ? a->ldr : r_bs) * 2};  // one batch: any
      rc = encode_tensor_map(&tm_res, dt, 3, a->residual, dims, res_str, box, CU_TENSOR_MAP_SWIZZLE_128B);
      if (rc != HB_OK) return rc;
    }
  }
  p.out = a->out;
  p.row_scale = a->row_scale;
  p.residual = a->residual;
  p.bias = a->bias;
  p.rope_cos = a->rope_cos;
  p.rope_sin = a->rope_sin;
  p.rope16 = rope16 ? 1 : 0;
  p.status = st->status_word;
  p.ldo = a->ldo;
  p.ldr = a->ldr;
  p.M = a->M;
  p.N_out = n_out;
  p.K = a->K;
  p.tile_cols = (use_split ? split.width : kGemmBN) / (epi_class == kEpiSwiglu ? 2 : 1);
  const int tile_rows = pair ? kPairBM : kGemmBM;
  p.tiles_m = (a->M + tile_rows - 1) / tile_rows;
  p.tiles_n = (n_out + p.tile_cols - 1) / p.tile_cols;
  p.tiles_per_batch = p.tiles_m * p.tiles_n;
  const long long tiles = (long long)p.tiles_m * p.tiles_n * batch;
  if (tiles > 0x7fffffffLL || (long long)batch * a->M > 0x7fffffffLL)
    return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: too many tiles");
  p.num_tiles = (int)tiles;
  p.batch = batch;
  const int last_rows = p.tiles_m - (p.tiles_m - 1) / kGemmGroupM * kGemmGroupM;
  p.div_batch = make_fast_div((uint32_t)p.tiles_per_batch);
  p.div_group = make_fast_div((uint32_t)((long long)kGemmGroupM * p.tiles_n));
  p.div_rows = make_fast_div(kGemmGroupM);
  p.div_last = make_fast_div((uint32_t)last_rows);
  p.w_kn = w_kn ? 1 : 0;
  p.o_batch_stride = o_bs;
  p.r_batch_stride = r_bs;
  if (!use_split) p.k_steps = k_steps;
  p.act = (a->epilogue >= HB_EPI_SILU && a->epilogue <= HB_EPI_TANH) ? a->epilogue : kActNone;
  p.rope_seq = a->rope_seq;
  p.head_dim = a->head_dim;
  p.rope_cols = a->rope_cols;
  p.w_row2_offset = n_out;
  // shared-memory split of the pair kernel: the deepest ring, except for a K loop of one or two steps, whose time is the
  // epilogue's: it gives stages to staging slabs.  us with 1 | 2 | 4 slabs, 64 x [2048, K] . [K, 2048]: K = 128 125 | 123 | 114,
  // K = 256 152 | 152 | 176, K = 384 191 | 196 | 229.
  // With a residual, two slabs hold a tile's part of it (GemmPairParams).
  p.out_slabs = res_tma ? 2 : p.k_steps <= 2 ? 4 : 1;
  p.pair_stages = kPairSlots - p.out_slabs;

  const int grid = pair ? 2 * (int)std::min<long long>(tiles, st->sm_count / 2) : (int)std::min<long long>(tiles, st->sm_count);
  cudaStream_t stream = static_cast<cudaStream_t>(a->stream);
  if (use_split) {
    sp.width = split.width;
    sp.splits = split.splits;
    const int stage_bytes = (sp.a_rows + sp.width) * kGemmBK * 2 * sp.slabs;
    // the last A box of the ring is read as 128 rows: 16 KB of shared memory behind its start have to exist
    sp.stages = std::min(kGemmSplitMaxStages, (kGemmSplitRing - 16384) / stage_bytes);
    sp.tmem_cols = 32;
    while (sp.tmem_cols < sp.width) sp.tmem_cols *= 2;
    if (tiles * sp.splits > 0x7fffffffLL) return set_error(HB_ERR_UNSUPPORTED, "hb_gemm_epilogue: too many tiles");
    const int split_grid = (int)tiles * sp.splits;
    if (split_tail)
      return a->dtype == HB_BF16 ? dispatch_gemm_split<__nv_bfloat16, true>(epi_class, sp, split_grid, st, stream)
                                 : dispatch_gemm_split<__half, true>(epi_class, sp, split_grid, st, stream);
    GemmSplitArgs<false> plain;
    static_cast<GemmSplitParams&>(plain) = sp;
    return a->dtype == HB_BF16 ? dispatch_gemm_split<__nv_bfloat16, false>(epi_class, plain, split_grid, st, stream)
                               : dispatch_gemm_split<__half, false>(epi_class, plain, split_grid, st, stream);
  }
  if (pair) {
    const CUtensorMap* const res = res_tma ? &tm_res : nullptr;
    return a->dtype == HB_BF16 ? dispatch_gemm_pair<__nv_bfloat16>(epi_class, p, res, grid, st, stream)
                               : dispatch_gemm_pair<__half>(epi_class, p, res, grid, st, stream);
  }
  return a->dtype == HB_BF16 ? dispatch_gemm<__nv_bfloat16>(epi_class, p, grid, st, stream)
                             : dispatch_gemm<__half>(epi_class, p, grid, st, stream);
}

static int rowstat_impl(const void* x, const void* residual, void* y_out, float* rstd, int M, int N, long long ldx,
                        float eps, int dtype, void* stream) {
  if (M < 0 || N <= 0) return set_error(HB_ERR_BAD_ARG, "hb_rms_rowstat: bad extents M=%d N=%d", M, N);
  if (dtype != HB_BF16 && dtype != HB_FP16) return set_error(HB_ERR_UNSUPPORTED, "hb_rms_rowstat: dtype %d", dtype);
  if (M == 0) return HB_OK;
  if (x == nullptr || rstd == nullptr) return set_error(HB_ERR_BAD_ARG, "hb_rms_rowstat: x and rstd must be non-NULL");
  if ((N % 8) || (ldx % 8) || ldx < N || !aligned16(x) || !aligned16(residual) || !aligned16(y_out))
    return set_error(HB_ERR_ALIGN, "hb_rms_rowstat: N and ldx must be multiples of 8, pointers 16-byte aligned");
  DeviceState* st = nullptr;
  int rc = get_device_state(&st);
  if (rc != HB_OK) return rc;
  const int grid = (M + 7) / 8;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == HB_BF16) {
    HB_CUDA_CHECK(launch_dependent(rms_rowstat_kernel<__nv_bfloat16>, grid, 256, 0, s, 0, static_cast<const __nv_bfloat16*>(x),
                                   static_cast<const __nv_bfloat16*>(residual), static_cast<__nv_bfloat16*>(y_out), rstd, M, N,
                                   ldx, eps));
  } else {
    HB_CUDA_CHECK(launch_dependent(rms_rowstat_kernel<__half>, grid, 256, 0, s, 0, static_cast<const __half*>(x),
                                   static_cast<const __half*>(residual), static_cast<__half*>(y_out), rstd, M, N, ldx, eps));
  }
  return HB_OK;
}

int gemm_smem_bytes() { return (int)sizeof(GemmSmem); }

}  // namespace hb

extern "C" {

int hb_gemm_epilogue(const hb_gemm_args* args) {
  hb::clear_error();
  return hb::gemm_impl(args);
}

int hb_rms_rowstat(const void* x, const void* residual, void* y_out, float* rstd, int32_t M, int32_t N, int64_t ldx,
                   float eps, int32_t dtype, void* stream) {
  hb::clear_error();
  return hb::rowstat_impl(x, residual, y_out, rstd, M, N, ldx, eps, dtype, stream);
}

}  // extern "C"

extern "C" int hb_prepare_weight(const hb_prepare_args* a) {
  using namespace hb;
  if (a == nullptr) return set_error(HB_ERR_BAD_ARG, "hb_prepare_weight: args is NULL");
  if (a->n_src < 1 || a->n_src > 4) return set_error(HB_ERR_BAD_ARG, "hb_prepare_weight: n_src must be 1..4");
  if (a->dtype != HB_BF16 && a->dtype != HB_FP16)
    return set_error(HB_ERR_UNSUPPORTED, "hb_prepare_weight: dtype %d not supported (bf16, fp16)", a->dtype);
  if (a->K <= 0 || a->K % 8 != 0) return set_error(HB_ERR_ALIGN, "hb_prepare_weight: K must be a positive multiple of 8");
  if (a->out == nullptr) return set_error(HB_ERR_BAD_ARG, "hb_prepare_weight: out is NULL");
  if (a->ld_out < a->K || a->ld_out % 8 != 0 || (reinterpret_cast<uintptr_t>(a->out) & 15) != 0)
    return set_error(HB_ERR_ALIGN, "hb_prepare_weight: out needs 16-byte alignment and a row stride that is a multiple of 8");
  if (a->gamma != nullptr && (reinterpret_cast<uintptr_t>(a->gamma) & 15) != 0)
    return set_error(HB_ERR_ALIGN, "hb_prepare_weight: gamma needs 16-byte alignment");
  PrepareParams p;
  memset(&p, 0, sizeof(p));
  long long rows = 0;
  for (int i = 0; i < a->n_src; ++i) {
    if (a->src[i] == nullptr || a->rows[i] <= 0) return set_error(HB_ERR_BAD_ARG, "hb_prepare_weight: source %d is empty", i);
    if (a->ld_src[i] < a->K || a->ld_src[i] % 8 != 0 || (reinterpret_cast<uintptr_t>(a->src[i]) & 15) != 0)
      return set_error(HB_ERR_ALIGN, "hb_prepare_weight: source %d needs 16-byte alignment and a row stride that is a multiple of 8", i);
    rows += a->rows[i];
    if (rows > 0x7fffffffLL) return set_error(HB_ERR_UNSUPPORTED, "hb_prepare_weight: too many rows");
    p.src[i] = a->src[i];
    p.ld_src[i] = a->ld_src[i];
    p.row_end[i] = static_cast<int>(rows);
  }
  for (int i = a->n_src; i < 4; ++i) p.row_end[i] = static_cast<int>(rows);
  p.n_src = a->n_src;
  p.K = a->K;
  p.gamma = a->gamma;
  p.out = a->out;
  p.ld_out = a->ld_out;
  DeviceState* st = nullptr;
  int rc = get_device_state(&st);
  if (rc != HB_OK) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(a->stream);
  const long long total = rows * (a->K / 8);
  const int grid = static_cast<int>(std::min<long long>((total + 255) / 256, 16ll * st->sm_count));
  if (a->dtype == HB_BF16) {
    prepare_weight_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(p);
  } else {
    prepare_weight_kernel<__half><<<grid, 256, 0, stream>>>(p);
  }
  HB_CUDA_CHECK(cudaGetLastError());
  return HB_OK;
}
