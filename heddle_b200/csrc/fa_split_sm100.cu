// Launch of the split-key attention kernel (fa_split_sm100.cuh): the rule that takes a call there, the workspace it needs and
// the two launches.
#include "fa_split_sm100.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>

#include "fa_split.h"
#include "host_common.h"

namespace hb {

static FaSplitPlan fa_split_plan(const hb_fa_args* a, int sm_count) {
  return fa_split_plan(a->B, a->Hq, a->Hkv, a->Sq, a->Skv, sm_count);
}

bool fa_split_takes(const hb_fa_args* a, int sm_count) {
  // The query rows of at least one head fit one 128-row tile.  Longer prompts fill the general kernel's 256-row blocks.
  if ((a->dtype != HB_BF16 && a->dtype != HB_FP16) || a->Sq <= 0 || a->Sq > kTileM) return false;
  return !fa_split_general_wins(fa_split_plan(a, sm_count), a->D, sm_count);
}

uint64_t fa_split_workspace(const hb_fa_args* a, int sm_count) {
  const FaSplitPlan pl = fa_split_plan(a, sm_count);
  return pl.cuts ? 2ull * pl.pipes * pl.rows * (a->D + 1) * sizeof(float) : 0;
}

static std::mutex g_split_mutex;

template <typename T, int D, int RC, int NH>
static int launch_split(const FaSplitParams& p, int grid, bool combine, int smem_optin, cudaStream_t stream) {
  using Smem = FaSplitSmem<T, D, RC>;
  if ((int)sizeof(Smem) > smem_optin)
    return set_error(HB_ERR_UNSUPPORTED, "hb_fa_fwd_ws: kernel needs %d bytes of shared memory, device offers %d",
                     (int)sizeof(Smem), smem_optin);
  auto kernel = fa_split_kernel<T, D, RC, NH>;
  static bool configured[64] = {};
  int dev = 0;
  HB_CUDA_CHECK(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(g_split_mutex);
    if (!configured[dev & 63]) {
      HB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem)));
      configured[dev & 63] = true;
    }
  }
  HB_CUDA_CHECK(launch_dependent(kernel, grid, kSplitThreads, sizeof(Smem), stream, 0, p));
  if (combine) {
    const FaSplitPlan& pl = p.plan;
    const long long segments = ((long long)pl.pipes + pl.items - 1) / pl.items + 1;  // of one item, at most
    const unsigned warps = (unsigned)std::min<long long>(kCombineMaxWarps, (segments + 3) / 4);
    auto merge = pl.pipes <= pl.items ? fa_split_combine_kernel<T, D, true> : fa_split_combine_kernel<T, D, false>;
    HB_CUDA_CHECK(launch_dependent(merge, (unsigned)(fa_split_candidates(pl) * pl.rows), 32 * warps, 0, stream, 0, p));
  }
  return HB_OK;
}

template <typename T, int D>
static int launch_split_rows(const FaSplitParams& p, int grid, bool combine, int smem_optin, cudaStream_t stream) {
  if (p.plan.rows <= 8) return launch_split<T, D, 64, 1>(p, grid, combine, smem_optin, stream);
  if (p.plan.rows <= 16) return launch_split<T, D, 64, 2>(p, grid, combine, smem_optin, stream);
  if (p.plan.rows <= 64) return launch_split<T, D, 64, 0>(p, grid, combine, smem_optin, stream);
  return launch_split<T, D, 128, 0>(p, grid, combine, smem_optin, stream);
}
template <typename T>
static int launch_split_d(const FaSplitParams& p, int D, int grid, bool combine, int smem_optin, cudaStream_t stream) {
  return D == 128 ? launch_split_rows<T, 128>(p, grid, combine, smem_optin, stream) : launch_split_rows<T, 64>(p, grid, combine, smem_optin, stream);
}

int fa_split_run(const hb_fa_args* a, const DeviceState* st, void* workspace, uint64_t workspace_bytes) {
  const FaSplitPlan pl = fa_split_plan(a, st->sm_count);
  const bool cuts = pl.cuts != 0;
  const uint64_t need = fa_split_workspace(a, st->sm_count);
  if (cuts && (workspace == nullptr || workspace_bytes < need))
    return set_error(HB_ERR_BAD_ARG, "hb_fa_fwd_ws: needs a workspace of %llu bytes, got %llu", (unsigned long long)need,
                     (unsigned long long)(workspace == nullptr ? 0 : workspace_bytes));
  if (cuts && (reinterpret_cast<uintptr_t>(workspace) & 15u) != 0)
    return set_error(HB_ERR_ALIGN, "hb_fa_fwd_ws: the workspace must be 16-byte aligned");
  FaSplitParams p;
  memset(&p, 0, sizeof(p));
  const CUtensorMapDataType dt = a->dtype == HB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  {
    const uint32_t box[4] = {64, (uint32_t)a->Sq, (uint32_t)pl.hb, 1};
    const uint64_t dims[4] = {(uint64_t)a->D, (uint64_t)a->Sq, (uint64_t)a->Hq, (uint64_t)a->B};
    const uint64_t str[3] = {(uint64_t)a->q_stride_s * 2, (uint64_t)a->q_stride_h * 2, (uint64_t)a->q_stride_b * 2};
    const int rc = encode_tensor_map(&p.tm_q, dt, 4, a->q, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != HB_OK) return rc;
  }
  const uint32_t box[4] = {64, (uint32_t)kTileN, 1, 1};
  const uint64_t dims[4] = {(uint64_t)a->D, (uint64_t)a->Skv, (uint64_t)a->Hkv, (uint64_t)a->B};
  {
    const uint64_t str[3] = {(uint64_t)a->k_stride_s * 2, (uint64_t)a->k_stride_h * 2, (uint64_t)a->k_stride_b * 2};
    const int rc = encode_tensor_map(&p.tm_k, dt, 4, a->k, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != HB_OK) return rc;
  }
  {
    const uint64_t str[3] = {(uint64_t)a->v_stride_s * 2, (uint64_t)a->v_stride_h * 2, (uint64_t)a->v_stride_b * 2};
    const int rc = encode_tensor_map(&p.tm_v, dt, 4, a->v, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != HB_OK) return rc;
  }
  p.o = a->o;
  p.lse = a->lse;
  p.part_o = static_cast<float*>(workspace);
  p.part_lse = cuts ? p.part_o + 2ll * pl.pipes * pl.rows * a->D : nullptr;
  p.status = st->status_word;
  p.o_sb = a->o_stride_b;
  p.o_sh = a->o_stride_h;
  p.o_ss = a->o_stride_s;
  p.B = a->B;
  p.Hq = a->Hq;
  p.Hkv = a->Hkv;
  p.Sq = a->Sq;
  p.Skv = a->Skv;
  p.group = a->Hq / a->Hkv;
  p.causal = a->causal ? 1 : 0;
  p.plan = pl;
  const float scale = a->softmax_scale > 0.f ? a->softmax_scale : 1.0f / sqrtf((float)a->D);
  p.scale_log2 = scale * 1.4426950408889634f;
  const int grid = std::min(pl.pipes, st->sm_count);
  cudaStream_t stream = static_cast<cudaStream_t>(a->stream);
  return a->dtype == HB_BF16 ? launch_split_d<__nv_bfloat16>(p, a->D, grid, cuts, st->smem_optin, stream)
                             : launch_split_d<__half>(p, a->D, grid, cuts, st->smem_optin, stream);
}

}  // namespace hb
