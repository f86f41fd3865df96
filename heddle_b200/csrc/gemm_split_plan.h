// Which tile width and cluster size the split-K GEMM takes, and whether it or a persistent kernel runs a product.  Host code
// without CUDA, so that the rule is tested on a CPU.
#pragma once

#include <algorithm>

#include "gemm_shape.h"

namespace hb {

constexpr int kMaxSplits = 8;  // CTAs of a cluster, at most

struct GemmSplitChoice {
  int width = 0, splits = 0, slabs = 0;
  double ns = 0.0;       // what the choice among widths and clusters goes by
  double rule_ns = 0.0;  // what the split-K kernel is compared with a persistent one by
};

// K slabs per stage: about 40 KB, so that four or more stages fit the ring.  A K that is not a multiple of 64 leaves a tail, which is a
// stage of its own behind the whole slabs.
struct GemmSplitStages {
  int slabs, stages;
};
inline GemmSplitStages gemm_split_stages(int a_rows, int width, int k_steps, bool whole_slabs) {
  const int whole = whole_slabs ? k_steps : k_steps - 1;
  const int slabs = std::max(1, std::min({4, whole, 40 * 1024 / ((a_rows + width) * 128)}));
  return {slabs, (whole + slabs - 1) / slabs + (k_steps - whole)};
}

// Estimated time (ns) of one launch, fitted to a sweep of widths 64 .. 256 and clusters 1 .. 8 on 24 .. 256 x 4096 .. 22016 x
// 4096 .. 11008: an SM streams weights from HBM at 60 B/ns and all operands at 120; a 128 x 256 x 64 slab takes 270 ns on the
// tensor cores, and never less than the 125 ns its four MMAs take to issue; HBM gives 6 KB/ns and L2 14 KB/ns in all; a wave
// costs 5 us for its start, its first load and its stores, 450 ns more per CTA of a cluster, and 100 ns per 1000 accumulators
// read back.  `slots[s]`: CTAs that run at one time in clusters of s.
inline GemmSplitChoice gemm_split_choose(const int* slots, int sm_count, int epi_class, int M, int n_out, int k_steps,
                                         bool whole_slabs, int batch, int head_dim, bool w_kn) {
  GemmSplitChoice best;
  const int tiles_m = (M + kGemmBM - 1) / kGemmBM;
  const int a_rows = tiles_m > 1 ? kGemmBM : (M + 7) / 8 * 8;
  const int unit = epi_class == kEpiRope ? head_dim : w_kn ? 64 : 16;
  const int per_col = epi_class == kEpiSwiglu ? 2 : 1;  // accumulator columns per output column
  const double hbm = 128.0 * k_steps * batch * ((double)n_out * per_col + M) / 6000.0;
  for (int width = unit; width <= kGemmBN; width += unit) {
    const long long tiles = (long long)tiles_m * ((n_out * per_col + width - 1) / width) * batch;
    const double slab = std::max({width * 128.0 / 60.0, (width + a_rows) * 128.0 / 120.0, width * (270.0 / 256.0), 125.0});
    const double l2 = 128.0 * (width + a_rows) * tiles * (double)k_steps / 14000.0;
    const auto [slabs, stages] = gemm_split_stages(a_rows, width, k_steps, whole_slabs);
    for (int splits = 1; splits <= std::min(kMaxSplits, stages); ++splits) {
      const double fixed = 5000.0 + (splits > 1 ? 450.0 * splits : 0.0) + std::min(M, kGemmBM) * (double)width / 10.0;
      // no cluster of this size or larger is faster than this; the search is host time of every call with few tiles, 0.9 us
      // without this line and 0.3 to 0.7 with it
      if (best.width != 0 && std::max(hbm, l2) + fixed >= best.ns) break;
      const long long waves = (tiles * splits + slots[splits] - 1) / slots[splits];
      const double stream = slab * slabs * ((stages + splits - 1) / splits);
      // CTAs of later waves start as SMs come free, so most of their fixed time hides under the others' streaming ...
      const double ns = std::max({hbm, l2, waves * stream}) + fixed * (0.7 + 0.3 * waves);
      // ... while that is bound by HBM.  A CTA has its SM to itself, so an SM's own waves come one after the other.
      if (best.width == 0 || ns < best.ns)
        best = {width, splits, slabs, ns, 0.8 * std::max(ns, waves * (1.3 * stream + 0.9 * fixed) + 500.0)};
    }
    if (tiles > 4ll * sm_count && width >= 128) break;  // wider tiles only leave fewer of them
  }
  return best;
}

// The persistent kernel for the same product (CTA pairs on 256 x 256 tiles when there is more than one 128-row tile of rows, else
// single CTAs on 128 x 256): its rounds of tiles, or its bytes.
struct GemmWide {
  bool one_row;
  long long tiles;
  int slots;
};
inline GemmWide gemm_wide(int sm_count, int M, int N, int batch) {
  GemmWide w;
  w.one_row = M <= kGemmBM;
  const int rows = w.one_row ? kGemmBM : kPairBM;
  w.tiles = (long long)((M + rows - 1) / rows) * ((N + kGemmBN - 1) / kGemmBN) * batch;
  w.slots = w.one_row ? sm_count : std::max(1, sm_count / 2);
  return w;
}
// Beyond these rounds the persistent kernel has always been the faster one, and nothing is estimated.
inline bool gemm_split_eligible(const GemmWide& w) { return w.tiles < (w.one_row ? 8ll : 2ll) * w.slots; }

// Both estimates were fitted to products without a residual: half of either side's lie between 0.87 and 1.1 of the measured time, the
// rest between 0.6 and 1.45.  The 1.76 us a round for what is not plain is one figure for all epilogues.  Medians of 500 products, over
// what is estimated without it: SiLU 3.5, tanh GELU 4.9, SwiGLU 0.2; a residual takes 1.4 and counts as plain, and the split-K kernel takes
// 1.2 of its estimate with one.  That matters near the line only: of 260 draws over 1 .. 3000 rows, 64 .. 30000 columns, K 64 .. 12000,
// with activations and residuals, the rule takes the slower kernel by more than 5 % in one; of 240 more whose estimates lie within 0.6 to 1.6
// of each other, in 12 (179 x 14800 x 64 SiLU + residual split-K 16.3 | 9.0 us, 463 x 3808 x 512 + residual split-K 11.5 | 9.0, 273 x 7856 x 1984
// GELU 17.7 | 20.4 persistent).
// us, split-K | the persistent kernel, taken where the first is smaller: 24 x 22016 x 4096 33 | 39; 120 x 4096 x 11008 25 | 66; 120 x 12288 x 4096
// 27 | 42; 1 x 4096 x 4096 10 | 26; 64 x 50000 x 4096 75 | 88; 256 x 4096 x 4096 17 | 24; 512 x 4096 x 4096 23.6 | 24.3; 1000 x 4096 x
// 4096 36 | 32; 256 x 22016 x 4096 60 | 58; 151 x 928 x 10768 SiLU 14.5 | 56; batches of short products run several waves: 122 x (52 x 1056 x
// 88) 38 | 12; 62 x (21 x 1320 x 248) 26 | 11; 35 x (62 x 1976 x 160) 15 | 8.3; 4 x (510 x 152 x 168) 3.9 | 5.4.
inline bool gemm_split_wins(const GemmSplitChoice& split, const GemmWide& w, int k_steps, bool plain, double bytes) {
  const double round = k_steps * (w.one_row ? 424.0 : 316.0) + (w.one_row ? 880.0 : 1280.0) + (plain ? 0.0 : 1760.0);
  const long long rounds = (w.tiles + w.slots - 1) / w.slots;
  return split.rule_ns < std::max(rounds * round, bytes / 6250.0) + 3440.0;
}

}  // namespace hb
