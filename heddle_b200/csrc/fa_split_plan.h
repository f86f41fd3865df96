// The work of the split-key attention kernel (fa_split_sm100.cuh): the list of key tiles, the runs it is cut into, the workspace
// slots of partial segments and the items that have any.  Shared by the launch, the kernels and a test on the CPU.
#pragma once

#include <algorithm>

#include "fast_div.h"

namespace hb {

constexpr int kFaSplitTile = 128;  // rows of a packed query tile, keys of a key tile

struct FaSplitPlan {
  int hb;       // query heads of a row tile
  int hgroups;  // row tiles per (batch, kv head) = ceil(group / hb)
  int rows;     // hb * Sq <= 128
  int nkv;      // 128-key tiles
  int items;    // B * Hkv * hgroups
  int pipes;    // runs the list of items * nkv tiles is cut into
  int cuts;     // 0: every run is a run of whole items
};

inline FaSplitPlan fa_split_plan(int B, int Hq, int Hkv, int Sq, int Skv, int sm_count) {
  FaSplitPlan pl;
  const int group = Hq / Hkv;
  pl.hgroups = (group + kFaSplitTile / Sq - 1) / (kFaSplitTile / Sq);
  pl.hb = (group + pl.hgroups - 1) / pl.hgroups;
  pl.hgroups = (group + pl.hb - 1) / pl.hb;
  pl.rows = pl.hb * Sq;
  pl.nkv = (Skv + kFaSplitTile - 1) / kFaSplitTile;
  pl.items = B * Hkv * pl.hgroups;  // fits: the caller bounds B * Hq
  // How many runs: the tiles of the longest one, plus what partial results cost in tiles (the combine launch, and each
  // partial segment's rows written and read again).  Items left whole; every item cut into the same number of runs; all
  // pipelines an equal share whatever the items.
  const long long total = (long long)pl.items * pl.nkv, cap = 2ll * sm_count;
  const long long whole = (pl.items + cap - 1) / cap * pl.nkv;
  pl.pipes = (int)std::min<long long>(cap, pl.items);
  pl.cuts = 0;
  long long best = whole;
  const long long even = std::min<long long>(cap / pl.items, pl.nkv);
  if (even > 1) {
    const long long cost = (pl.nkv + even - 1) / even + 3 + pl.rows / 12;
    if (cost < best) {
      best = cost;
      pl.pipes = (int)(pl.items * even);
      pl.cuts = 1;
    }
  }
  const long long flat = std::min(cap, total);
  if ((total + flat - 1) / flat + 3 + pl.rows / 10 < best) {
    pl.pipes = (int)flat;
    pl.cuts = 1;
  }
  return pl;
}

// Whether the general kernel (a 256-row block per query head, an SM each) is the faster one for a call of at most 128 query rows.
// Where one head fills a row tile nothing is packed, and where items stay whole nothing is shared out; then the general kernel's
// rounds of blocks are finer than this kernel's, two items an SM at a time.  It matters where three of them stand against two of
// these: us, here | general, D 128: 368 prompts of 128 rows 16.0 | 12.9, 384 of 100 rows 15.7 | 13.7, 352 of 100 rows on 442 keys 33.8
// | 30.2, 304 on 357 27.0 | 22.9.  Elsewhere a round here is 0.8 of the time (608 prompts of 128 rows on 413 keys 45 | 47, 2100 on 314
// 91 | 109), less with up to 96 rows (1552 of 65 rows 34 | 45) and with D 64 (1600 of 120 rows 30 | 40).
inline bool fa_split_general_wins(const FaSplitPlan& p, int D, int sm_count) {
  return D == 128 && p.hb == 1 && p.rows > 96 && !p.cuts && p.items > 2 * sm_count && p.items <= 3 * sm_count;
}

// Run of pipeline w: key tiles [begin(w), begin(w + 1)) of the list.
HB_HD long long fa_split_begin(const FaSplitPlan& p, int w) {
  const long long n = static_cast<long long>(w) * p.items;
  return p.cuts ? n * p.nkv / p.pipes : n / p.pipes * p.nkv;
}
// The segment of a run that starts at list position t: key tiles [j0, j1) of an item.
HB_HD void fa_split_segment(const FaSplitPlan& p, long long t, long long end, int& item, int& j0, int& j1) {
  item = static_cast<int>(t / p.nkv);
  j0 = static_cast<int>(t - static_cast<long long>(item) * p.nkv);
  const long long last = j0 + (end - t);
  j1 = last < p.nkv ? static_cast<int>(last) : p.nkv;
}
// Pipelines [w0, w1] have a part of an item (cuts != 0): the pipeline of tile t is the last w with begin(w) <= t.
HB_HD void fa_split_pipes_of(const FaSplitPlan& p, int item, int& w0, int& w1) {
  const long long total = static_cast<long long>(p.items) * p.nkv, t0 = static_cast<long long>(item) * p.nkv;
  w0 = static_cast<int>(((t0 + 1) * p.pipes - 1) / total);
  w1 = static_cast<int>(((t0 + p.nkv) * p.pipes - 1) / total);
}
// Workspace slot of pipeline w's part of an item.  A run has at most two parts of items: its first segment and, where that is
// another one, its last.
HB_HD int fa_split_slot(const FaSplitPlan& p, int w, int item) {
  return fa_split_begin(p, w) / p.nkv == item ? 2 * w : 2 * w + 1;
}
// Candidates for an item in parts: every item, or, where there are fewer, every boundary between two runs.
HB_HD int fa_split_candidates(const FaSplitPlan& p) { return p.pipes <= p.items ? p.pipes - 1 : p.items; }
// The candidate's item, -1 if the boundary cuts none or the item is the one of the boundary before.
HB_HD int fa_split_candidate(const FaSplitPlan& p, int c) {
  if (p.pipes > p.items) return c;
  const long long b = fa_split_begin(p, c + 1), item = b / p.nkv, t0 = item * p.nkv;
  if (b == t0 || (c > 0 && fa_split_begin(p, c) > t0)) return -1;
  return static_cast<int>(item);
}

}  // namespace hb
