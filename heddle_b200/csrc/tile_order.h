// Order in which the persistent attention kernels (forward, H2O score, both backward kernels) walk their work, one entry being
// one block of rows or keys of one head.  Every CTA of the grid takes entries blockIdx.x, blockIdx.x + gridDim.x, ...
//
//   kOrderPairs   entry g is the PAIR (rank r, rank nb - 1 - r) of one head, where rank 0 is the block that costs most; under
//                 a causal mask all pairs cost the same.  Head after head: few heads share L2 at one time.  Best when there are
//                 many pairs per SM, else the last round of pairs leaves most of the chip idle.
//   kOrderSnake   entries are single blocks, the dearest blocks of all heads first; odd rounds run backwards over the CTAs, so
//                 a CTA that got a dear block gets a cheap one.  All heads are in flight at one time, so this is the order
//                 where what they read stays in L2.
//   kOrderHeads   single blocks, head after head, where that is fewer blocks for the longest CTA (no mask: all blocks cost the
//                 same; at a tie the pairs are 3 % faster: dK/dV B8 H12 S577 D64 42.3 | 43.8 us).
//
// us, pairs | single blocks (bf16, D 128): forward, causal, B2 Hq32 Hkv8 S3000 165 | 146, B1 H128 (Hkv16) S2023 196 | 161, B7 H8
// S1077 on 1318 keys 72 | 43, B1 H8 S1287 43 | 30; unmasked B8 H12 S577 D64 46 | 28.  dQ, first case: 217 | 200.  With more
// than L2 to share the pairs win: forward B8 H32 S2048 (268 MB) 291 | 310, dK/dV B1 H128 (Hkv16) S2023 (132 MB) 271 | 332.
#pragma once

#include "fast_div.h"

namespace hb {

enum : int { kOrderPairs = 0, kOrderSnake = 1, kOrderHeads = 2 };

struct TileOrder {
  int heads, blocks;
  int mode;
  int npairs;           // kOrderPairs: ceil(blocks / 2)
  int total;            // bound of the entry index (kOrderSnake: rounded up to whole rounds)
  FastDiv by_npairs, by_blocks, by_heads, by_grid;
};

// Entry g of the list (half 0 or 1 of a pair): head and rank, or false where there is none.
HB_HD bool tile_order_get(const TileOrder& o, int g, int half, int& head, int& rank) {
  if (o.mode == kOrderPairs) {
    head = fast_div(g, o.by_npairs);
    const int pair = g - head * o.npairs;
    rank = half == 0 ? pair : o.blocks - 1 - pair;
    return half == 0 || rank != pair;  // the middle block of an odd count is one entry
  }
  if (half != 0) return false;
  if (o.mode == kOrderHeads) {
    head = fast_div(g, o.by_blocks);
    rank = g - head * o.blocks;
    return true;
  }
  const int grid = static_cast<int>(o.by_grid.d);
  const int round = fast_div(g, o.by_grid), cta = g - round * grid;
  const int u = round * grid + ((round & 1) ? grid - 1 - cta : cta);
  if (u >= o.heads * o.blocks) return false;
  rank = fast_div(u, o.by_heads);
  head = u - rank * o.heads;
  return true;
}

// From which fill of the rounds of pairs on pairs are the faster order under a mask: snake then gains little and its heads, all in
// flight, share L2 worse, the more so the more of it they need.  That is for the mask of a square problem: with more than a block
// of earlier keys pairs cost unequal amounts, and snake is the better balance (dK/dV B5 Hq32 Hkv16 S823 on 1775 keys D64, fill
// 0.95: 181 | 164 us).  The forward kernel stays with snake whatever the fill (0.81 to 1.03 of the pairs' time at fills of 0.93 to
// 1); dQ with D 64 too (0.92 to 0.99, one 1.003).  us, pairs | snake, bf16: H2O score B10 Hq32 Hkv16 S1166 D128 (fill 0.98) 92 | 107,
// B4 H32 S1931 D128 (0.99) 88 | 99, B10 H32 S955 D64 (0.96) 64 | 68, below it B3 Hq64 Hkv16 S1361 D64 (0.89) 82 | 80; dK/dV B9 H16
// S1264 D128 (0.97) 134 | 150, B3 H32 S3735 D64 (0.97) 522 | 552, below it B6 Hq16 Hkv8 S2881 D64 (0.93) 316 | 309; dQ B9 H16 S1264
// D128 (0.97) 103 | 111, below it B1 Hq128 Hkv32 S3852 D128 (0.96) 628 | 616.  Over 75 MB: H2O B3 Hq256 Hkv32 S425 D128 (0.94) 50 | 54,
// B5 Hq32 Hkv16 S1891 D128 (0.90) 105 | 108, dK/dV B2 H32 S2614 D128 (0.91) 228 | 237.
struct PairsFrom {
  double fill, crowded;  // up to 75 MB of common operands, and over it
};
constexpr PairsFrom kPairsFromH2o = {0.945, 0.90}, kPairsFromDkdv = {0.94, 0.90}, kPairsFromDq128 = {0.965, 0.965}, kPairsNever = {2.0, 2.0};
inline PairsFrom pairs_from(const PairsFrom& square, int Sq, int Skv) { return Skv - Sq <= 128 ? square : kPairsNever; }

// `bytes_per_head`: what the blocks of one head read in common.  Returns the grid size.
inline int tile_order_fill(TileOrder* o, long long heads, int blocks, bool masked, double bytes_per_head, int sm_count,
                           const PairsFrom& pairs_from = kPairsNever) {
  constexpr double kL2Budget = 96e6;  // of 126 MB: the rest is for what the blocks do not share
  constexpr double kL2Crowded = 75e6;
  o->heads = static_cast<int>(heads);
  o->blocks = blocks;
  o->npairs = (blocks + 1) / 2;
  const long long units = heads * blocks, pairs = heads * o->npairs;
  // rounds of the longest CTA, in blocks
  const long long rounds = (units + sm_count - 1) / sm_count, pair_rounds = 2 * ((pairs + sm_count - 1) / sm_count);
  const double pairs_fill = (double)units / ((double)pair_rounds * sm_count);
  const double common = heads * bytes_per_head, limit = common > kL2Crowded ? pairs_from.crowded : pairs_from.fill;
  if (masked) o->mode = common <= kL2Budget && pairs_fill < limit ? kOrderSnake : kOrderPairs;
  else o->mode = rounds < pair_rounds ? kOrderHeads : kOrderPairs;
  if (units > 0x3fff0000LL) o->mode = kOrderPairs;
  const long long entries = o->mode == kOrderPairs ? pairs : units;
  const int grid = static_cast<int>(entries < sm_count ? entries : sm_count);
  o->total = static_cast<int>(o->mode == kOrderSnake ? (entries + grid - 1) / grid * grid : entries);
  o->by_npairs = make_fast_div(static_cast<uint32_t>(o->npairs));
  o->by_blocks = make_fast_div(static_cast<uint32_t>(blocks));
  o->by_heads = make_fast_div(static_cast<uint32_t>(o->heads));
  o->by_grid = make_fast_div(static_cast<uint32_t>(grid));
  return grid;
}

// Steps of 128 keys (or queries) of an average CTA: `per_block` is the most a block has, a masked one half of that on average.
inline double tile_order_steps(const TileOrder& o, bool masked, double per_block) {
  return static_cast<double>(o.heads) * o.blocks * per_block * (masked ? 0.5 : 1.0) / o.by_grid.d;
}

}  // namespace hb
