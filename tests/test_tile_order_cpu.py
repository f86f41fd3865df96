"""The work lists of the persistent attention kernels: whatever the order, every block of every head is taken exactly once; the division they are decoded with is exact."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r'''
#include <cstdio>
#include <vector>
#include "heddle_b200/csrc/tile_order.h"
int main() {
  int lists = 0;
  for (int heads : {1, 2, 7, 64, 149, 1000})
    for (int blocks : {1, 2, 3, 5, 16, 33})
      for (int masked : {0, 1})
        for (double bytes : {1.0, 1e12})
          for (int sms : {1, 2, 148}) {
            hb::TileOrder o;
            const int grid = hb::tile_order_fill(&o, heads, blocks, masked != 0, bytes, sms);
            if (grid < 1 || grid > sms) return printf("grid %d of %d\n", grid, sms), 1;
            std::vector<int> seen(heads * blocks, 0);
            for (int cta = 0; cta < grid; ++cta)
              for (int g = cta; g < o.total; g += grid)
                for (int half = 0; half < 2; ++half) {
                  int head, rank;
                  if (!hb::tile_order_get(o, g, half, head, rank)) continue;
                  if (head < 0 || head >= heads || rank < 0 || rank >= blocks) return printf("out of range\n"), 1;
                  ++seen[head * blocks + rank];
                }
            for (int n : seen)
              if (n != 1) return printf("heads %d blocks %d mode %d: taken %d times\n", heads, blocks, o.mode, n), 1;
            ++lists;
          }
  for (unsigned d = 1; d < 3000; ++d) {  // the division behind it, at every multiple's edge and at the ends of its range
    const hb::FastDiv f = hb::make_fast_div(d);
    for (long long n = 0; n < 4000000; n += d)
      if (hb::fast_div((int)n, f) != (int)(n / d) || (n > 0 && hb::fast_div((int)n - 1, f) != (int)((n - 1) / d))) return printf("%lld / %u\n", n, d), 1;
    for (int n : {2147483647, 2147483646, 1 << 30, (1 << 30) - 1})
      if (hb::fast_div(n, f) != (int)(n / d)) return printf("%d / %u\n", n, d), 1;
  }
  for (unsigned d : {2147483647u, 2147483646u, 1u << 30, (1u << 30) + 1, 65537u, 1000003u})
    for (int n : {0, 1, 65536, 65537, 1000002, 1000003, 2147483647, 2147483646, 1 << 30, (1 << 30) + 1})
      if (hb::fast_div(n, hb::make_fast_div(d)) != (int)(n / d)) return printf("%d / %u\n", n, d), 1;
  printf("%d lists\n", lists);
}
'''


def test_every_block_is_taken_once(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.strip() == "432 lists"


MODES = r'''
#include <cstdio>
#include "heddle_b200/csrc/tile_order.h"
int main() {
  struct { int heads, blocks; double bytes; hb::PairsFrom from; int mode; } cases[] = {
      {320, 10, 2.0 * 1166 * 128, hb::kPairsFromH2o, hb::kOrderPairs},   // pairs fill their rounds: 92 us, snake 107
      {128, 16, 2.0 * 1931 * 128, hb::kPairsFromH2o, hb::kOrderPairs},   // 88 | 99
      {64, 24, 2.0 * 3000 * 128, hb::kPairsFromH2o, hb::kOrderSnake},    // 102 | 92
      {192, 11, 2.0 * 1361 * 64, hb::kPairsFromH2o, hb::kOrderSnake},    // 82 | 80
      {144, 10, 4.0 * 1264 * 128, hb::kPairsFromDkdv, hb::kOrderPairs},  // 134 | 150
      {48, 23, 4.0 * 2881 * 64 * 2, hb::kPairsFromDkdv, hb::kOrderSnake},  // 316 | 309
      {144, 10, 4.0 * 1264 * 128, hb::kPairsFromDq128, hb::kOrderPairs},   // 103 | 111
      {128, 31, 4.0 * 3852 * 128 / 4, hb::kPairsFromDq128, hb::kOrderSnake},  // 628 | 616
      {768, 4, 2.0 * 425 * 128, hb::kPairsFromH2o, hb::kOrderPairs},        // 84 MB: 50 | 54
      {64, 21, 4.0 * 2614 * 128, hb::kPairsFromDkdv, hb::kOrderPairs},      // 86 MB: 228 | 237
      {80, 14, 4.0 * 823 * 64 * 2, hb::pairs_from(hb::kPairsFromDkdv, 823, 1775), hb::kOrderSnake},  // not square: 181 | 164
      {256, 28, 2.0 * 3562 * 64 / 2, hb::pairs_from(hb::kPairsFromH2o, 3562, 3587), hb::kOrderPairs},
      {96, 7, 4.0 * 1600 * 128, hb::kPairsNever, hb::kOrderSnake},
      {128, 16, 4.0 * 4096 * 128, hb::kPairsNever, hb::kOrderPairs},     // 268 MB: more than L2
  };
  int i = 0;
  for (auto& c : cases) {
    hb::TileOrder o;
    hb::tile_order_fill(&o, c.heads, c.blocks, true, c.bytes, 148, c.from);
    if (o.mode != c.mode) return printf("case %d: mode %d\n", i, o.mode), 1;
    ++i;
  }
}
'''


def test_the_order_is_the_one_that_was_measured_faster(tmp_path):
    (tmp_path / "m.cpp").write_text(MODES)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT), str(tmp_path / "m.cpp"), "-o", str(tmp_path / "m")], check=True)
    r = subprocess.run([str(tmp_path / "m")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
