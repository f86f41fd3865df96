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
