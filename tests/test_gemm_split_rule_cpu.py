"""Which kernel AUTO runs for a product with few tiles: the rule takes the one that was measured to be the faster (both sides on
one B200, weights from HBM), and it does not depend on anything but sizes."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

# epilogue (0 plain, 1 SwiGLU, 2 RoPE; -1 plain with an activation), batch, M, N, K, [K, N] operand, us split-K, us persistent
MEASURED = [
    # one product: decode steps and short prompts, where tiles of 256 columns leave most SMs idle
    (1, 1, 24, 22016, 4096, 0, 32.8, 38.7), (0, 1, 120, 4096, 11008, 0, 25.7, 65.5), (2, 1, 120, 12288, 4096, 0, 26.7, 42.1),
    (0, 1, 1, 4096, 4096, 0, 9.9, 26.3), (0, 1, 64, 50000, 4096, 0, 75.2, 87.7), (0, 1, 256, 4096, 4096, 0, 16.7, 23.7),
    (0, 1, 512, 4096, 4096, 0, 23.6, 24.3), (0, 1, 1000, 4096, 4096, 0, 36.1, 31.8), (1, 1, 256, 22016, 4096, 0, 60.1, 57.7),
    (0, 1, 26, 25104, 1720, 0, 20.5, 26.4), (0, 1, 5, 23568, 840, 0, 11.2, 15.2), (0, 1, 548, 3584, 5624, 0, 37.4, 39.3),
    (2, 1, 344, 1408, 328, 0, 8.2, 18.4), (-1, 1, 151, 928, 10768, 0, 14.5, 56.0), (1, 1, 1913, 2368, 6072, 0, 87.5, 77.2),
    (1, 1, 2721, 1600, 4928, 0, 58.9, 52.6), (0, 1, 1581, 2896, 64, 0, 11.2, 5.6), (0, 1, 411, 11200, 208, 0, 14.2, 8.1),
    # SiLU and tanh GELU with a few hundred rows
    (-1, 1, 295, 2224, 1792, 0, 10.7, 17.6), (-1, 1, 598, 3088, 3136, 0, 18.7, 24.6), (-1, 1, 1014, 4352, 152, 0, 12.6, 11.2),
    (-1, 1, 714, 7472, 7616, 0, 103.5, 89.2), (-1, 1, 225, 10336, 800, 0, 12.3, 17.3), (-1, 1, 389, 11920, 1080, 0, 32.6, 27.6),
    # batches of short products: several waves of CTAs, each with its own start
    (0, 122, 52, 1056, 88, 0, 38.0, 12.4), (0, 62, 21, 1320, 248, 1, 26.3, 11.3), (0, 26, 442, 272, 376, 0, 16.1, 9.0),
    (0, 35, 62, 1976, 160, 1, 15.0, 8.3), (0, 46, 96, 792, 160, 1, 14.0, 8.0), (0, 49, 180, 264, 120, 0, 10.8, 7.3),
    (0, 82, 12, 336, 144, 0, 8.6, 6.2), (0, 4, 510, 152, 168, 0, 3.9, 5.4), (0, 2, 663, 112, 64, 0, 3.0, 3.8),
]

PROGRAM = r'''
#include <cstdio>
#include "heddle_b200/csrc/gemm_split_plan.h"
using namespace hb;
int main() {
  const int slots[kMaxSplits + 1] = {0, 148, 148, 135, 132, 130, 126, 126, 120};
  int epi, batch, M, N, K, kn;
  while (scanf("%d %d %d %d %d %d", &epi, &batch, &M, &N, &K, &kn) == 6) {
    const int cls = epi < 0 ? 0 : epi, n_out = cls == kEpiSwiglu ? N / 2 : N, steps = (K + 63) / 64;
    const GemmWide w = gemm_wide(148, M, N, batch);
    bool wins = false;
    if (gemm_split_eligible(w)) {
      const GemmSplitChoice c = gemm_split_choose(slots, 148, cls, M, n_out, steps, K % 64 == 0, batch, 128, kn != 0);
      if (c.width < 16 || c.width > 256 || c.splits < 1 || c.splits > kMaxSplits || c.slabs < 1 || c.slabs > 4) return 1;
      wins = gemm_split_wins(c, w, steps, epi == 0, 2.0 * batch * ((double)M * K + (double)N * K + (double)M * n_out));
    }
    printf("%d\n", wins);
  }
}
'''


def test_the_rule_takes_the_faster_kernel(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    lines = "".join(" ".join(str(x) for x in row[:6]) + "\n" for row in MEASURED)
    r = subprocess.run([str(tmp_path / "t")], input=lines, capture_output=True, text=True)
    assert r.returncode == 0
    wrong = [row for row, wins in zip(MEASURED, r.stdout.split()) if (wins == "1") != (row[6] < row[7])]
    assert not wrong
