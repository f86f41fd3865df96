"""Which kernel AUTO runs for a product with few tiles: the rule takes the one that was measured to be the faster (both sides on
one B200, weights from HBM), and it does not depend on anything but sizes."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

# epilogue (0 plain, 1 SwiGLU, 2 RoPE; -1 plain with an activation), batch, M, N, K, [K, N] operand, us split-K, us persistent
MEASURED = [
    # one product: decode steps and short prompts, where tiles of 256 columns leave most SMs idle
    (1, 1, 24, 22016, 4096, 0, 33, 42), (0, 1, 120, 4096, 11008, 0, 25, 67), (2, 1, 120, 12288, 4096, 0, 30, 40),
    (0, 1, 1, 4096, 4096, 0, 11, 28), (0, 1, 64, 50000, 4096, 0, 75, 83), (0, 1, 256, 4096, 4096, 0, 17, 25),
    (0, 1, 512, 4096, 4096, 0, 23, 26), (0, 1, 1000, 4096, 4096, 0, 31, 28), (1, 1, 256, 22016, 4096, 0, 61, 56),
    (0, 1, 26, 25104, 1720, 0, 18.7, 28.9), (0, 1, 5, 23568, 840, 0, 10.7, 15.5), (0, 1, 548, 3584, 5624, 0, 34.9, 38.3),
    (2, 1, 344, 1408, 328, 0, 8.7, 13.9), (-1, 1, 151, 928, 10768, 0, 17.9, 86.0), (1, 1, 1913, 2368, 6072, 0, 99.2, 83.1),
    (1, 1, 2721, 1600, 4928, 0, 65.1, 54.3), (0, 1, 1581, 2896, 64, 0, 11.0, 5.8), (0, 1, 411, 11200, 208, 0, 13.7, 8.2),
    # batches of short products: several waves of CTAs, each with its own start
    (0, 122, 52, 1056, 88, 0, 39.0, 12.9), (0, 62, 21, 1320, 248, 1, 26.3, 11.0), (0, 26, 442, 272, 376, 0, 15.9, 9.0),
    (0, 35, 62, 1976, 160, 1, 14.7, 8.3), (0, 46, 96, 792, 160, 1, 13.7, 8.2), (0, 49, 180, 264, 120, 0, 10.8, 7.3),
    (0, 82, 12, 336, 144, 0, 9.0, 6.6), (0, 4, 510, 152, 168, 0, 4.2, 5.8), (0, 2, 663, 112, 64, 0, 3.2, 4.0),
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
