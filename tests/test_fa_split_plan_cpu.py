"""How the split-key attention kernel cuts its list of key tiles: every tile is walked once, every part of an item has a slot of its
own, and the merge visits each item in parts once and reads exactly the slots that were written."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r'''
#include <cstdio>
#include <vector>
#include "heddle_b200/csrc/fa_split_plan.h"
using namespace hb;
static int fail(const char* what, int B, int Hq, int Hkv, int Sq, int Skv) {
  printf("%s: B%d Hq%d Hkv%d Sq%d Skv%d\n", what, B, Hq, Hkv, Sq, Skv);
  return 1;
}
int main() {
  int whole = 0, even = 0, flat = 0, few = 0, crossing = 0, middle = 0;
  for (int sms : {1, 4, 132, 148})
    for (int B : {1, 2, 5, 13, 16, 38, 200})
      for (int Hkv : {1, 4, 8, 32})
        for (int group : {1, 3, 8, 17})
          for (int Sq : {1, 4, 16, 17, 65, 128})
            for (int Skv : {1, 128, 129, 1000, 3000, 6001, 40000}) {
              if (Skv < Sq || (long long)B * Hkv * group * Skv > 40000000) continue;
              const int Hq = Hkv * group;
              const FaSplitPlan p = fa_split_plan(B, Hq, Hkv, Sq, Skv, sms);
              const long long total = (long long)p.items * p.nkv;
              if (p.rows != p.hb * Sq || p.rows > 128 || p.hb * p.hgroups < group || p.pipes < 1 || p.pipes > 2 * sms)
                return fail("plan", B, Hq, Hkv, Sq, Skv);
              if (fa_split_begin(p, 0) != 0 || fa_split_begin(p, p.pipes) != total) return fail("ends", B, Hq, Hkv, Sq, Skv);
              std::vector<int> owner(2 * p.pipes, -1), parts(p.items, 0), done(p.items, 0);
              long long next = 0;
              for (int w = 0; w < p.pipes; ++w) {
                const long long end = fa_split_begin(p, w + 1);
                bool first = true;
                for (long long t = fa_split_begin(p, w); t < end; first = false) {
                  int item, j0, j1;
                  fa_split_segment(p, t, end, item, j0, j1);
                  if (t != next || item < 0 || item >= p.items || j0 < 0 || j1 <= j0 || j1 > p.nkv || item * (long long)p.nkv + j0 != t)
                    return fail("walk", B, Hq, Hkv, Sq, Skv);
                  next += j1 - j0;
                  t += j1 - j0;
                  if (j0 == 0 && j1 == p.nkv) {
                    ++done[item];
                    middle += p.cuts && !first && t < end;
                    continue;
                  }
                  if (!p.cuts) return fail("a part without cuts", B, Hq, Hkv, Sq, Skv);
                  const long long slot = 2ll * w + (first ? 0 : 1);  // as the kernel's roles count
                  if (slot != fa_split_slot(p, w, item) || owner[slot] != -1) return fail("slot", B, Hq, Hkv, Sq, Skv);
                  owner[slot] = item;
                  ++parts[item];
                  crossing += !first;
                }
              }
              if (next != total) return fail("tiles left", B, Hq, Hkv, Sq, Skv);
              const bool is_even = p.cuts && p.pipes % p.items == 0 && total % p.pipes == 0;
              ++(!p.cuts ? whole : is_even ? even : flat);
              if (!p.cuts) {
                for (int n : done)
                  if (n != 1) return fail("item", B, Hq, Hkv, Sq, Skv);
                continue;
              }
              few += p.pipes <= p.items;
              const int candidates = fa_split_candidates(p);
              if (candidates < 1) return fail("no candidate", B, Hq, Hkv, Sq, Skv);
              for (int c = 0; c < candidates; ++c) {
                const int item = fa_split_candidate(p, c);
                if (item < 0) continue;
                int w0, w1;
                fa_split_pipes_of(p, item, w0, w1);
                if (w0 == w1) continue;  // the kernel wrote it itself
                ++done[item];
                if (w1 - w0 + 1 != parts[item]) return fail("parts", B, Hq, Hkv, Sq, Skv);
                for (int w = w0; w <= w1; ++w)
                  if (owner[w == w0 ? fa_split_slot(p, w0, item) : 2ll * w] != item) return fail("read", B, Hq, Hkv, Sq, Skv);
              }
              for (int n : done)
                if (n != 1) return fail("item in parts", B, Hq, Hkv, Sq, Skv);
            }
  if (!whole || !even || !flat || !few || !crossing || !middle) return fail("a form is missing", 0, 0, 0, 0, 0);
  printf("whole %d even %d flat %d, fewer runs than items %d\n", whole, even, flat, few);
  // whole items of one head each between two and three rounds of SMs: the general kernel (us here | there in the header)
  struct { int B, Hq, Hkv, Sq, Skv, D; bool general; } calls[] = {
      {23, 16, 4, 128, 128, 128, true}, {3, 128, 16, 100, 100, 128, true}, {22, 16, 16, 100, 442, 128, true}, {19, 16, 16, 100, 357, 128, true},
      {76, 8, 2, 128, 413, 128, false}, {1050, 2, 2, 128, 314, 128, false}, {97, 16, 16, 65, 65, 128, false}, {25, 64, 16, 120, 120, 64, false},
      {18, 16, 16, 128, 128, 128, false}, {23, 16, 4, 128, 128, 64, false}, {40, 32, 4, 1, 300, 128, false}, {16, 64, 8, 1, 6001, 128, false}};
  for (auto& c : calls)
    if (fa_split_general_wins(fa_split_plan(c.B, c.Hq, c.Hkv, c.Sq, c.Skv, 148), c.D, 148) != c.general)
      return fail("general", c.B, c.Hq, c.Hkv, c.Sq, c.Skv);
  // the merge is as large as what there is to merge, not as the number of items
  const FaSplitPlan p = fa_split_plan(38, 256, 32, 16, 4096, 148);
  if (!p.cuts || fa_split_candidates(p) * p.rows > 2 * 148 * 128) return fail("merge", 38, 256, 32, 16, 4096);
}
'''


def test_every_tile_once_and_every_part_merged(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(ROOT), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    print(r.stdout)
