"""The work split of the persistent GEMM kernels (csrc/schedule.h), compiled for the CPU: every K block of every tile is
worked on exactly once, a CTA has at most one part (its last item), and nothing takes longer than whole tiles would."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "torch-tpu_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "schedule.h"
#define REQUIRE(c) do { if (!(c)) { std::printf("tiles %d KB %d G %d rows %d: %s\n", tiles, KB, G, rows, #c); return 1; } } while (0)
static int check(int tiles, int KB, int G, int rows) {
  const WorkPlan p = work_plan(tiles, KB, G, rows);
  std::vector<int> seen((size_t)tiles * KB, 0);
  long longest = 0;
  REQUIRE(p.parts >= 1 && p.parts <= kMaxParts && p.items - p.whole <= G && (p.parts == 1 || p.whole % G == 0));
  for (int c = 0; c < G; ++c) {
    long blocks = 0;
    for (int t = c; t < p.items; t += G) {
      const WorkItem w = work_item(p, t);
      REQUIRE(w.KB > 0 && w.kb0 >= 0 && w.kb0 + w.KB <= KB && w.tile >= 0 && w.tile < tiles);
      REQUIRE((t < p.whole) == (w.KB == KB) && (t < p.whole || t + G >= p.items));
      if (t >= p.whole) REQUIRE(w.tile == p.whole + work_shared(p, t) && work_shared(p, t) * p.parts + p.whole <= t);
      for (int k = 0; k < w.KB; ++k) ++seen[(size_t)w.tile * KB + w.kb0 + k];
      blocks += w.KB;
    }
    longest = blocks > longest ? blocks : longest;
  }
  for (int s : seen) REQUIRE(s == 1);
  REQUIRE(longest <= (long)((tiles + G - 1) / G) * KB);
  // fewer CTAs walk the same items: every part still has a slot of its own (its number among the parts)
  for (int g : {1, G / 3 + 1, G}) {
    std::vector<int> taken(G, 0);
    for (int c = 0; c < g; ++c)
      for (int t = c; t < p.items; t += g)
        if (t >= p.whole) REQUIRE(t - p.whole < G && ++taken[t - p.whole] == 1);
  }
  return 0;
}
int main() {
  std::srand(1);
  for (int G : {1, 5, 98, 148, 160})
    for (int KB : {1, 2, 4, 6, 8, 16, 32, 56, 112, 337})
      for (int n = 0; n < 80; ++n) {
        const int tiles = n < 12 ? n : n < 30 ? G - 9 + n - 12 : 1 + std::rand() % (n < 60 ? 3 * G : 5000);
        if (tiles >= 0 && check(tiles, KB, G, std::rand() % 129)) return 1;
      }
  // the cut is made where it pays and not where it does not
  if (work_plan(192, 32, 148, 8).parts < 2 || work_plan(192, 112, 148, 128).parts < 2) return std::printf("not cut\n"), 1;
  if (work_plan(192, 32, 148, 128).parts != 1 || work_plan(296, 32, 148, 128).parts != 1) return std::printf("cut\n"), 1;
  return 0;
}
"""


def test_every_k_block_is_worked_on_once(tmp_path):
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
