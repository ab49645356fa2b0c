// Work items of the persistent GEMM kernels.  Plain integer code, the same on host and device
// (tests/test_schedule_cpu.py compiles it for the CPU).
//
// `tiles` output tiles of KB K blocks each are dealt out to G CTAs in rounds, item t to CTA t % G.  When tiles is just
// above a multiple of G the last round leaves most CTAs idle (192 tiles on 148 SMs: 44 of them work on the second round).
// Then each of the last `rem` tiles is cut along K into `parts` items, one per CTA, and the CTA that finishes a tile's last
// part adds the partial sums up.  A cut tile sums its K range in other groups than a whole one, so an output row's last
// bits depend on whether its tile is cut: on the number of tiles (the batch), but not on how many CTAs walk the items.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define MOE_HD __host__ __device__ __forceinline__
#else
#define MOE_HD inline
#endif

constexpr int kMaxParts = 8;

struct WorkPlan {
  int whole;  // items [0, whole) are whole tiles
  int parts;  // items [whole, items) are parts, `parts` of them to a tile
  int items;
  int KB;
};

// rows: rows of an average tile, for what the partial sums cost.  Measured in K blocks of the FP8 kernels (about 0.6 us):
// with 128 rows, three parts of 11 K blocks took as long as the whole tile of 32, three of 37 saved a third of 112 (the
// down GEMM of the Mixtral shape at 512 tokens, 192 tiles on 148 SMs: 145 -> 118 us).
MOE_HD WorkPlan work_plan(int tiles, int KB, int G, int rows) {
  WorkPlan p{tiles, 1, tiles, KB};
  const int rem = tiles % G;
  if (rem == 0 || 2 * rem > G) return p;
  int most = G / rem;
  if (most > kMaxParts) most = kMaxParts;
  int best = KB - 1;  // a cut has to save two K blocks at least
  for (int s = 2; s <= most && s * 4 <= KB; ++s) {
    const int cost = (KB + s - 1) / s + 2 + rows * (2 + 6 * s) / 128;
    if (cost < best) best = cost, p.parts = s;
  }
  if (p.parts > 1) {
    p.whole = tiles - rem;
    p.items = p.whole + rem * p.parts;
  }
  return p;
}

struct WorkItem {
  int tile, kb0, KB;
};
MOE_HD WorkItem work_item(const WorkPlan& p, int t) {
  if (t < p.whole) return WorkItem{t, 0, p.KB};
  const int u = t - p.whole, q = u / p.parts, i = u - q * p.parts;
  const int b = p.KB * i / p.parts, e = p.KB * (i + 1) / p.parts;
  return WorkItem{p.whole + q, b, e - b};
}
// part item t belongs to shared tile work_shared(t); the items of shared tile q are whole + q * parts + [0, parts)
MOE_HD int work_shared(const WorkPlan& p, int t) { return (t - p.whole) / p.parts; }
