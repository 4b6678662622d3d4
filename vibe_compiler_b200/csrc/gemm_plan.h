// How a tensor-core GEMM (gemm_umma.cu) is cut over the SMs: host arithmetic only.
#pragma once

#include <algorithm>
#include <cmath>

#include "kernels.h"

namespace wb200 {

constexpr int kBM = 128, kBN = 256, kBK = 64;

// How a problem is cut for the one-tile-per-CTA kernel (see choose_tile).
constexpr int kMaxTileStages = 10;
struct TilePlan {
  int tile_cols;    // output columns per tile: 64 or 128
  int tile_rows;    // output rows per tile: a multiple of 16 up to 256
  int stages;       // TMA ring; a stage holds two 64-element blocks of K
  int wide;         // 1: two stages serve as one of four blocks
  int row_bytes;    // bytes of A per block of K
  int tmem_cols;
};

constexpr int kTileSmemShared = 108 * 1024;   // ring of a CTA that shares its SM with another one
constexpr int kTileSmemAlone = 208 * 1024;

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

inline int64_t tile_count(const TilePlan &tile, const GemmUmmaArgs &a) { return static_cast<int64_t>(ceil_div(a.n, tile.tile_cols)) * ceil_div(a.m, tile.tile_rows); }

// Fills in what follows from the tile's size.
inline TilePlan make_tile(int tile_cols, int tile_rows, const GemmUmmaArgs &a, int sm_count) {
  TilePlan plan;
  plan.tile_cols = tile_cols;
  plan.tile_rows = tile_rows;
  plan.row_bytes = a.lhs_transposed ? ceil_div(tile_rows, 64) * 8192 : tile_rows * 128;
  const int stage = 2 * (tile_cols * kBK * 2 + plan.row_bytes);
  const bool alone = static_cast<int64_t>(ceil_div(a.n, tile_cols)) * ceil_div(a.m, tile_rows) <= sm_count || tile_rows > 64;
  // the ring is also the accumulator's staging area; more stages than blocks of K would stay empty
  const int need = std::max({ceil_div(a.k, 2 * kBK), ceil_div(tile_rows * tile_cols * 4, stage), 2});
  plan.stages = std::min({(alone ? kTileSmemAlone : kTileSmemShared) / stage, kMaxTileStages, need});
  // A stage costs the issuing warp about 310 clocks besides its products (the wait, descriptors, election, commit), which take
  // 28 clocks each at 64 columns: four blocks of K to a stage where at least four such stages fit.
  plan.wide = plan.stages >= 8;
  if (plan.wide) plan.stages &= ~1;
  plan.tmem_cols = 32;
  while (plan.tmem_cols < tile_rows) plan.tmem_cols *= 2;
  return plan;
}

// Estimated clocks of a launch of either kernel; the cheaper one runs. Measured at 1.9 GHz with cold caches (both sides in
// us, the launch on an idle stream included): a block of 64 of K costs a CTA about 300 clocks however few rows or columns it
// covers (two blocks to a stage; about 190 with four, but none of 19861 shapes drawn from 8 to 8192 rows, 256 to 28672 columns and
// 256 to 14336 of K is cut differently with that), or its products, or its operand bytes at about 52 per clock, whichever is
// more; a pair of CTAs needs about 650 clocks for the same block of a 256 x 256 tile. Rows x columns x K: 16 x 6144 x 4096 pair 31 / tile 19, 128 x 4096 x 4096 30 / 20, 512 x 4096 x 4096 32 / 28,
// 1024 x 1024 x 8192 49 / 34, 8192 x 256 x 2048 24 / 22; the pairs win once their tiles fill the SMs: 1000 x 6144 x 4096
// 54 / 68, 512 x 28672 x 4096 101 / 165.
inline double tile_cost(const TilePlan &plan, const GemmUmmaArgs &a, int sm_count) {
  const double per_sm = std::ceil(static_cast<double>(ceil_div(a.n, plan.tile_cols)) * ceil_div(a.m, plan.tile_rows) / sm_count);
  const double block = std::max({300.0, 2.0 * plan.tile_rows, (plan.tile_cols * kBK * 2 + plan.row_bytes) / 52.0});
  return per_sm * ceil_div(a.k, kBK) * block + 5000.0 + 20.0 * plan.tile_rows;
}
inline double pair_cost(const GemmUmmaArgs &a, int sm_count) {
  const double waves = std::ceil(static_cast<double>(ceil_div(a.m, 2 * kBM)) * ceil_div(a.n, kBN) / (sm_count / 2));
  return waves * ceil_div(a.k, kBK) * 650.0 + 10000.0;
}

// The cheapest cut of at most `max_tiles` tiles; none (tile_rows = 0) if there is no such cut.
inline TilePlan choose_tile(const GemmUmmaArgs &a, int sm_count, int64_t max_tiles, double *cost) {
  TilePlan best{};
  *cost = 0;
  int last_rows = 0;
  for (const int limit : {256, 192, 128, 96, 64}) {
    const int tile_rows = ceil_div(ceil_div(a.m, ceil_div(a.m, limit)), 16) * 16;
    if (tile_rows == last_rows) continue;
    last_rows = tile_rows;
    for (const int tile_cols : {128, 64}) {
      const TilePlan plan = make_tile(tile_cols, tile_rows, a, sm_count);
      if (tile_count(plan, a) > max_tiles) continue;
      const double c = tile_cost(plan, a, sm_count);
      if (best.tile_rows == 0 || c < *cost) { best = plan; *cost = c; }
    }
  }
  return best;
}

struct GemmPlan {
  bool pairs;       // CTA pairs on 256 x 256 tiles; else one tile per CTA
  TilePlan tile;
  int grid;         // CTAs
};

// `sm_count`: SMs to use. `beside`: the others are kept for a kernel that runs beside this one, so at most sm_count CTAs are
// launched: the pairs are persistent on as many, and a cut into more tiles is out.
inline GemmPlan plan_gemm(const GemmUmmaArgs &a, int sm_count, bool beside) {
  GemmPlan plan;
  double tile_clocks;
  plan.tile = choose_tile(a, sm_count, beside ? sm_count : INT64_MAX, &tile_clocks);
  plan.pairs = plan.tile.tile_rows == 0 || pair_cost(a, sm_count) < tile_clocks;
  plan.grid = plan.pairs ? 2 * std::min(sm_count / 2, ceil_div(a.m, 2 * kBM) * ceil_div(a.n, kBN)) : static_cast<int>(tile_count(plan.tile, a));
  return plan;
}

}  // namespace wb200
