// Host check of the cut of tensor-core GEMMs (csrc/gemm_plan.h): what the kernels rely on, and the number of CTAs where SMs are
// kept for a kernel that runs beside the GEMM.
#include "../../vibe_compiler_b200/csrc/gemm_plan.h"

using namespace wb200;

int main() {
  int failures = 0, beside_tiles = 0, cut_differently = 0;
  auto expect = [&](bool ok, const char *what, const GemmUmmaArgs &a, int sms) {
    if (!ok && ++failures < 10) printf("%s: %d x %d x %d on %d SMs\n", what, a.m, a.n, a.k, sms);
  };
  for (int m : {8, 16, 24, 72, 128, 136, 256, 264, 512, 1000, 2048, 4096, 8192, 65528})
    for (int n : {8, 64, 96, 256, 512, 768, 1024, 3584, 4096, 6144, 7168, 28672})
      for (int k : {8, 64, 136, 512, 1792, 4096, 14336})
        for (int transposed : {0, 1})
          for (int sms : {148, 144, 140, 132, 124, 16})
            for (bool beside : {false, true}) {
              GemmUmmaArgs a{};
              a.m = m; a.n = n; a.k = k; a.lhs_transposed = transposed;
              const GemmPlan plan = plan_gemm(a, sms, beside);
              expect(plan.grid >= 1 && (!beside || plan.grid <= sms), "more CTAs than SMs", a, sms);
              if (beside && plan_gemm(a, sms, false).grid > sms) ++cut_differently;
              if (plan.pairs) {
                expect(plan.grid % 2 == 0 && plan.grid <= sms, "pairs", a, sms);
                continue;
              }
              beside_tiles += beside;
              const TilePlan &t = plan.tile;
              const int block = t.tile_cols * kBK * 2 + t.row_bytes;
              expect((t.tile_cols == 64 || t.tile_cols == 128) && t.tile_rows % 16 == 0 && t.tile_rows >= 16 && t.tile_rows <= 256, "tile", a, sms);
              expect(t.stages >= 2 && t.stages <= kMaxTileStages && 2 * t.stages * block <= kTileSmemAlone, "ring", a, sms);
              expect(t.tile_rows * t.tile_cols * 4 <= 2 * t.stages * block, "staging of the accumulator", a, sms);
              expect(t.tmem_cols >= t.tile_rows && t.tmem_cols >= 32 && (t.tmem_cols & (t.tmem_cols - 1)) == 0, "tensor memory", a, sms);
              expect(plan.grid == tile_count(t, a), "every tile has a CTA", a, sms);
            }
  if (!beside_tiles || !cut_differently) { printf("the ranges miss a case\n"); ++failures; }
  printf(failures ? "FAILED %d\n" : "PASS\n", failures);
  return failures != 0;
}
