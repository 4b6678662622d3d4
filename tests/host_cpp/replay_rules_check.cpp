// Host check of the rules by which commands of a replayed Tile program share a launch (csrc/replay_rules.h): whatever they let
// join, run in any order, leaves memory as the commands in their own order do, for every Tile.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "../../vibe_compiler_b200/csrc/replay_rules.h"

using namespace wb200;

static int failures = 0;
static void expect(bool ok, const char *what) {
  if (!ok && ++failures < 10) printf("%s\n", what);
}

// Copies between a Tile's scratch-pad and DDR, 64 bytes each.
static void run_copy(const ReplayCopy &copy, int tile, std::vector<uint8_t> &spm, std::vector<uint8_t> &ddr) {
  std::vector<uint8_t> &from = copy.load ? ddr : spm, &to = copy.load ? spm : ddr;
  const size_t source = copy.source.begin + tile * copy.source.step, destination = copy.destination.begin + tile * copy.destination.step;
  const std::vector<uint8_t> moved(from.begin() + source, from.begin() + source + (copy.source.end - copy.source.begin));
  std::copy(moved.begin(), moved.end(), to.begin() + destination);
}

static void check_copies() {
  std::mt19937 random(1);
  auto below = [&](int n) { return static_cast<int>(random() % n); };
  const int spm_image = 0, ddr_image = 0;
  int joined = 0, several_steps = 0;
  for (int round = 0; round < 200000; ++round) {
    const int tiles = 1 + below(4), count = 2 + below(3);
    std::vector<ReplayCopy> copies;
    for (int i = 0; i < count; ++i) {
      const uint64_t bytes = 1 + below(6), spm = below(60 - bytes), step = below(3) * 4;
      // Tile addresses stay inside DDR whichever way they go
      const bool down = below(4) == 0;
      const uint64_t ddr = down ? (tiles - 1) * step + below(24) : below(24);
      const ReplayRange in_spm{&spm_image, spm, spm + bytes, 0};
      const ReplayRange in_ddr{&ddr_image, ddr, ddr + bytes, down ? -static_cast<int64_t>(step) : static_cast<int64_t>(step)};
      const bool load = below(2);
      copies.push_back({load ? in_ddr : in_spm, load ? in_spm : in_ddr, below(4) ? 1u : 4u, load});
    }
    int held = 1;
    while (held < count && copies_join(copies.data(), held, copies[held], tiles)) ++held;
    if (held == 1) continue;
    ++joined;
    for (int i = 1; i < held; ++i) several_steps += copies[i].destination.step != copies[0].destination.step;
    for (int tile = 0; tile < tiles; ++tile) {
      std::vector<uint8_t> spm(64), ddr(64);
      for (int i = 0; i < 64; ++i) { spm[i] = i; ddr[i] = 128 + i; }
      std::vector<uint8_t> want_spm = spm, want_ddr = ddr;
      for (int i = 0; i < held; ++i) run_copy(copies[i], tile, want_spm, want_ddr);
      std::vector<int> order(held);
      for (int i = 0; i < held; ++i) order[i] = i;
      do {
        std::vector<uint8_t> got_spm = spm, got_ddr = ddr;
        for (int i : order) run_copy(copies[i], tile, got_spm, got_ddr);
        expect(got_spm == want_spm && got_ddr == want_ddr, "copies that joined depend on their order");
      } while (std::next_permutation(order.begin(), order.end()));
    }
  }
  expect(joined > 1000 && several_steps > 100, "the copies drawn miss a case");
  // Tile t stores to slot 2t and then to slot 1 + t: apart for Tile 0, one slot for Tile 1.
  auto store = [&](uint64_t from, uint64_t slot, int64_t step) {
    return ReplayCopy{{&spm_image, from, from + 4, 0}, {&ddr_image, 4 * slot, 4 * slot + 4, 4 * step}, 4, false};
  };
  const ReplayCopy first = store(0, 0, 2), second = store(8, 1, 1), same_step = store(8, 1, 2);
  expect(copies_join(&first, 1, second, 1) && !copies_join(&first, 1, second, 2) && copies_join(&first, 1, same_step, 8), "stores of two steps");
}

int main() {
  check_copies();
  printf(failures ? "FAILED %d\n" : "PASS\n", failures);
  return failures != 0;
}
