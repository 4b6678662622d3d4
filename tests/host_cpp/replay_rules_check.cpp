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

// Elementwise commands over single bytes: the result depends on both operands and on the command.
static uint8_t evaluate(uint8_t lhs, uint8_t rhs, int step) { return static_cast<uint8_t>(3 * lhs + 5 * rhs + 17 * step + 1); }
static uint8_t second_operand(const ChainOperands &c, const std::vector<uint8_t> &memory, int element) {
  return c.rhs_bytes ? memory[c.rhs + element % c.rhs_bytes] : 9;
}

static void check_chains() {
  std::mt19937 random(2);
  auto below = [&](int n) { return static_cast<int>(random() % n); };
  int joined = 0, units = 0, revisits = 0, registers = 0;
  for (int round = 0; round < 200000; ++round) {
    const int bytes = 3 + below(8), places = 4;
    // Vectors at few places, some shifted by a byte or two; units in front of and inside them
    auto place = [&]() { return static_cast<uint64_t>(below(places) * 12 + (below(4) ? 0 : below(3))); };
    std::vector<ChainOperands> commands;
    for (int i = 0; i < 5; ++i) {
      ChainOperands c{place(), 0, place(), static_cast<uint64_t>(bytes), 0};
      if (i > 0 && below(2)) c.lhs = commands[i - 1].destination;
      const int form = below(3);
      if (form == 1) { c.rhs = place(); c.rhs_bytes = bytes; }
      if (form == 2) { c.rhs_bytes = 1 + below(bytes - 1); c.rhs = below(2) ? 48 + below(4) : place() + below(4); }
      commands.push_back(c);
    }
    if (chain_refuses(commands[0])) continue;
    int held = 1;
    while (held < 5 && chain_extends(commands.data(), held, commands[held])) ++held;
    std::vector<uint8_t> memory(64);
    for (int i = 0; i < 64; ++i) memory[i] = static_cast<uint8_t>(random());
    std::vector<uint8_t> want = memory;
    for (int s = 0; s < held; ++s) {   // command by command, every element read before any is stored
      const ChainOperands &c = commands[s];
      std::vector<uint8_t> results(bytes);
      for (int e = 0; e < bytes; ++e) results[e] = evaluate(want[c.lhs + e], second_operand(c, want, e), s);
      std::copy(results.begin(), results.end(), want.begin() + c.destination);
    }
    if (held > 1) ++joined;
    for (int s = 0; s < held; ++s) units += held > 1 && commands[s].rhs_bytes && commands[s].rhs_bytes < commands[s].bytes;
    for (int s = 1; s < held; ++s) {
      registers += commands[s].lhs == commands[s - 1].destination;
      for (int r = 0; r < s; ++r) revisits += commands[s].destination == commands[r].lhs;
    }
    // The fused kernel: threads one after another, upwards, downwards and shuffled, each taking its elements (one or two)
    // through all commands; the previous result stays with the thread.
    for (int order = 0; order < 3; ++order)
      for (int per = 1; per <= 2; ++per) {
        std::vector<int> threads;
        for (int e = 0; e < bytes; e += per) threads.push_back(e);
        if (order == 1) std::reverse(threads.begin(), threads.end());
        if (order == 2) std::shuffle(threads.begin(), threads.end(), random);
        std::vector<uint8_t> got = memory;
        for (int first : threads) {
          uint8_t value[2] = {0, 0}, b[2];
          for (int s = 0; s < held; ++s) {
            const ChainOperands &c = commands[s];
            const bool carried = s > 0 && c.lhs == commands[s - 1].destination;
            for (int e = 0; e < per && first + e < bytes; ++e) {
              if (!carried) value[e] = got[c.lhs + first + e];
              b[e] = second_operand(c, got, first + e);
            }
            for (int e = 0; e < per && first + e < bytes; ++e) got[c.destination + first + e] = value[e] = evaluate(value[e], b[e], s);
          }
        }
        expect(got == want, "a chain's result depends on its threads");
      }
  }
  expect(joined > 1000 && units > 1000 && revisits > 1000 && registers > 1000, "the chains drawn miss a case");
}

int main() {
  check_copies();
  check_chains();
  printf(failures ? "FAILED %d\n" : "PASS\n", failures);
  return failures != 0;
}
