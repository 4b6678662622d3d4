// Which commands of a replayed Tile program may share a launch: host rules without device types, so that a host program can
// compare them with the order of the commands (tests/host_cpp/replay_rules_check.cpp).
#pragma once
#include <cstdint>

namespace wb200 {

// Bytes [begin, end) of an image that a command reads or writes. In a command of several Tiles they are Tile 0's, and Tile t's
// lie t * step behind them: each Tile has a scratch-pad image of its own (step 0), DDR is common to all.
struct ReplayRange {
  const void *image;
  uint64_t begin, end;
  int64_t step;
};

// Does any of the Tiles find its two ranges overlapping? Ranges of one step keep the distance that Tile 0's have.
inline bool ranges_touch(const ReplayRange &a, const ReplayRange &b, uint32_t tiles) {
  if (a.image != b.image) return false;
  for (uint64_t t = 0; t < (a.step == b.step ? 1u : tiles); ++t) {
    const uint64_t a_shift = t * static_cast<uint64_t>(a.step), b_shift = t * static_cast<uint64_t>(b.step);   // modulo 2^64
    if (a.begin + a_shift < b.end + b_shift && b.begin + b_shift < a.end + a_shift) return true;
  }
  return false;
}

// A DMA command as the rule below sees it.
struct ReplayCopy {
  ReplayRange source, destination;
  uint32_t unit;   // bytes a thread of the launch moves at once
  bool load;       // DDR to scratch-pad
};

// May `next` be copied in one launch with the commands held before it, in no order? Neither reads or writes what the other
// writes, for any Tile. Loads and stores do not mix: what one Tile stores to DDR may be what another one loads.
inline bool copies_join(const ReplayCopy *held, int count, const ReplayCopy &next, uint32_t tiles) {
  for (int i = 0; i < count; ++i)
    if (held[i].unit != next.unit || held[i].load != next.load || ranges_touch(next.destination, held[i].source, tiles) ||
        ranges_touch(next.destination, held[i].destination, tiles) || ranges_touch(next.source, held[i].destination, tiles))
      return false;
  return true;
}

// The operands of an elementwise command of `bytes` bytes of results. The second one has rhs_bytes: none or an immediate (0), a
// vector like the first (`bytes`) or a shorter unit that is repeated.
struct ChainOperands {
  uint64_t lhs, rhs, destination, bytes, rhs_bytes;
};

// May a chain store to [destination, + bytes) and read [address, + read)? Equally long ranges, when they coincide or do not
// touch: a thread of the fused kernel owns the same elements of every vector, so only a shifted overlap would cross threads.
// A repeated unit, which is shorter, is read by all threads and must not be stored to.
inline bool ranges_compatible(uint64_t destination, uint64_t bytes, uint64_t address, uint64_t read) {
  return (destination == address && read == bytes) || destination + bytes <= address || address + read <= destination;
}

// A command whose own operands rule it out of every chain.
inline bool chain_refuses(const ChainOperands &c) {
  return !ranges_compatible(c.destination, c.bytes, c.lhs, c.bytes) || (c.rhs_bytes && !ranges_compatible(c.destination, c.bytes, c.rhs, c.rhs_bytes));
}

// May `next` follow the held commands, of its format and length, in one launch? Nothing that either stores is read, or stored
// to, by other threads.
inline bool chain_extends(const ChainOperands *held, int count, const ChainOperands &next) {
  if (chain_refuses(next)) return false;
  for (int s = 0; s < count; ++s) {
    const ChainOperands &c = held[s];
    if (!ranges_compatible(next.destination, next.bytes, c.lhs, c.bytes) || !ranges_compatible(next.destination, next.bytes, c.destination, c.bytes) ||
        (c.rhs_bytes && !ranges_compatible(next.destination, next.bytes, c.rhs, c.rhs_bytes)) ||
        !ranges_compatible(c.destination, c.bytes, next.lhs, next.bytes) ||
        (next.rhs_bytes && !ranges_compatible(c.destination, c.bytes, next.rhs, next.rhs_bytes)))
      return false;
  }
  return true;
}

}  // namespace wb200
