// A walk over physical storage in groups of eight elements, for commands whose operands are placed alike: linear layouts,
// and Cx / NCx tensors of one shape (channel blocks of 64, then the aligned tail; slices padded to bank lines). The
// alternative, an element per thread through the row-major-to-physical map, spends its time on 64-bit divisions and moves
// two or four bytes per access (a 256 x 520 Cx convert took 8 us).
#pragma once

#include "common.cuh"

namespace wb200 {

struct StorageWalk {
  int64_t units;                  // groups in all: a thread takes them one by one, whichever slice they belong to
  int dense;                      // every physical element is a logical one (no padding): `count` consecutive elements
  int64_t count;
  int64_t slices;                 // else: NCx leading slices,
  int64_t groups;                 //   groups of a slice,
  int64_t src_stride, dst_stride; //   elements between slices,
  int64_t full;                   //   elements of a slice's full channel blocks,
  int64_t used;                   //   elements of a slice before its end padding,
  int64_t block_elements;         //   elements of a channel block (outer extent x 64),
  int64_t channels;               //   logical channels,
  uint32_t keep, tail;            //   logical channels of the tail, width of the tail
};

// `src` and `dst` describe tensors of one shape and layout (their formats, and so their slice strides, may differ).
inline StorageWalk storage_walk(const LayoutMap &src, const LayoutMap &dst) {
  StorageWalk w{};
  w.dense = src.physical_elements == src.element_count && dst.physical_elements == dst.element_count;
  w.count = src.element_count;
  w.units = (w.count + 7) / 8;
  if (w.dense) return w;
  const bool sliced = src.layout == WB200_LAYOUT_NCX && src.rank > 1;
  w.slices = sliced ? src.shape[0] : 1;
  w.src_stride = src.outer_slice_stride;
  w.dst_stride = dst.outer_slice_stride;
  w.block_elements = src.block_outer_elements * src.c_block;
  w.channels = src.shape[src.rank - 1];
  w.tail = static_cast<uint32_t>(src.c0);
  w.keep = w.tail ? static_cast<uint32_t>(w.channels - src.cx_blocks * src.c_block) : 0u;
  w.full = src.cx_blocks * src.block_outer_elements * src.c_block;
  w.used = w.full + src.block_outer_elements * src.c0;
  w.groups = (w.used + 7) / 8;
  w.units = w.slices * w.groups;
  return w;
}

// Blocks of `threads` that give every group a thread, up to 32 per SM of 148.
inline int walk_blocks(const StorageWalk &w, int threads) {
  const int64_t blocks = (w.units + threads - 1) / threads;
  return static_cast<int>(blocks < 1 ? 1 : blocks > 148 * 32 ? 148 * 32 : blocks);
}

// Bit e: element `offset` + e of a slice is a logical element.
__host__ __device__ inline uint32_t walk_valid(const StorageWalk &w, int64_t offset) {
  if (offset < w.full) {
    // 64-bit divisions only where a slice's blocks need them; block_elements is at most `full`
    const int64_t block = w.full < (1ll << 32) ? static_cast<uint32_t>(offset) / static_cast<uint32_t>(w.block_elements) : offset / w.block_elements;
    const int64_t left = w.channels - (block * 64 + (offset & 63));
    return left >= 8 ? 0xffu : left <= 0 ? 0u : (1u << static_cast<int>(left)) - 1u;
  }
  uint32_t mask = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (offset + e < w.used && static_cast<uint32_t>((offset - w.full + e) & (w.tail - 1)) < w.keep) mask |= 1u << e;   // the width is a power of two
  return mask;
}

// Calls visit(src element, dst element, valid mask) for the groups `first`, `first` + `stride`, ...
#pragma nv_exec_check_disable   // a kernel's visitor is device code
template <typename Visit>
__host__ __device__ inline void walk_groups(const StorageWalk &w, int64_t first, int64_t stride, Visit &&visit) {
  for (int64_t u = first; u < w.units; u += stride) {
    if (w.dense) {
      const int64_t left = w.count - u * 8;
      visit(u * 8, u * 8, left >= 8 ? 0xffu : (1u << static_cast<int>(left)) - 1u);
      continue;
    }
    int64_t slice = 0, at = u * 8;
    if (w.slices > 1) {
      slice = w.units < (1ll << 32) ? static_cast<uint32_t>(u) / static_cast<uint32_t>(w.groups) : u / w.groups;
      at = (u - slice * w.groups) * 8;
    }
    const uint32_t valid = walk_valid(w, at);
    if (valid) visit(slice * w.src_stride + at, slice * w.dst_stride + at, valid);
  }
}

}  // namespace wb200
