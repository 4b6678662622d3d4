// Host check of the storage walk (csrc/storage_walk.cuh) against the row-major-to-physical map: every logical element is
// visited once, at the same place of source and destination, and no padding element is.
#include <random>
#include <vector>

#include "../../vibe_compiler_b200/csrc/storage_walk.cuh"

using namespace wb200;

static LayoutMap map_of(int format, int layout, const std::vector<uint64_t> &shape) {
  wb200_tensor_desc d{};
  d.format = static_cast<uint8_t>(format); d.layout = static_cast<uint8_t>(layout); d.rank = static_cast<uint8_t>(shape.size());
  for (size_t i = 0; i < shape.size(); ++i) d.shape[i] = shape[i];
  LayoutMap map;
  if (make_layout_map(d, &map, nullptr) != WB200_OK) { printf("layout refused\n"); exit(2); }
  return map;
}

static int failures = 0;
static void expect(bool ok, const char *what, const std::vector<uint64_t> &shape, int64_t at) {
  if (ok) return;
  if (++failures < 10) {
    printf("%s at %lld, shape", what, static_cast<long long>(at));
    for (uint64_t n : shape) printf(" %llu", static_cast<unsigned long long>(n));
    printf("\n");
  }
}

// Every group of a small tensor.
static void check_all(int from, int to, int layout, const std::vector<uint64_t> &shape) {
  const LayoutMap src = map_of(from, layout, shape), dst = map_of(to, layout, shape);
  const StorageWalk w = storage_walk(src, dst);
  std::vector<int64_t> place(src.physical_elements, -1);   // source element -> destination element
  auto visit = [&](int64_t s, int64_t d, uint32_t valid) {
    for (int e = 0; e < 8; ++e)
      if (valid >> e & 1u) {
        expect(s + e < src.physical_elements && place[s + e] < 0, "visited twice or out of range", shape, s + e);
        if (s + e < src.physical_elements) place[s + e] = d + e;
      }
  };
  for (int64_t first = 0; first < 3; ++first) walk_groups(w, first, 3, visit);   // as three threads would
  for (int64_t i = 0; i < src.element_count; ++i) {
    const int64_t at = physical_index(src, i);
    expect(place[at] == physical_index(dst, i), "wrong or missing element", shape, i);
    place[at] = -1;
  }
  for (int64_t at = 0; at < src.physical_elements; ++at) expect(place[at] < 0, "padding visited", shape, at);
}

// Groups are spread over threads across the slices: a thread per group as long as the machine has room for them.
static void check_threads(int layout, const std::vector<uint64_t> &shape) {
  const LayoutMap map = map_of(WB200_BF16, layout, shape);
  const int64_t groups = map.physical_elements / 8, threads = 256ll * walk_blocks(storage_walk(map, map), 256);
  expect(threads >= (groups < 256 * 148 * 32 ? map.element_count / 8 : 256 * 148 * 32), "too few threads", shape, threads);
}

// Samples of a tensor too large to hold.
static void check_some(int layout, const std::vector<uint64_t> &shape) {
  const LayoutMap map = map_of(WB200_BF16, layout, shape);
  const StorageWalk w = storage_walk(map, map);
  expect(!w.dense, "not a padded tensor", shape, 0);
  std::mt19937_64 rng(7);
  for (int n = 0; n < 20000; ++n) {
    const int64_t i = static_cast<int64_t>(rng() % static_cast<uint64_t>(map.element_count)), at = physical_index(map, i) % map.outer_slice_stride;
    expect(walk_valid(w, at / 8 * 8) >> (at % 8) & 1u, "element missed", shape, i);
    const int64_t channel = map.shape[map.rank - 1] - 1, row = i / map.shape[map.rank - 1];   // the element behind a row's last channel
    const int64_t behind = physical_index(map, row * map.shape[map.rank - 1] + channel) % map.outer_slice_stride + 1;
    if (channel % 64 != 63 && (map.c0 == 0 || (channel - map.cx_blocks * 64) + 1 < map.c0))
      expect(!(walk_valid(w, behind / 8 * 8) >> (behind % 8) & 1u), "padding taken", shape, behind);
  }
}

int main() {
  const int formats[3] = {WB200_BF16, WB200_F16, WB200_F32};
  const std::vector<std::vector<uint64_t>> shapes = {{1}, {7}, {64}, {97}, {3, 5}, {5, 66}, {7, 97}, {33, 64}, {3, 130}, {2, 3, 65}, {9, 1, 64}, {9, 1, 3},
                                                     {17, 2, 100}, {3, 2, 5, 129}, {40, 1, 1, 33}, {2, 3, 2, 2, 68}, {0, 5}, {3, 0}, {0, 2, 5}};
  for (int layout : {WB200_LAYOUT_TENSOR, WB200_LAYOUT_NTENSOR, WB200_LAYOUT_CX, WB200_LAYOUT_NCX})
    for (const auto &shape : shapes)
      for (int from : formats)
        for (int to : formats) check_all(from, to, layout, shape);
  for (const auto &shape : std::vector<std::vector<uint64_t>>{{4096, 1, 64}, {4096, 1, 40}, {512, 7, 97}, {1, 1 << 20, 3}, {1 << 20, 1, 130}})
    check_threads(WB200_LAYOUT_NCX, shape);
  const uint64_t outer = 1ull << 26;   // 64 * outer passes 32 bits
  check_some(WB200_LAYOUT_CX, {outer - 1, 130});
  check_some(WB200_LAYOUT_CX, {outer, 130});
  check_some(WB200_LAYOUT_CX, {outer + 3, 200});
  check_some(WB200_LAYOUT_NCX, {2, outer, 67});
  check_some(WB200_LAYOUT_CX, {2, (1ull << 33) + 5});
  printf(failures ? "FAILED %d\n" : "PASS\n", failures);
  return failures != 0;
}
