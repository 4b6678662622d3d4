// Flash-decoding (split-KV attention for query length 1, grouped queries) for sm_100a.
//
// Arithmetic follows the reference's online-attention materialisation:
//   per KV tile   lib/Wafer/Transforms/Linalg/OnlineAttentionDecomposition.cpp:568-594
//   state merge   lib/Wafer/Transforms/Linalg/OnlineAttentionMaterialization.cpp:264-373
//   finalize      lib/Wafer/Transforms/Linalg/OnlineAttentionMaterialization.cpp:196-262
//   fold order    lib/Wafer/Transforms/Linalg/SpatialRegionMaterialization.cpp:2420-2433 (ascending)
// exp is the target's ExpLp, exp2(x * log2e) in f32
// (lib/Wafer/Simulator/Reference/ManagedReferenceTargetModel.cpp:265-270).
//
// fd_partial_kernel: the keys of a (batch, kv head) are cut over `cluster * splits` CTAs. Each of a CTA's 4 warps streams
// its own contiguous quarter of the CTA's KV interval through a private 3-deep cp.async ring of 16-row
// tiles (128-bit coalesced copies, XOR-swizzled rows), computes S = Q K^T and acc += P V with
// mma.sync m16n8k16 on the group's query heads (rows padded to 16) and carries (m, l, acc) in
// registers. Warps then fold their states in ascending KV order through shared memory; the CTAs of a cluster hand
// theirs to the cluster's first CTA through distributed shared memory. With one cluster per (batch, kv head) that CTA
// finalizes; otherwise it writes one (acc[D], m, l) record, and the cluster that finishes last folds the records of the
// group's query heads and finalizes. A decode step is one launch either way.
// The kernel is HBM-bound for long caches: algorithmic bytes per launch are the K and V bytes of the visible keys, read
// exactly once. Short ones are a latency chain (launch, first tile, merge), which the cluster merge shortens: no record
// goes through global memory and nothing is fenced or counted.
// Measured per launch (bf16, launches replayed back to back as a graph, caches rotated through 400 MB), two launches with a
// combine kernel -> this form: 28/4 heads, 1 x 1537 keys 8.3 -> 6.7 us; 32/8 heads, 8 x 4000 keys 28.7 -> 25.1 us (20.0 at the
// copy rate), 33 x 900 keys 29.1 -> 20.8 us (18.6), 64 x 333 keys 30.0 -> 17.0 us (13.3), 1 x 1 Mi keys 629 -> 600 us.
#include "kernels.h"
#include "ptx_sm100.cuh"

namespace wb200 {
namespace {

constexpr int kD = 128;            // head dimension
constexpr int kTileRows = 16;      // KV rows per warp tile
constexpr int kWarps = 4;
constexpr int kStagesFd = 3;
constexpr int kTileBytes = kTileRows * kD * 2;  // 4 KiB for K, same for V
constexpr int kRecord = kD + 2;    // acc[D], m, l
constexpr int kSmemRecord = kD + 4;   // the same in shared memory, rows 16-byte aligned
constexpr int kMaxGroup = 16;      // query heads per KV head
constexpr int kFdSmemBytes = kWarps * kStagesFd * 2 * kTileBytes;
// The rings are reused for the warps' records and, behind them, the CTA's merged record.
constexpr int kMergedOffset = kWarps * kMaxGroup * kSmemRecord;   // floats
static_assert((kMergedOffset + kMaxGroup * kSmemRecord) * 4 <= kFdSmemBytes, "merge records must fit the rings");

__device__ __forceinline__ float exp_lp(float x) { return exp2f(x * 0x1.715476p+0f); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
template <bool kBf16>
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBf16) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}
template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (kBf16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
  }
}

struct FdParams {
  int batch, q_heads, kv_heads, group;
  int kv_len;         // rows physically present per (batch, kv head)
  int kv_visible;     // keys [0, kv_visible) are visible
  int splits;         // records per query head = clusters per (batch, kv head)
  int cluster;        // CTAs per cluster
  int rows_per_cta, rows_per_warp;
  float scale;
  const uint16_t *q, *k, *v;
  float *partials;    // [batch, q_heads, splits, kRecord]
};

// What the last CTA of a (batch, kv head) to finish stage 1 does with the records: fold, then write the outputs or the
// un-finalized state (kTailLocal), or exchange the state with the other ranks first (kTailExchange, fd_exchange_rows: the
// exchange buffers of all ranks and this rank's epoch words).
enum { kTailNone = 0, kTailLocal = 1, kTailExchange = 2 };
constexpr int kMaxExchangeRanks = 16;
struct FdTailParams {
  int rank, world;
  float *peer[kMaxExchangeRanks];    // exchange buffers of all ranks, [rank] = this rank's own
  unsigned int *epoch;               // this rank's {epoch, finished rows}, zero-initialised
  unsigned int *arrivals;            // [batch * kv_heads] of fd_arrive(), zero-initialised
  int out_format, zero_fully_masked;
  void *out;
  float *lse, *row_max, *row_sum;
  float *state_out;                  // kTailLocal: non-null = write the merged state here instead of out / lse
  int *status;
};
template <int kRowsAtOnce>
__device__ void fd_exchange_rows(const FdTailParams &x, const float *records, int splits, int first_row, int row_count, int rows_total);

__device__ __forceinline__ void fd_merge_right(float &m, float &l, float4 &a, float m_right, float l_right, const float4 &a_right) {
  const float m_new = fmaxf(m, m_right);
  const float m_exp = (m_new == -INFINITY) ? 0.f : m_new;
  const float scale_left = exp_lp(m - m_exp), scale_right = exp_lp(m_right - m_exp);
  l = l * scale_left + l_right * scale_right;
  a.x = a.x * scale_left + a_right.x * scale_right;
  a.y = a.y * scale_left + a_right.y * scale_right;
  a.z = a.z * scale_left + a_right.z * scale_right;
  a.w = a.w * scale_left + a_right.w * scale_right;
  m = m_new;
}
// Four consecutive floats of a record (records are 130 floats long: 8-byte, not 16-byte, aligned), read past L1.
__device__ __forceinline__ float4 ldcg_quad(const float *address) {
  const float2 lo = __ldcg(reinterpret_cast<const float2 *>(address)), hi = __ldcg(reinterpret_cast<const float2 *>(address + 2));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}
// Fold of a row's split records by one warp (lane: four head dimensions). The common exponent reference of all records is
// their maximum, so the weights come from one pass over the (m, l) pairs with a lane per record, and the accumulators are
// summed in ascending record order with independent loads (eight records in flight). Against the pairwise left fold this
// takes the chain of exponentials out of the loop; a one-sequence decode has the fold on its critical path.
__device__ __forceinline__ void fd_fold_records(const float *rec, int records, int lane, float &m, float &l, float4 &a) {
  float top = -INFINITY;
  for (int i = lane; i < records; i += 32) top = fmaxf(top, __ldcg(rec + static_cast<size_t>(i) * kRecord + kD));
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
  const float m_exp = (top == -INFINITY) ? 0.f : top;
  float sum = 0.f;
  a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int base = 0; base < records; base += 32) {
    float weight = 0.f;
    if (base + lane < records) {
      const float2 ml = __ldcg(reinterpret_cast<const float2 *>(rec + static_cast<size_t>(base + lane) * kRecord + kD));
      weight = exp_lp(ml.x - m_exp);
      sum = fmaf(ml.y, weight, sum);
    }
    const int count = min(32, records - base);
    const float *src = rec + static_cast<size_t>(base) * kRecord + 4 * lane;
    auto add = [&](int i, const float4 &right) {
      const float w = __shfl_sync(0xffffffffu, weight, i);
      a.x = fmaf(right.x, w, a.x); a.y = fmaf(right.y, w, a.y);
      a.z = fmaf(right.z, w, a.z); a.w = fmaf(right.w, w, a.w);
    };
    int i = 0;
    for (; i + 8 <= count; i += 8) {
      float4 right[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) right[u] = ldcg_quad(src + static_cast<size_t>(i + u) * kRecord);
#pragma unroll
      for (int u = 0; u < 8; ++u) add(i + u, right[u]);
    }
    for (; i < count; ++i) add(i, ldcg_quad(src + static_cast<size_t>(i) * kRecord));
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  m = top;
  l = sum;
}
// Finalizes a row: out = acc / l with one narrowing, log-sum-exp and the carried state; lane = four head dimensions.
__device__ __forceinline__ void fd_write_row(const FdTailParams &x, int row, int lane, float m, float l, const float4 &a) {
  float coefficient = 1.0f / l;
  if (x.zero_fully_masked && l == 0.f) coefficient = 0.f;
  const float value[4] = {a.x * coefficient, a.y * coefficient, a.z * coefficient, a.w * coefficient};
  if (x.out_format == WB200_F32) {
    *(reinterpret_cast<float4 *>(x.out) + static_cast<size_t>(row) * (kD / 4) + lane) = make_float4(value[0], value[1], value[2], value[3]);
  } else {
    uint32_t bits[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) bits[i] = narrow_bits(value[i], x.out_format);
    if ((reinterpret_cast<uintptr_t>(x.out) & 7u) == 0) {
      *(reinterpret_cast<uint2 *>(x.out) + static_cast<size_t>(row) * (kD / 4) + lane) = make_uint2(bits[0] | (bits[1] << 16), bits[2] | (bits[3] << 16));
    } else {
      uint16_t *dst = reinterpret_cast<uint16_t *>(x.out) + static_cast<size_t>(row) * kD + 4 * lane;
#pragma unroll
      for (int i = 0; i < 4; ++i) dst[i] = static_cast<uint16_t>(bits[i]);
    }
  }
  if (lane == 0) {
    if (x.lse) x.lse[row] = (l == 0.f) ? -INFINITY : m + logf(l);
    if (x.row_max) x.row_max[row] = m;
    if (x.row_sum) x.row_sum[row] = l;
  }
}
// The complete state of a row: un-finalized to `state_out`, or finalized.
__device__ __forceinline__ void fd_deliver_row(const FdTailParams &x, int row, int lane, float m, float l, const float4 &a) {
  if (!x.state_out) { fd_write_row(x, row, lane, m, l, a); return; }
  float *state = x.state_out + static_cast<size_t>(row) * kRecord;
  state[4 * lane] = a.x; state[4 * lane + 1] = a.y; state[4 * lane + 2] = a.z; state[4 * lane + 3] = a.w;
  if (lane == 0) { state[kD] = m; state[kD + 1] = l; }
}
// Rows [first_row, first_row + row_count) by one CTA, a warp per row.
__device__ void fd_local_rows(const FdTailParams &x, const float *records, int splits, int first_row, int row_count) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = warp; r < row_count; r += kWarps) {
    const int row = first_row + r;
    float m, l;
    float4 a;
    fd_fold_records(records + static_cast<size_t>(row) * splits * kRecord, splits, lane, m, l, a);
    fd_deliver_row(x, row, lane, m, l, a);
  }
}
// Counts the arrival of cluster `index` of a (batch, kv head) unit's `clusters`; true for the last one. The shares of a launch
// add up to 2^32, that is to nothing, and are added whatever the word holds: the word is back at zero after every launch, also
// after launches that wrongly overlapped on one scratch, which can spoil each other's results but not those of later ones.
// The sum is zero only at the last arrival: the others give 1 each, the first cluster 1 - clusters.
__device__ __forceinline__ bool fd_arrive(unsigned int *word, unsigned int index, unsigned int clusters) {
  const unsigned int share = index == 0u ? 1u - clusters : 1u;
  return atomicAdd(word, share) + share == 0u;
}
// Swizzled byte offset of 16-byte chunk `c` of row `r` inside a 16 x 256-byte tile.
__device__ __forceinline__ uint32_t tile_offset(int r, int c) {
  return static_cast<uint32_t>(r * 256 + ((c ^ (r & 7)) << 4));
}

// kNarrow: groups of at most 8 query heads. Scores are computed with the heads as the MMA rows either way (C fragment: head
// g, keys 2t, 2t + 1), which is the B fragment of the transposed PV product out^T [d, heads] += V^T P^T: 8 products per
// 16 keys instead of 16, half the accumulators, and one softmax row per lane instead of two. A CTA's rate is set by the
// chain of a tile (scores, maximum, exponentials, products), so this is what a cache that does not fill the chip gains from.
template <bool kBf16, int kTail, bool kNarrow>
__global__ void __launch_bounds__(kWarps * 32, 2) fd_partial_kernel(const FdParams p, const FdTailParams tail) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int hk = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;

  // This warp's KV interval.
  const int warp_begin = static_cast<int>(blockIdx.x) * p.rows_per_cta + warp * p.rows_per_warp;
  int warp_end = warp_begin + p.rows_per_warp;
  if (warp_end > p.kv_visible) warp_end = p.kv_visible;
  const int tiles = warp_end > warp_begin ? (warp_end - warp_begin + kTileRows - 1) / kTileRows : 0;

  const size_t head_offset = (static_cast<size_t>(b) * p.kv_heads + hk) * static_cast<size_t>(p.kv_len) * kD;
  const uint16_t *k_base = p.k + head_offset;
  const uint16_t *v_base = p.v + head_offset;
  uint8_t *ring = smem + warp * (kStagesFd * 2 * kTileBytes);
  const uint32_t ring_addr = static_cast<uint32_t>(__cvta_generic_to_shared(ring));

  auto issue_tile = [&](int tile, int slot) {
    if (tile < tiles) {
      const int row0 = warp_begin + tile * kTileRows;
      const uint32_t k_dst = ring_addr + slot * (2 * kTileBytes);
      const uint32_t v_dst = k_dst + kTileBytes;
#pragma unroll
      for (int i = 0; i < (kTileRows * 16) / 32; ++i) {
        const int idx = i * 32 + lane;
        const int r = idx >> 4, c = idx & 15;
        const int row = row0 + r;
        const bool in_range = row < warp_end;   // rows behind the visible keys are zero-filled, not read
        const size_t src = static_cast<size_t>(in_range ? row : 0) * kD + c * 8;
        cp_async16(k_dst + tile_offset(r, c), k_base + src, in_range ? 16u : 0u);
        cp_async16(v_dst + tile_offset(r, c), v_base + src, in_range ? 16u : 0u);
      }
    }
    cp_async_commit();
  };

  constexpr int kHalves = kNarrow ? 1 : 2;        // softmax rows per lane: heads g (and g + 8)
  constexpr int kAccs = kNarrow ? kD / 16 : kD / 8;   // accumulator fragments: d blocks of 16 x 8 heads, or 16 heads x d blocks of 8
  float m_run[kHalves], l_run[kHalves];               // l_run: this lane's share of the row sum
#pragma unroll
  for (int h = 0; h < kHalves; ++h) { m_run[h] = -INFINITY; l_run[h] = 0.f; }
  float acc[kAccs][4];
#pragma unroll
  for (int j = 0; j < kAccs; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;

  pdl_wait();   // everything this kernel reads may come from the kernel before it
#pragma unroll
  for (int s = 0; s < kStagesFd; ++s) issue_tile(s, s);
  pdl_launch_dependents();
  // The group's query rows as A fragments, straight from global memory behind the first tiles' copies (rows of the 16 that
  // the group does not fill are zero).
  uint32_t q_frag[kD / 16][4];
  {
    const uint32_t *q_src = reinterpret_cast<const uint32_t *>(p.q + (static_cast<size_t>(b) * p.q_heads + static_cast<size_t>(hk) * p.group) * kD);
    const bool lo = g < p.group, hi = g + 8 < p.group;
    const uint32_t *row_lo = q_src + g * (kD / 2) + t, *row_hi = row_lo + 8 * (kD / 2);
#pragma unroll
    for (int ks = 0; ks < kD / 16; ++ks) {
      q_frag[ks][0] = lo ? row_lo[ks * 8] : 0u;
      q_frag[ks][1] = hi ? row_hi[ks * 8] : 0u;
      q_frag[ks][2] = lo ? row_lo[ks * 8 + 4] : 0u;
      q_frag[ks][3] = hi ? row_hi[ks * 8 + 4] : 0u;
    }
  }

  for (int tile = 0; tile < tiles; ++tile) {
    cp_async_wait<kStagesFd - 1>();
    __syncwarp();
    const uint32_t k_src = ring_addr + (tile % kStagesFd) * (2 * kTileBytes);
    const uint32_t v_src = k_src + kTileBytes;
    const int row0 = warp_begin + tile * kTileRows;

    // S = Q K^T for 16 keys: two n-tiles of 8 keys, even and odd k-steps accumulated apart (four short chains).
    float part[2][2][4] = {};
#pragma unroll
    for (int ks = 0; ks < kD / 16; ++ks) {
      const int mi = lane >> 3;
      const int r = (mi >> 1) * 8 + (lane & 7);
      const int c = 2 * ks + (mi & 1);
      uint32_t bfrag[4];
      ldmatrix_x4(k_src + tile_offset(r, c), bfrag);
      mma_16816<kBf16>(part[ks & 1][0], q_frag[ks], bfrag[0], bfrag[1]);
      mma_16816<kBf16>(part[ks & 1][1], q_frag[ks], bfrag[2], bfrag[3]);
    }
    // score region: scale, then mask keys outside the visible interval.
    const int key0 = row0 + 2 * t;
    float alpha[kHalves];
    float pr[kHalves][4];   // [row half][key 2t, 2t+1, 8+2t, 8+2t+1]
#pragma unroll
    for (int h = 0; h < kHalves; ++h) {
      float sc[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sc[i] = (part[0][i >> 1][2 * h + (i & 1)] + part[1][i >> 1][2 * h + (i & 1)]) * p.scale;
        if (key0 + (i >> 1) * 8 + (i & 1) >= warp_end) sc[i] = -INFINITY;
      }
      float tile_max = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
      tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 1));
      tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 2));
      const float m_new = fmaxf(tile_max, m_run[h]);
      const float m_exp = (m_new == -INFINITY) ? 0.f : m_new;
      alpha[h] = exp_lp(m_run[h] - m_exp);
      float row_sum = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        pr[h][i] = exp_lp(sc[i] - m_exp);
        row_sum += pr[h][i];
      }
      l_run[h] = l_run[h] * alpha[h] + row_sum;
      m_run[h] = m_new;
    }
    // Probabilities are rounded to the storage type of V at the PV input.
    if constexpr (kNarrow) {
      const uint32_t p_lo = pack2<kBf16>(pr[0][0], pr[0][1]), p_hi = pack2<kBf16>(pr[0][2], pr[0][3]);
      const float alpha0 = __shfl_sync(0xffffffffu, alpha[0], 8 * t), alpha1 = __shfl_sync(0xffffffffu, alpha[0], 8 * t + 4);   // heads 2t, 2t + 1
#pragma unroll
      for (int j = 0; j < kAccs; ++j) {
        const int mi = lane >> 3;
        const int r = (mi >> 1) * 8 + (lane & 7);
        const int c = 2 * j + (mi & 1);
        uint32_t vfrag[4];
        ldmatrix_x4_trans(v_src + tile_offset(r, c), vfrag);
        acc[j][0] *= alpha0; acc[j][1] *= alpha1; acc[j][2] *= alpha0; acc[j][3] *= alpha1;
        mma_16816<kBf16>(acc[j], vfrag, p_lo, p_hi);
      }
    } else {
      const uint32_t p_frag[4] = {pack2<kBf16>(pr[0][0], pr[0][1]), pack2<kBf16>(pr[kHalves - 1][0], pr[kHalves - 1][1]),
                                  pack2<kBf16>(pr[0][2], pr[0][3]), pack2<kBf16>(pr[kHalves - 1][2], pr[kHalves - 1][3])};
#pragma unroll
      for (int j = 0; j < kAccs; ++j) {
        acc[j][0] *= alpha[0]; acc[j][1] *= alpha[0];
        acc[j][2] *= alpha[kHalves - 1]; acc[j][3] *= alpha[kHalves - 1];
      }
#pragma unroll
      for (int j = 0; j < kAccs; j += 2) {
        const int mi = lane >> 3;
        const int r = (mi & 1) * 8 + (lane & 7);
        const int c = j + (mi >> 1);
        uint32_t vfrag[4];
        ldmatrix_x4_trans(v_src + tile_offset(r, c), vfrag);
        mma_16816<kBf16>(acc[j], p_frag, vfrag[0], vfrag[1]);
        mma_16816<kBf16>(acc[j + 1], p_frag, vfrag[2], vfrag[3]);
      }
    }
    __syncwarp();   // every lane has read the slot
    issue_tile(tile + kStagesFd, tile % kStagesFd);
  }
  cp_async_wait<0>();
#pragma unroll
  for (int h = 0; h < kHalves; ++h) {
    l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 1);
    l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 2);
  }
  __syncthreads();  // every warp is done with its ring; reuse it for the merge records

  float *records = reinterpret_cast<float *>(smem);  // [warp][kMaxGroup][kSmemRecord]
  {
    float *mine = records + warp * (kMaxGroup * kSmemRecord);
    if constexpr (kNarrow) {
#pragma unroll
      for (int j = 0; j < kAccs; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (2 * t + (i & 1) < p.group) mine[(2 * t + (i & 1)) * kSmemRecord + j * 16 + g + 8 * (i >> 1)] = acc[j][i];
    }
#pragma unroll
    for (int h = 0; h < kHalves; ++h) {
      const int head = g + 8 * h;
      if (head < p.group) {
        if constexpr (!kNarrow) {
#pragma unroll
          for (int j = 0; j < kAccs; ++j)
            *reinterpret_cast<float2 *>(mine + head * kSmemRecord + j * 8 + 2 * t) = make_float2(acc[j][2 * h], acc[j][2 * h + 1]);
        }
        if (t == 0) *reinterpret_cast<float2 *>(mine + head * kSmemRecord + kD) = make_float2(m_run[h], l_run[h]);
      }
    }
  }
  __syncthreads();
  // Left fold over the warps (ascending KV order): a warp per query head, a lane per four head dimensions.
  float *merged = records + kMergedOffset;           // [kMaxGroup][kSmemRecord]
  const bool first_cta = p.cluster == 1 || cluster_cta_rank() == 0;
  const int cluster_index = p.cluster == 1 ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x) / p.cluster;
  // What becomes of the state of query head `head` once it is complete for the cluster's keys.
  auto deliver = [&](int head, float m, float l, const float4 &a) {
    const int row = b * p.q_heads + hk * p.group + head;
    if (kTail == kTailLocal && p.splits == 1) {
      fd_deliver_row(tail, row, lane, m, l, a);
    } else {
      float *out = p.partials + (static_cast<size_t>(row) * p.splits + cluster_index) * kRecord;
      *reinterpret_cast<float2 *>(out + 4 * lane) = make_float2(a.x, a.y);
      *reinterpret_cast<float2 *>(out + 4 * lane + 2) = make_float2(a.z, a.w);
      if (lane == 0) *reinterpret_cast<float2 *>(out + kD) = make_float2(m, l);
    }
  };
  for (int head = warp; head < p.group; head += kWarps) {
    const float *rec = records + head * kSmemRecord;
    float m = rec[kD], l = rec[kD + 1];
    float4 a = *reinterpret_cast<const float4 *>(rec + 4 * lane);
#pragma unroll
    for (int w = 1; w < kWarps; ++w) {
      const float *right = rec + w * (kMaxGroup * kSmemRecord);
      fd_merge_right(m, l, a, right[kD], right[kD + 1], *reinterpret_cast<const float4 *>(right + 4 * lane));
    }
    if (p.cluster == 1) {
      deliver(head, m, l, a);
    } else {
      *reinterpret_cast<float4 *>(merged + head * kSmemRecord + 4 * lane) = a;
      if (lane == 0) *reinterpret_cast<float2 *>(merged + head * kSmemRecord + kD) = make_float2(m, l);
    }
  }
  if (p.cluster > 1) {
    cluster_sync_all();   // the merged records of the cluster's CTAs are in their shared memory
    if (first_cta) {
      // Fold over the cluster's CTAs with their common maximum as the exponent reference (see fd_fold_records); lane r
      // holds CTA r's (m, l) of the head.
      for (int head = warp; head < p.group; head += kWarps) {
        const uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(merged + head * kSmemRecord));
        float2 ml = make_float2(-INFINITY, 0.f);
        if (lane < p.cluster) ml = ld_cluster_f32x2(cluster_map_shared(local + kD * 4, lane));
        float top = ml.x;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
        const float weight = exp_lp(ml.x - (top == -INFINITY ? 0.f : top));
        float sum = ml.y * weight;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int r = 0; r < p.cluster; ++r) {
          const float4 right = ld_cluster_f32x4(cluster_map_shared(local + 16 * lane, r));
          const float w = __shfl_sync(0xffffffffu, weight, r);
          a.x = fmaf(right.x, w, a.x); a.y = fmaf(right.y, w, a.y);
          a.z = fmaf(right.z, w, a.z); a.w = fmaf(right.w, w, a.w);
        }
        deliver(head, top, sum, a);
      }
    }
    cluster_sync_all();   // no CTA leaves while the first one may read its shared memory
    if (!first_cta) return;
  }
  if (kTail == kTailLocal && p.splits == 1) return;
  if constexpr (kTail != kTailNone) {
    // The cluster that finishes last among those of this (batch, kv head) folds the records of the group's query heads and
    // writes the outputs (with the exchange between the ranks in front of them): the decode step is this one launch.
    __shared__ bool last_of_head;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();      // cumulative over the CTA's record stores, which the barrier ordered before it
      last_of_head = fd_arrive(tail.arrivals + b * p.kv_heads + hk, static_cast<unsigned int>(cluster_index), static_cast<unsigned int>(p.splits));
      __threadfence();
    }
    __syncthreads();
    if (last_of_head) {
      const int first_row = b * p.q_heads + hk * p.group;
      if constexpr (kTail == kTailExchange)
        fd_exchange_rows<kD / 32>(tail, p.partials, p.splits, first_row, p.group, p.batch * p.q_heads);
      else
        fd_local_rows(tail, p.partials, p.splits, first_row, p.group);
    }
  }
}

struct FdCombineParams {
  int rows;            // batch * q_heads
  int records;         // number of records folded per row
  size_t row_stride;   // floats between consecutive rows of one record index
  size_t record_stride;// floats between consecutive records of one row
  const float *records_ptr;
  int out_format;
  int zero_fully_masked;
  void *out;
  float *lse, *row_max, *row_sum;
};

// Merge of the states of sequence shards (wb200_attention_fd_merge): left fold in ascending shard order, one thread per
// head dimension of a row.
__global__ void __launch_bounds__(kD) fd_combine_kernel(const FdCombineParams p) {
  const int row = blockIdx.x, d = threadIdx.x;
  const float *rec = p.records_ptr + row * p.row_stride;
  float m = rec[kD], l = rec[kD + 1], a = rec[d];
  for (int i = 1; i < p.records; ++i) {
    const float *right = rec + i * p.record_stride;
    const float m_right = right[kD], l_right = right[kD + 1], a_right = right[d];
    const float m_new = fmaxf(m, m_right);
    const float m_exp = (m_new == -INFINITY) ? 0.f : m_new;
    const float scale_left = exp_lp(m - m_exp), scale_right = exp_lp(m_right - m_exp);
    l = l * scale_left + l_right * scale_right;
    a = a * scale_left + a_right * scale_right;
    m = m_new;
  }
  float coefficient = 1.0f / l;
  if (p.zero_fully_masked && l == 0.f) coefficient = 0.f;
  const float value = a * coefficient;
  if (p.out_format == WB200_F32)
    reinterpret_cast<float *>(p.out)[static_cast<size_t>(row) * kD + d] = value;
  else
    reinterpret_cast<uint16_t *>(p.out)[static_cast<size_t>(row) * kD + d] =
        static_cast<uint16_t>(narrow_bits(value, p.out_format));
  if (d == 0) {
    if (p.lse) p.lse[row] = (l == 0.f) ? -INFINITY : m + logf(l);
    if (p.row_max) p.row_max[row] = m;
    if (p.row_sum) p.row_sum[row] = l;
  }
}

// Sequence-sharded decode, one shard per GPU: the fold over this GPU's splits, the exchange of the per-head states
// between the GPUs and the final merge in one kernel (one CTA per (batch, query head) row, thread = head dimension).
// Every rank owns an exchange buffer that all ranks can address (peer-mapped memory):
//   states [2][world][rows][kRecord] floats, then flags [2][world][rows] words, both indexed by the parity of an epoch
// that advances by one per call on every rank. A CTA writes its row's state into slot [parity][rank][row] of every
// rank's buffer with plain stores over NVLink, publishes it with a release store of the epoch tag to the matching
// flag, waits (bounded) until the flags of all ranks for its row carry the tag in its own buffer, and folds the world's
// states in ascending rank order - the shard order of the reference's spatial flash-decoding fold
// (lib/Wafer/Transforms/Linalg/SpatialRegionMaterialization.cpp:2420-2433). A rank can run at most one epoch ahead of
// another (its next exchange cannot complete before the other has entered it), so two parities suffice.
__device__ __forceinline__ void st_relaxed_sys(unsigned int *address, unsigned int value) {
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(address), "r"(value) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_sys(const unsigned int *address) {
  unsigned int value;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(value) : "l"(address) : "memory");
  return value;
}

// Rows [first_row, first_row + row_count) of the (batch, query head) rows, by one CTA of kD threads = four warps: a warp
// takes a row, a lane four consecutive head dimensions. Per batch of four rows: fold of the rows' split records in
// ascending order, stores of the states into every rank's buffer, flags, bounded wait for the world's flags, merge in
// ascending rank order, outputs. The rows of a batch travel together, so the NVLink round trip is paid once per batch.
template <int kRowsAtOnce>
__device__ void fd_exchange_rows(const FdTailParams &x, const float *records, int splits, int first_row, int row_count, int rows_total) {
  static_assert(kRowsAtOnce == kD / 32, "one warp per row");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned int epoch = *reinterpret_cast<volatile unsigned int *>(x.epoch);
  const unsigned int parity = epoch & 1u, tag = epoch + 1u;
  const size_t state_floats = static_cast<size_t>(2) * x.world * rows_total * kRecord;
  float *own = x.peer[x.rank];
  for (int base = 0; base < row_count; base += kRowsAtOnce) {
    const int count = row_count - base < kRowsAtOnce ? row_count - base : kRowsAtOnce;
    const int row = first_row + base + warp;
    const bool active = warp < count;
    if (active) {
      // fold this rank's splits (records of other CTAs: read past L1)
      float m, l;
      float4 a;
      fd_fold_records(records + static_cast<size_t>(row) * splits * kRecord, splits, lane, m, l, a);
      // the state into slot [parity][rank][row] of every rank's buffer (records are 130 floats: 8-byte aligned rows)
      const size_t my_slot = (static_cast<size_t>(parity) * x.world + x.rank) * rows_total + row;
      for (int r = 0; r < x.world; ++r) {
        float *dst = x.peer[r] + my_slot * kRecord;
        *reinterpret_cast<float2 *>(dst + 4 * lane) = make_float2(a.x, a.y);
        *reinterpret_cast<float2 *>(dst + 4 * lane + 2) = make_float2(a.z, a.w);
        if (lane == 0) *reinterpret_cast<float2 *>(dst + kD) = make_float2(m, l);
      }
    }
    __syncthreads();   // the rows are written before they are published
    // One thread per (row, peer): a system-scope fence (cumulative over the rows' stores, which the barrier ordered
    // before it) and then the flag; the fences of the peers run side by side. Then the bounded wait for every rank's
    // flag of every row, again one thread per (row, rank).
    for (int j = tid; j < count * x.world; j += kD) {
      const int flag_row = first_row + base + j / x.world, peer = j % x.world;
      const size_t my_slot = (static_cast<size_t>(parity) * x.world + x.rank) * rows_total + flag_row;
      __threadfence_system();
      st_relaxed_sys(reinterpret_cast<unsigned int *>(x.peer[peer] + state_floats) + my_slot, tag);
    }
    for (int j = tid; j < count * x.world; j += kD) {
      const int flag_row = first_row + base + j / x.world, source = j % x.world;
      const unsigned int *flag = reinterpret_cast<const unsigned int *>(own + state_floats) + (static_cast<size_t>(parity) * x.world + source) * rows_total + flag_row;
      const long long start = clock64();
      unsigned int polls = 0;
      while (ld_acquire_sys(flag) != tag) {
        if ((++polls & 63u) == 0u && clock64() - start > 2000000000LL) {   // about a second: give up, report, carry on
          raise_status(x.status, 2);
          break;
        }
      }
    }
    __syncthreads();
    if (active) {
      // merge the world's states in ascending shard order (L1 is bypassed: peers wrote these lines)
      auto load_state = [&](int r, float &m, float &l, float4 &a) {
        const float *state = own + ((static_cast<size_t>(parity) * x.world + r) * rows_total + row) * kRecord;
        const float2 ml = __ldcg(reinterpret_cast<const float2 *>(state + kD));
        a = ldcg_quad(state + 4 * lane);
        m = ml.x; l = ml.y;
      };
      float m, l;
      float4 a;
      load_state(0, m, l, a);
      int r = 1;
      for (; r + 7 <= x.world; r += 7) {   // the states of seven more ranks in flight together (eight GPUs: one batch)
        float mr[7], lr[7];
        float4 ar[7];
#pragma unroll
        for (int u = 0; u < 7; ++u) load_state(r + u, mr[u], lr[u], ar[u]);
#pragma unroll
        for (int u = 0; u < 7; ++u) fd_merge_right(m, l, a, mr[u], lr[u], ar[u]);
      }
      for (; r < x.world; ++r) {
        float m_right, l_right;
        float4 a_right;
        load_state(r, m_right, l_right, a_right);
        fd_merge_right(m, l, a, m_right, l_right, a_right);
      }
      fd_write_row(x, row, lane, m, l, a);
    }
  }
  // the CTA that completes the last rows of the launch advances the epoch for the next call
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(x.epoch + 1, static_cast<unsigned int>(row_count)) + row_count == static_cast<unsigned int>(rows_total)) {
      x.epoch[1] = 0u;
      __threadfence();
      *reinterpret_cast<volatile unsigned int *>(x.epoch) = epoch + 1u;
    }
  }
}

// The same tail as a launch of its own (four rows per CTA), behind a stage 1 without it.
__global__ void __launch_bounds__(kD) fd_exchange_kernel(const FdTailParams x, const float *records, int splits, int rows_total) {
  const int first_row = blockIdx.x * (kD / 32);
  const int row_count = rows_total - first_row < kD / 32 ? rows_total - first_row : kD / 32;
  fd_exchange_rows<kD / 32>(x, records, splits, first_row, row_count, rows_total);
}

int visible_keys(const AttentionArgs &a) {
  int64_t visible = a.kv_valid < a.kv_len ? a.kv_valid : a.kv_len;
  if (a.causal && a.causal_offset + 1 < visible) visible = a.causal_offset + 1;
  return visible < 0 ? 0 : static_cast<int>(visible);
}

}  // namespace

bool attention_fd_supports(const AttentionArgs &a) {
  if (a.q_len != 1 || a.head_dim != kD) return false;
  if (a.format != WB200_BF16 && a.format != WB200_F16) return false;
  if (a.kv_heads <= 0 || a.q_heads % a.kv_heads != 0 || a.q_heads / a.kv_heads > 16) return false;
  if ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v)) & 15u)
    return false;
  return a.kv_len > 0 && a.batch > 0;
}

FdPlan fd_choose_plan(const AttentionArgs &a, int sm_count) {
  const int64_t visible = visible_keys(a);
  const int64_t units = static_cast<int64_t>(a.batch) * a.kv_heads;
  const int64_t all_slots = 2LL * sm_count;             // two CTAs are resident per SM
  // More (batch, kv head) units than resident slots: 2048-key splits give many short CTAs, which the hardware deals out
  // as slots free up (the tail is one short CTA), and the fold over a unit's few records is short.
  if (units >= all_slots) {
    const int64_t base = (visible + 2047) / 2048;
    return {1u, static_cast<uint32_t>(base < 1 ? 1 : (base > 4096 ? 4096 : base))};
  }
  // Otherwise the candidate with the least estimated time, in nanoseconds. A CTA keeps 64 to 96 KiB of copies in flight, about
  // 70 bytes / ns, and the HBM gives 6500 to all of them. Clusters of eight leave a part of every GPC unused. Merging inside a cluster costs about 1 us; a fold through global
  // records (fence, counter, second read) about 3 us more, plus the fold's own reads.
  FdPlan best{1u, 1u};
  double best_cost = -1;
  auto consider = [&](int64_t cluster, int64_t records) {
    const int64_t ctas = cluster * records;
    if (ctas > 1 && ctas * 64 > visible + 63) return;   // less than one tile per warp
    const double rows = static_cast<double>(((visible + ctas - 1) / ctas + 63) / 64 * 64);
    const double bytes = rows * (4.0 * kD);
    const int64_t slots = cluster == kMaxFdCluster ? all_slots * 7 / 8 : all_slots;
    double streaming = 0;
    for (int64_t left = units * ctas; left > 0; left -= slots) {
      const double active = static_cast<double>(left < slots ? left : slots);
      const double shared = active * bytes / 6500.0, alone = bytes / 70.0;
      streaming += (shared > alone ? shared : alone) + 500.0;
    }
    const double cost = streaming + (cluster > 1 ? 1000.0 : 0.0) + (records > 1 ? 3000.0 + 40.0 * static_cast<double>(records) : 0.0);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = {static_cast<uint32_t>(cluster), static_cast<uint32_t>(records)}; }
  };
  for (int64_t cluster = 1; cluster <= kMaxFdCluster; cluster *= 2) consider(cluster, 1);
  for (int64_t cluster = 1; cluster <= kMaxFdCluster; cluster *= 8)
    for (int64_t records = 2; records <= 256 && units * cluster * records <= 2 * all_slots; ++records) consider(cluster, records);
  return best;
}

size_t fd_partial_floats(const AttentionArgs &a, uint32_t records) {
  return static_cast<size_t>(a.batch) * a.q_heads * records * kRecord;
}

namespace {
wb200_status launch_fd_stage1(const AttentionArgs &a, FdPlan plan, float *partials, cudaStream_t stream, int tail_kind,
                              const FdTailParams &tail);
}

size_t fd_exchange_floats(int rows, int world) {
  // states [2][world][rows][kRecord] floats followed by flags [2][world][rows] words
  return static_cast<size_t>(2) * world * rows * (kRecord + 1);
}

wb200_status launch_attention_fd_exchange(const AttentionArgs &a, FdPlan plan, float *partials, int rank, int world,
                                          void *const *peer_buffers, unsigned int *epoch, unsigned int *arrivals,
                                          int *device_status, cudaStream_t stream) {
  if (world < 1 || world > kMaxExchangeRanks || rank < 0 || rank >= world)
    return fail(WB200_ERR_INVALID_ARGUMENT, "exchange takes 1 to 16 ranks and a rank inside the world");
  FdTailParams x;
  x.rank = rank; x.world = world;
  for (int r = 0; r < kMaxExchangeRanks; ++r) x.peer[r] = r < world ? static_cast<float *>(peer_buffers[r]) : nullptr;
  x.epoch = epoch;
  x.arrivals = arrivals;
  x.out_format = a.format;
  x.zero_fully_masked = a.zero_fully_masked;
  x.out = a.out; x.lse = a.lse; x.row_max = a.row_max; x.row_sum = a.row_sum;
  x.status = device_status;
  // With arrival counters the tail runs inside stage 1 (its last CTA per (batch, kv head)): one launch per step.
  // Without them it is a launch of its own behind stage 1.
  wb200_status st = launch_fd_stage1(a, plan, partials, stream, arrivals ? kTailExchange : kTailNone, x);
  if (st != WB200_OK) return st;
  if (!arrivals) {
    const int rows = a.batch * a.q_heads;
    fd_exchange_kernel<<<(rows + kD / 32 - 1) / (kD / 32), kD, 0, stream>>>(x, partials, static_cast<int>(plan.records), rows);
    WB200_CUDA_CHECK(cudaGetLastError());
  }
  return WB200_OK;
}

wb200_status launch_attention_fd(const AttentionArgs &a, FdPlan plan, float *partials, unsigned int *arrivals,
                                 float *state_out, cudaStream_t stream) {
  FdTailParams x{};
  x.arrivals = arrivals;
  x.out_format = a.format;
  x.zero_fully_masked = a.zero_fully_masked;
  x.out = a.out; x.lse = a.lse; x.row_max = a.row_max; x.row_sum = a.row_sum; x.state_out = state_out;
  return launch_fd_stage1(a, plan, partials, stream, kTailLocal, x);
}

namespace {
using FdKernel = void (*)(const FdParams, const FdTailParams);
template <int kTail, bool kNarrow>
constexpr FdKernel fd_kernel(bool bf16) { return bf16 ? fd_partial_kernel<true, kTail, kNarrow> : fd_partial_kernel<false, kTail, kNarrow>; }
const FdKernel kFdKernels[12] = {   // [tail][narrow][bf16]
    fd_kernel<kTailNone, false>(false),     fd_kernel<kTailNone, false>(true),     fd_kernel<kTailNone, true>(false),     fd_kernel<kTailNone, true>(true),
    fd_kernel<kTailLocal, false>(false),    fd_kernel<kTailLocal, false>(true),    fd_kernel<kTailLocal, true>(false),    fd_kernel<kTailLocal, true>(true),
    fd_kernel<kTailExchange, false>(false), fd_kernel<kTailExchange, false>(true), fd_kernel<kTailExchange, true>(false), fd_kernel<kTailExchange, true>(true)};

wb200_status launch_fd_stage1(const AttentionArgs &a, FdPlan plan, float *partials, cudaStream_t stream, int tail_kind,
                              const FdTailParams &tail) {
  if (!attention_fd_supports(a)) return fail(WB200_ERR_UNSUPPORTED, "flash-decoding request outside the kernel's domain");
  if (plan.records < 1 || plan.cluster < 1) return fail(WB200_ERR_INVALID_ARGUMENT, "kv_splits must be positive");
  FdParams p;
  p.batch = a.batch; p.q_heads = a.q_heads; p.kv_heads = a.kv_heads; p.group = a.q_heads / a.kv_heads;
  p.kv_len = a.kv_len;
  p.kv_visible = visible_keys(a);
  p.splits = static_cast<int>(plan.records);
  p.cluster = static_cast<int>(plan.cluster);
  const int64_t ctas = static_cast<int64_t>(plan.records) * plan.cluster;
  const int64_t per_cta = (static_cast<int64_t>(p.kv_visible) + ctas - 1) / ctas;
  const int64_t granule = kWarps * kTileRows;
  p.rows_per_cta = static_cast<int>(((per_cta + granule - 1) / granule) * granule);
  if (p.rows_per_cta == 0) p.rows_per_cta = static_cast<int>(granule);
  p.rows_per_warp = p.rows_per_cta / kWarps;
  p.scale = a.scale;
  p.q = static_cast<const uint16_t *>(a.q);
  p.k = static_cast<const uint16_t *>(a.k);
  p.v = static_cast<const uint16_t *>(a.v);
  p.partials = partials;

  static PerDeviceOnce attributes;
  const wb200_status attribute_status = attributes.run([]() -> wb200_status {
    for (const auto kernel : kFdKernels)
      WB200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFdSmemBytes));
    return WB200_OK;
  });
  if (attribute_status != WB200_OK) return attribute_status;
  static_assert(kWarps * 32 == kD, "the tail of the sharded decode runs with one thread per head dimension");
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(ctas), a.kv_heads, a.batch);
  config.blockDim = dim3(kWarps * 32);
  config.dynamicSmemBytes = kFdSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attribute[2];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  attribute[1].id = cudaLaunchAttributeClusterDimension;
  attribute[1].val.clusterDim.x = plan.cluster; attribute[1].val.clusterDim.y = 1; attribute[1].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = plan.cluster > 1 ? 2 : 1;
  WB200_CUDA_CHECK(cudaLaunchKernelEx(&config, kFdKernels[4 * tail_kind + (p.group <= 8 ? 2 : 0) + (a.format == WB200_BF16 ? 1 : 0)], p, tail));
  return WB200_OK;
}
}  // namespace

wb200_status launch_attention_fd_merge(const AttentionArgs &a, const float *states, uint32_t shard_count,
                                       cudaStream_t stream) {
  if (a.head_dim != kD) return fail(WB200_ERR_UNSUPPORTED, "merge supports head_dim 128");
  if (shard_count < 1) return fail(WB200_ERR_INVALID_ARGUMENT, "shard_count must be positive");
  FdCombineParams c;
  c.rows = a.batch * a.q_heads;
  c.records = static_cast<int>(shard_count);
  c.row_stride = kRecord;
  c.record_stride = static_cast<size_t>(c.rows) * kRecord;
  c.records_ptr = states;
  c.out_format = a.format;
  c.zero_fully_masked = a.zero_fully_masked;
  c.out = a.out; c.lse = a.lse; c.row_max = a.row_max; c.row_sum = a.row_sum;
  fd_combine_kernel<<<c.rows, kD, 0, stream>>>(c);
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

}  // namespace wb200

// ------------------------------------------------------------------ allocation-free entry point
// Some callers may not allocate device memory when they reach this library: a latency-critical
// serving loop whose memory was carved up at start-up and where a cudaMalloc (an implicit device
// synchronisation) is not acceptable, a host that shares the GPU under a fixed memory budget, or code
// that runs at a point where the CUDA runtime refuses allocation calls. For them the split-KV partial records live in
// a fixed array inside the library image instead of in a buffer the backend allocates on demand.
#include <mutex>

#include "backend.h"

namespace wb200 {
namespace {

constexpr size_t kStaticScratchFloats = size_t(4) << 20;   // 16 MiB, held by every GPU that loads the library
static __device__ __align__(256) float g_fd_static_scratch[kStaticScratchFloats];
// Arrival words of the (batch, kv head) units (fd_arrive); a unit has at least one row of at least one record.
constexpr size_t kStaticArrivals = kStaticScratchFloats / kRecord;
static __device__ unsigned int g_fd_static_arrivals[kStaticArrivals];

constexpr int kMaxDevices = 64;
float *g_fd_static_scratch_address[kMaxDevices] = {nullptr};
unsigned int *g_fd_static_arrivals_address[kMaxDevices] = {nullptr};
std::mutex g_fd_static_scratch_mutex;

// In host code `g_fd_static_scratch` names a host-side handle, not device memory; the address a kernel
// can use has to be asked for, once per device, with that device current.
wb200_status static_scratch_for_device(int device, float **out, unsigned int **arrivals) {
  if (device < 0 || device >= kMaxDevices) return fail(WB200_ERR_LIMIT, "device index beyond the static scratch table");
  std::lock_guard<std::mutex> lock(g_fd_static_scratch_mutex);
  if (!g_fd_static_scratch_address[device]) {
    void *address = nullptr;
    WB200_CUDA_CHECK(cudaGetSymbolAddress(&address, g_fd_static_arrivals));
    g_fd_static_arrivals_address[device] = static_cast<unsigned int *>(address);
    WB200_CUDA_CHECK(cudaGetSymbolAddress(&address, g_fd_static_scratch));
    g_fd_static_scratch_address[device] = static_cast<float *>(address);
  }
  *out = g_fd_static_scratch_address[device];
  *arrivals = g_fd_static_arrivals_address[device];
  return WB200_OK;
}

}  // namespace
}  // namespace wb200

extern "C" wb200_status wb200_attention_fd_static(wb200_backend *backend, const wb200_attention_params *p,
                                                  uint32_t kv_splits) {
  using namespace wb200;
  if (!backend || !p) return fail(WB200_ERR_INVALID_ARGUMENT, "null argument");
  if (p->memory != WB200_MEM_DEVICE)
    return fail(WB200_ERR_UNSUPPORTED, "the allocation-free decode takes device buffers only (staging host buffers would allocate)");
  if (!p->q || !p->k || !p->v || !p->out) return fail(WB200_ERR_INVALID_ARGUMENT, "q, k, v and out must not be null");
  if (p->q_len != 1) return fail(WB200_ERR_INVALID_ARGUMENT, "flash-decoding takes query length 1");
  if (p->batch == 0 || p->q_heads == 0 || p->kv_heads == 0 || p->kv_len == 0 || p->q_heads % p->kv_heads != 0 ||
      p->kv_len > 0x7fffffffu)
    return fail(WB200_ERR_INVALID_ARGUMENT, "invalid attention extents");
  AttentionArgs a{};
  a.batch = p->batch; a.q_heads = p->q_heads; a.kv_heads = p->kv_heads;
  a.q_len = 1; a.kv_len = p->kv_len; a.head_dim = p->head_dim;
  a.format = p->format;
  a.causal = p->causal ? 1 : 0;
  a.zero_fully_masked = p->zero_fully_masked ? 1 : 0;
  a.scale = p->scale;
  a.causal_offset = p->query_start - p->key_start;
  a.kv_valid = p->key_end > 0 ? p->key_end - p->key_start : static_cast<int64_t>(p->kv_len);
  a.q = p->q; a.k = p->k; a.v = p->v; a.out = p->out;
  a.lse = p->lse; a.row_max = p->row_max; a.row_sum = p->row_sum;
  if (!attention_fd_supports(a))
    return fail(WB200_ERR_UNSUPPORTED, "flash-decoding kernel takes f16/bf16 storage, head_dim 128, group size <= 16");
  DeviceGuard guard(backend->device);
  FdPlan plan{1u, kv_splits};
  if (kv_splits == 0) {
    plan = fd_choose_plan(a, backend->sm_count);
    while (plan.records > 2 && fd_partial_floats(a, plan.records) > kStaticScratchFloats) plan.records = (plan.records + 1) / 2;
  }
  const size_t needed = fd_partial_floats(a, plan.records);
  if (needed > kStaticScratchFloats)
    return fail(WB200_ERR_LIMIT, "allocation-free decode: batch * q_heads * kv_splits * (head_dim + 2) = " + std::to_string(needed) +
                                     " floats exceeds the fixed scratch of " + std::to_string(kStaticScratchFloats) + " floats (16 MiB)");
  float *scratch = nullptr;
  unsigned int *arrivals = nullptr;
  wb200_status st = static_scratch_for_device(backend->device, &scratch, &arrivals);
  if (st != WB200_OK) return st;
  // Stage 1 writes every record stage 2 reads, so nothing left by an earlier call needs clearing.
  st = launch_attention_fd(a, plan, scratch, arrivals, nullptr, static_cast<cudaStream_t>(p->stream));
  if (st == WB200_OK) backend->launches += 1;
  return st;
}
