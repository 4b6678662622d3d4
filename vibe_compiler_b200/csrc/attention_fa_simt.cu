// Flash-attention prefill on CUDA cores, f32 arithmetic throughout: the path for f32 storage (where
// the 1e-5 parity bound rules out tensor-core inputs narrower than f32) and for shapes the tcgen05
// kernel does not take. In the general kernel one warp owns one query row and walks the keys in tiles of 32 that the block's sixteen
// rows share through shared memory, applying the reference's online update literally
// (lib/Wafer/Transforms/Linalg/OnlineAttentionDecomposition.cpp:568-594):
//   s = (q.k)*scale (+mask); m' = max(m, max s); m_e = (m' == -inf ? 0 : m'); alpha = ExpLp(m - m_e);
//   l = l*alpha + sum ExpLp(s - m_e); acc = acc*alpha + round_to_storage(P) V
// and the finalize acc * (1/l) of OnlineAttentionMaterialization.cpp:196-262. ExpLp is
// exp2(x * log2e) in f32 (lib/Wafer/Simulator/Reference/ManagedReferenceTargetModel.cpp:265-270).
#include "kernels.h"
#include "ptx_sm100.cuh"

namespace wb200 {
namespace {

constexpr int kWarpsPerBlock = 16;   // query rows of one head per block; they share every staged K / V tile
constexpr int kMaxDPerLane = 8;      // head_dim <= 256
constexpr int kTileKeys = 32;

struct SimtParams {
  AttentionArgs a;
  int group;
  int kv_visible;
  int vector;   // K and V are 16-byte aligned: the staging loop may use wide loads
};

__device__ __forceinline__ float exp_lp(float x) { return exp2f(__fmul_rn(x, 0x1.715476p+0f)); }

// Shared memory: q rows [kWarpsPerBlock][D], the K tile [32][D + 1] (the pad keeps the per-lane row reads of the score
// loop on distinct banks) and the V tile [32][D], all widened to f32 once per block instead of once per query row.
// kD fixes head_dim at compile time (0: runtime) so the score and PV loops unroll and their shared-memory reads pipeline.
template <int kD>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) fa_simt_kernel(const SimtParams p) {
  const AttentionArgs &a = p.a;
  extern __shared__ float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * kWarpsPerBlock + warp;
  const int bh = blockIdx.y;
  const int b = bh / a.q_heads, h = bh % a.q_heads;
  const int D = kD ? kD : a.head_dim;
  const int per_lane = D / 32;
  const bool active = row < a.q_len;
  float *q_smem = smem, *k_tile = smem + kWarpsPerBlock * D, *v_tile = k_tile + kTileKeys * (D + 1);

  const size_t q_off = (static_cast<size_t>(bh) * a.q_len + (active ? row : 0)) * D;
  const size_t kv_off = (static_cast<size_t>(b) * a.kv_heads + h / p.group) * static_cast<size_t>(a.kv_len) * D;
  const uint8_t *q = static_cast<const uint8_t *>(a.q);
  const uint8_t *k = static_cast<const uint8_t *>(a.k);
  const uint8_t *v = static_cast<const uint8_t *>(a.v);
  float *my_q = q_smem + warp * D;
  if (active)
    for (int d = lane; d < D; d += 32) my_q[d] = widen_bits(load_element_bits(q, q_off + d, a.format), a.format);

  auto visible_of = [&](int r) {
    long long last = static_cast<long long>(p.kv_visible) - 1;
    if (a.causal && a.causal_offset + r < last) last = a.causal_offset + r;
    return last < 0 ? 0 : static_cast<int>(last + 1);
  };
  const int visible = active ? visible_of(row) : 0;
  // the last row of the block sees the most keys
  const int last_row = min(static_cast<int>(blockIdx.x) * kWarpsPerBlock + kWarpsPerBlock - 1, a.q_len - 1);
  const int block_visible = visible_of(last_row);

  float m_run = -INFINITY, l_run = 0.0f;
  float acc[kMaxDPerLane];
#pragma unroll
  for (int i = 0; i < kMaxDPerLane; ++i) acc[i] = 0.0f;

  for (int key0 = 0; key0 < block_visible; key0 += kTileKeys) {
    __syncthreads();   // the previous tile has been consumed (and, first time round, the q rows are written)
    const int tile_keys = min(kTileKeys, block_visible - key0);
    // four consecutive elements per thread and step (head_dim is a multiple of 32): the loads of a step are issued
    // together, 128 bits wide for f32 storage and 64 bits wide for the 16-bit formats
    const int quads = p.vector ? tile_keys * D / 4 : 0;
    for (int e = threadIdx.x; e < quads; e += kWarpsPerBlock * 32) {
      const int j = (e * 4) / D, d = e * 4 - j * D;
      const size_t at = kv_off + static_cast<size_t>(key0 + j) * D + d;
      float kf[4], vf[4];
      if (a.format == WB200_F32) {
        const float4 kq = *reinterpret_cast<const float4 *>(k + at * 4), vq = *reinterpret_cast<const float4 *>(v + at * 4);
        kf[0] = kq.x; kf[1] = kq.y; kf[2] = kq.z; kf[3] = kq.w;
        vf[0] = vq.x; vf[1] = vq.y; vf[2] = vq.z; vf[3] = vq.w;
      } else {
        const uint2 kq = *reinterpret_cast<const uint2 *>(k + at * 2), vq = *reinterpret_cast<const uint2 *>(v + at * 2);
        kf[0] = widen_bits(kq.x & 0xffffu, a.format); kf[1] = widen_bits(kq.x >> 16, a.format);
        kf[2] = widen_bits(kq.y & 0xffffu, a.format); kf[3] = widen_bits(kq.y >> 16, a.format);
        vf[0] = widen_bits(vq.x & 0xffffu, a.format); vf[1] = widen_bits(vq.x >> 16, a.format);
        vf[2] = widen_bits(vq.y & 0xffffu, a.format); vf[3] = widen_bits(vq.y >> 16, a.format);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        k_tile[j * (D + 1) + d + i] = kf[i];
        v_tile[j * D + d + i] = vf[i];
      }
    }
    if (!p.vector)
      for (int e = threadIdx.x; e < tile_keys * D; e += kWarpsPerBlock * 32) {
        const int j = e / D, d = e - j * D;
        const size_t at = kv_off + static_cast<size_t>(key0 + j) * D + d;
        k_tile[j * (D + 1) + d] = widen_bits(load_element_bits(k, at, a.format), a.format);
        v_tile[j * D + d] = widen_bits(load_element_bits(v, at, a.format), a.format);
      }
    __syncthreads();
    if (key0 >= visible) continue;   // this row's keys ended in an earlier tile (causal rows above the block's last)
    const int key = key0 + lane;
    float s = -INFINITY;
    if (key < visible) {
      float dot = 0.0f;
      const float *k_row = k_tile + lane * (D + 1);
#pragma unroll 16
      for (int d = 0; d < D; ++d) dot = __fmaf_rn(my_q[d], k_row[d], dot);
      s = __fmul_rn(dot, a.scale);
    }
    float tile_max = s;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, off));
    const float m_new = fmaxf(tile_max, m_run);
    const float m_exp = (m_new == -INFINITY) ? 0.0f : m_new;
    const float alpha = exp_lp(__fsub_rn(m_run, m_exp));
    const float prob = exp_lp(__fsub_rn(s, m_exp));
    float tile_sum = prob;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) tile_sum += __shfl_xor_sync(0xffffffffu, tile_sum, off);
    l_run = __fadd_rn(__fmul_rn(l_run, alpha), tile_sum);
    m_run = m_new;
    // P is rounded to the storage type of V before the PV contraction.
    const float prob_rounded = widen_bits(narrow_bits(prob, a.format), a.format);
#pragma unroll
    for (int i = 0; i < kMaxDPerLane; ++i) acc[i] = __fmul_rn(acc[i], alpha);
    const int count = min(kTileKeys, visible - key0);
#pragma unroll 8
    for (int j = 0; j < count; ++j) {
      const float pj = __shfl_sync(0xffffffffu, prob_rounded, j);
      const float *v_row = v_tile + j * D;
#pragma unroll
      for (int i = 0; i < kMaxDPerLane; ++i)
        if (i < per_lane) acc[i] = __fmaf_rn(pj, v_row[i * 32 + lane], acc[i]);
    }
  }
  if (!active) return;

  float coefficient = __fdiv_rn(1.0f, l_run);
  if (a.zero_fully_masked && l_run == 0.0f) coefficient = 0.0f;
  uint8_t *out = static_cast<uint8_t *>(a.out);
  const size_t out_off = a.out_token_major ? ((static_cast<size_t>(b) * a.q_len + row) * a.q_heads + h) * D : q_off;
#pragma unroll
  for (int i = 0; i < kMaxDPerLane; ++i)
    if (i < per_lane)
      store_element_bits(out, out_off + i * 32 + lane, a.format, narrow_bits(__fmul_rn(acc[i], coefficient), a.format));
  if (lane == 0) {
    const size_t stat = static_cast<size_t>(bh) * a.q_len + row;
    if (a.lse) a.lse[stat] = (l_run == 0.0f) ? -INFINITY : m_run + logf(l_run);
    if (a.row_max) a.row_max[stat] = m_run;
    if (a.row_sum) a.row_sum[stat] = l_run;
  }
}

// ---------------------------------------------------------------- f32 storage, head_dim 64 or 128: register tiles
// A block owns 32 query rows of one (batch, head). Its two or four groups of 128 threads (f32_groups below) walk the tiles of
// 64 keys in turn, each with a state of its own; the states are merged once at the end. A thread holds
// 4 rows x 4 keys of the scores (keys tx, tx + 16, ...) and 4 rows x D/16 columns of the accumulator, so 64 multiply-adds
// follow on 8 shared-memory vectors; the 16 threads of a row are half a warp, which keeps the row statistics and P inside
// the warp. K and V have a buffer each, refilled by cp.async as soon as the group has read it: K of the next tile travels
// under the softmax and the PV product, V under the next scores.
// Bound by the f32 multiply-adds (8 heads x 512 x 512 x 64: 0.27 G, 7 us at the rate of 148 SMs; 128 of them have a block)
// and the shared-memory vectors that feed them: 73.7 us with a warp per row, 24.4 us with two groups, 22.4 us with four (16
// warps hide more of the latency of loads, shuffles and exponentials). The warp-per-row kernel stays for other widths, 16-bit
// storage and unaligned buffers.
constexpr int kTileRows = 32, kTileKeysWide = 64, kGroupThreads = 128;

template <int kD, int kGroups>
struct TiledSmem {
  static constexpr int kKPitch = kD + 4;   // rows 16 bytes apart modulo the banks: eight lanes' vectors cover all banks
  static constexpr int kPPitch = kTileKeysWide + 4;
  static constexpr int kQ = 0;
  static constexpr int kGroup0 = kTileRows * kKPitch;
  static constexpr int kV = kTileKeysWide * kKPitch;                 // within a group
  static constexpr int kP = kV + kTileKeysWide * kD;
  static constexpr int kGroupFloats = kP + kTileRows * kPPitch;
  static constexpr size_t kBytes = (kGroup0 + kGroups * kGroupFloats) * sizeof(float);
};

template <int kD, int kGroups>
__global__ void __launch_bounds__(kGroups * kGroupThreads) fa_f32_kernel(const SimtParams p) {
  using L = TiledSmem<kD, kGroups>;
  const AttentionArgs &a = p.a;
  extern __shared__ float4 smem_vectors[];
  float *smem = reinterpret_cast<float *>(smem_vectors);
  const int group_id = threadIdx.x / kGroupThreads, tid = threadIdx.x % kGroupThreads;
  const int tx = tid & 15, ty = tid >> 4;
  const int row_block = static_cast<int>(gridDim.x - 1 - blockIdx.x) * kTileRows;   // causal: the longest rows first
  const int bh = blockIdx.y;
  const int b = bh / a.q_heads, h = bh % a.q_heads;
  float *q_s = smem + L::kQ;
  float *k_s = smem + L::kGroup0 + group_id * L::kGroupFloats, *v_s = k_s + L::kV, *p_s = k_s + L::kP;
  const size_t kv_off = (static_cast<size_t>(b) * a.kv_heads + h / p.group) * static_cast<size_t>(a.kv_len) * kD;
  const float *q = static_cast<const float *>(a.q) + (static_cast<size_t>(bh) * a.q_len + row_block) * kD;
  const float *k = static_cast<const float *>(a.k) + kv_off, *v = static_cast<const float *>(a.v) + kv_off;

  auto visible_of = [&](int r) {
    long long last = static_cast<long long>(p.kv_visible) - 1;
    if (a.causal && a.causal_offset + r < last) last = a.causal_offset + r;
    return last < 0 ? 0 : static_cast<int>(last + 1);
  };
  const int rows = min(kTileRows, a.q_len - row_block);
  const int block_visible = visible_of(row_block + rows - 1);   // the last row of the block sees the most keys
  const int least_visible = visible_of(row_block);
  int visible[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) visible[i] = ty * 4 + i < rows ? visible_of(row_block + ty * 4 + i) : 0;

  auto fetch = [&](float *dst, int pitch, const float *src, int key0) {
    const int count = min(kTileKeysWide, block_visible - key0);   // keys behind it are never used
    for (int e = tid; e < count * (kD / 4); e += kGroupThreads) {
      const int j = e / (kD / 4), d = e % (kD / 4) * 4;
      cp_async16(smem_u32(dst + j * pitch + d), src + static_cast<size_t>(key0 + j) * kD + d, 16u);
    }
  };
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + group_id), "n"(kGroupThreads) : "memory"); };

  pdl_wait();
  pdl_launch_dependents();
  for (int e = threadIdx.x; e < kTileRows * (kD / 4); e += kGroups * kGroupThreads) {
    const int r = e / (kD / 4), d = e % (kD / 4) * 4;
    cp_async16(smem_u32(q_s + r * L::kKPitch + d), q + static_cast<size_t>(min(r, rows - 1)) * kD + d, 16u);
  }
  int key0 = group_id * kTileKeysWide;
  if (key0 < block_visible) fetch(k_s, L::kKPitch, k, key0);
  cp_async_commit();
  if (key0 < block_visible) fetch(v_s, kD, v, key0);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();   // every thread's part of Q (and of the first K) has landed

  float m_run[4], l_run[4], acc[4][kD / 16];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.0f;
#pragma unroll
    for (int c = 0; c < kD / 16; ++c) acc[i][c] = 0.0f;
  }

  for (; key0 < block_visible; key0 += kGroups * kTileKeysWide) {
    const int next = key0 + kGroups * kTileKeysWide;
    cp_async_wait<1>();   // K of this tile (its V may still travel)
    group_sync();
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
#pragma unroll 4
    for (int d = 0; d < kD; d += 4) {
      float4 qv[4], kv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4 *>(q_s + (ty * 4 + i) * L::kKPitch + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4 *>(k_s + (tx + 16 * j) * L::kKPitch + d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = __fmaf_rn(qv[i].x, kv[j].x, s[i][j]);
          s[i][j] = __fmaf_rn(qv[i].y, kv[j].y, s[i][j]);
          s[i][j] = __fmaf_rn(qv[i].z, kv[j].z, s[i][j]);
          s[i][j] = __fmaf_rn(qv[i].w, kv[j].w, s[i][j]);
        }
    }
    group_sync();
    if (next < block_visible) fetch(k_s, L::kKPitch, k, next);
    cp_async_commit();

    const bool masked = key0 + kTileKeysWide > least_visible;   // some row of the block does not see the whole tile
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float tile_max = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = (masked && key0 + tx + 16 * j >= visible[i]) ? -INFINITY : __fmul_rn(s[i][j], a.scale);
        tile_max = fmaxf(tile_max, s[i][j]);
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, off));
      const float m_new = fmaxf(tile_max, m_run[i]);
      const float m_exp = (m_new == -INFINITY) ? 0.0f : m_new;
      const float alpha = exp_lp(__fsub_rn(m_run[i], m_exp));
      float tile_sum = 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float prob = exp_lp(__fsub_rn(s[i][j], m_exp));
        tile_sum += prob;
        p_s[(ty * 4 + i) * L::kPPitch + tx + 16 * j] = prob;
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) tile_sum += __shfl_xor_sync(0xffffffffu, tile_sum, off);
      l_run[i] = __fadd_rn(__fmul_rn(l_run[i], alpha), tile_sum);
      m_run[i] = m_new;
#pragma unroll
      for (int c = 0; c < kD / 16; ++c) acc[i][c] = __fmul_rn(acc[i][c], alpha);
    }
    cp_async_wait<1>();   // V of this tile (K of the next one may still travel)
    group_sync();         // also: the half warp's P is written
    // keys that every row of the block sees, in fours
    const int common = masked ? max(least_visible - key0, 0) & ~3 : kTileKeysWide;
    {
#pragma unroll 2
      for (int j = 0; j < common; j += 4) {
        float4 pv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) pv[i] = *reinterpret_cast<const float4 *>(p_s + (ty * 4 + i) * L::kPPitch + j);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
#pragma unroll
          for (int c = 0; c < kD / 64; ++c) {
            const float4 vv = *reinterpret_cast<const float4 *>(v_s + (j + jj) * kD + c * 64 + tx * 4);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float pj = jj == 0 ? pv[i].x : jj == 1 ? pv[i].y : jj == 2 ? pv[i].z : pv[i].w;
              acc[i][4 * c] = __fmaf_rn(pj, vv.x, acc[i][4 * c]);
              acc[i][4 * c + 1] = __fmaf_rn(pj, vv.y, acc[i][4 * c + 1]);
              acc[i][4 * c + 2] = __fmaf_rn(pj, vv.z, acc[i][4 * c + 2]);
              acc[i][4 * c + 3] = __fmaf_rn(pj, vv.w, acc[i][4 * c + 3]);
            }
          }
      }
    }
    if (masked) {
      // A key a row does not see takes no part in its product: 0 * V would turn an infinity there into a NaN.
      const int count = min(kTileKeysWide, block_visible - key0);
#pragma unroll 1
      for (int j = common; j < count; ++j) {
        float vv[kD / 16];
#pragma unroll
        for (int c = 0; c < kD / 16; ++c) vv[c] = v_s[j * kD + (c / 4) * 64 + tx * 4 + c % 4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float pj = p_s[(ty * 4 + i) * L::kPPitch + j];
          if (key0 + j < visible[i]) {
#pragma unroll
            for (int c = 0; c < kD / 16; ++c) acc[i][c] = __fmaf_rn(pj, vv[c], acc[i][c]);
          }
        }
      }
    }
    group_sync();
    if (next < block_visible) fetch(v_s, kD, v, next);
    cp_async_commit();
  }
  cp_async_wait<0>();
  __syncthreads();

  // Merge: the other groups leave their states in their own K / V buffers, group 0 folds them in and finalizes.
  auto state_of = [&](int g) { return smem + L::kGroup0 + g * L::kGroupFloats; };   // [32][D], then m [32], l [32]
  if (group_id > 0) {
    float *state = state_of(group_id), *stats = state + kTileRows * kD;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int c = 0; c < kD / 64; ++c)
        *reinterpret_cast<float4 *>(state + (ty * 4 + i) * kD + c * 64 + tx * 4) =
            make_float4(acc[i][4 * c], acc[i][4 * c + 1], acc[i][4 * c + 2], acc[i][4 * c + 3]);
      if (tx == 0) {
        stats[ty * 4 + i] = m_run[i];
        stats[kTileRows + ty * 4 + i] = l_run[i];
      }
    }
  }
  __syncthreads();
  if (group_id > 0) return;
  float *out = static_cast<float *>(a.out);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i, row = row_block + r;
    if (r >= rows) continue;
    float m_all = m_run[i];
#pragma unroll
    for (int g = 1; g < kGroups; ++g) m_all = fmaxf(m_all, state_of(g)[kTileRows * kD + r]);
    const float m_exp = (m_all == -INFINITY) ? 0.0f : m_all;
    const float mine = exp_lp(__fsub_rn(m_run[i], m_exp));
    float l_all = __fmul_rn(l_run[i], mine), other[kGroups];
#pragma unroll
    for (int g = 1; g < kGroups; ++g) {
      const float *stats = state_of(g) + kTileRows * kD;
      other[g] = exp_lp(__fsub_rn(stats[r], m_exp));
      l_all = __fadd_rn(l_all, __fmul_rn(stats[kTileRows + r], other[g]));
    }
    float coefficient = __fdiv_rn(1.0f, l_all);
    if (a.zero_fully_masked && l_all == 0.0f) coefficient = 0.0f;
    float *dst = out + (a.out_token_major ? ((static_cast<size_t>(b) * a.q_len + row) * a.q_heads + h) * kD : (static_cast<size_t>(bh) * a.q_len + row) * kD);
#pragma unroll
    for (int c = 0; c < kD / 64; ++c) {
      float sum[4];
#pragma unroll
      for (int g = 1; g < kGroups; ++g) {
        const float4 o = *reinterpret_cast<const float4 *>(state_of(g) + r * kD + c * 64 + tx * 4);
        const float others[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] = g == 1 ? __fmul_rn(others[e], other[g]) : __fmaf_rn(others[e], other[g], sum[e]);
      }
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = narrow_bits(__fmul_rn(__fmaf_rn(acc[i][4 * c + e], mine, sum[e]), coefficient), WB200_F32);
      *reinterpret_cast<uint4 *>(dst + c * 64 + tx * 4) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (tx == 0) {
      const size_t stat = static_cast<size_t>(bh) * a.q_len + row;
      if (a.lse) a.lse[stat] = (l_all == 0.0f) ? -INFINITY : m_all + logf(l_all);
      if (a.row_max) a.row_max[stat] = m_all;
      if (a.row_sum) a.row_sum[stat] = l_all;
    }
  }
}

// Key groups of a block. At head_dim 64 shared memory holds four, one block to an SM, or two blocks of two groups each; at 128
// two. Four are for blocks that would have an SM to themselves with two: where no more blocks than SMs are launched, and on
// causal requests of few heads, whose long blocks outlast the short ones beside them. With no more than two tiles of keys half
// of them would idle. us with two / four groups, 64 columns, heads x rows (= keys): all keys 8 x 512 24.4 / 22.4, 8 x 1024
// 74.6 / 78.9, 32 x 256 21.4 / 24.6, 512 x 128 75.0 / 105.8, 512 x 512 1016 / 1169; causal 10 x 512 37.4 / 23.9, 8 x 1024
// 72.0 / 62.0, 20 x 1024 125 / 121, 20 x 512 42.8 / 42.6, 24 x 1024 139 / 140, 32 x 256 21.4 / 23.6. A row's bits depend on the
// number of groups, and so on the heads and sequences beside it.
int f32_groups(const AttentionArgs &a, int kv_visible, int64_t blocks) {
  const bool few = blocks <= 148 || (a.causal && a.batch * static_cast<int64_t>(a.q_heads) <= 20);
  return a.head_dim == 64 && kv_visible > 2 * kTileKeysWide && few ? 4 : 2;
}

}  // namespace

wb200_status launch_attention_fa_simt(const AttentionArgs &a, cudaStream_t stream) {
  if (!is_float_format(a.format)) return fail(WB200_ERR_UNSUPPORTED, "attention admits f16, bf16 and f32 storage");
  if (a.head_dim <= 0 || a.head_dim % 32 != 0 || a.head_dim > 32 * kMaxDPerLane)
    return fail(WB200_ERR_UNSUPPORTED, "head_dim must be a multiple of 32 up to 256");
  if (a.kv_heads <= 0 || a.q_heads % a.kv_heads != 0 || a.q_len <= 0 || a.kv_len <= 0 || a.batch <= 0)
    return fail(WB200_ERR_INVALID_ARGUMENT, "invalid attention extents");
  SimtParams p;
  p.a = a;
  p.group = a.q_heads / a.kv_heads;
  int64_t visible = a.kv_valid < a.kv_len ? a.kv_valid : a.kv_len;
  p.kv_visible = visible < 0 ? 0 : static_cast<int>(visible);
  // The register-tiled kernel takes every f32 request whose buffers allow 16-byte accesses.
  const bool aligned = ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v) |
                         reinterpret_cast<uintptr_t>(a.out)) & 15u) == 0;
  if (a.format == WB200_F32 && aligned && (a.head_dim == 64 || a.head_dim == 128)) {
    static PerDeviceOnce attributes;
    const wb200_status st = attributes.run([]() -> wb200_status {
      WB200_CUDA_CHECK(cudaFuncSetAttribute(fa_f32_kernel<64, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(TiledSmem<64, 2>::kBytes)));
      WB200_CUDA_CHECK(cudaFuncSetAttribute(fa_f32_kernel<64, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(TiledSmem<64, 4>::kBytes)));
      WB200_CUDA_CHECK(cudaFuncSetAttribute(fa_f32_kernel<128, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(TiledSmem<128, 2>::kBytes)));
      return WB200_OK;
    });
    if (st != WB200_OK) return st;
    const dim3 tiles((a.q_len + kTileRows - 1) / kTileRows, a.batch * a.q_heads);
    const int groups = f32_groups(a, p.kv_visible, static_cast<int64_t>(tiles.x) * tiles.y);
    if (a.head_dim == 128) WB200_CUDA_CHECK(launch_dependent(fa_f32_kernel<128, 2>, tiles, 2 * kGroupThreads, TiledSmem<128, 2>::kBytes, stream, p));
    else if (groups == 4) WB200_CUDA_CHECK(launch_dependent(fa_f32_kernel<64, 4>, tiles, 4 * kGroupThreads, TiledSmem<64, 4>::kBytes, stream, p));
    else WB200_CUDA_CHECK(launch_dependent(fa_f32_kernel<64, 2>, tiles, 2 * kGroupThreads, TiledSmem<64, 2>::kBytes, stream, p));
    return WB200_OK;
  }
  dim3 grid((a.q_len + kWarpsPerBlock - 1) / kWarpsPerBlock, a.batch * a.q_heads);
  const size_t smem_bytes = (static_cast<size_t>(kWarpsPerBlock) * a.head_dim + kTileKeys * (a.head_dim + 1) + kTileKeys * a.head_dim) * sizeof(float);
  // wide staging loads need 16-byte aligned K / V bases; head_dim % 32 == 0 keeps every row aligned
  p.vector = ((reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v)) & 15) == 0;
#define WB200_SIMT_LAUNCH(KD)                                                                                                  \
  do {                                                                                                                         \
    if (smem_bytes > 48 * 1024)                                                                                                \
      WB200_CUDA_CHECK(cudaFuncSetAttribute(fa_simt_kernel<KD>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_bytes))); \
    fa_simt_kernel<KD><<<grid, kWarpsPerBlock * 32, smem_bytes, stream>>>(p);                                                  \
  } while (0)
  if (a.head_dim == 64) WB200_SIMT_LAUNCH(64);
  else if (a.head_dim == 128) WB200_SIMT_LAUNCH(128);
  else WB200_SIMT_LAUNCH(0);
#undef WB200_SIMT_LAUNCH
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

}  // namespace wb200
