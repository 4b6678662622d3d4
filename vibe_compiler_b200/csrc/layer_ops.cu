// Memory-bound producer / epilogue pieces of a Llama-style decoder layer that sit between the GEMM and
// attention regions: RMSNorm, rotary embedding fused with the head-major relayout of the QKV projection,
// and the residual add. Arithmetic is f32 with one rounding to the storage type per produced element,
// the accumulation contract of the reference's elementwise chains
// (lib/Wafer/Simulator/Reference/ManagedReferenceTargetModel.cpp:230-342: decode to f32, operate, RNE encode).
// All three are HBM-bound: algorithmic bytes = bytes read + bytes written once.
#include "kernels.h"
#include "ptx_sm100.cuh"

namespace wb200 {
namespace {

constexpr int kNormThreads = 256;

template <bool kBf16>
__device__ __forceinline__ float2 unpack2(uint32_t bits) {
  if constexpr (kBf16) return make_float2(__uint_as_float(bits << 16), __uint_as_float(bits & 0xffff0000u));
  else return __half22float2(*reinterpret_cast<const __half2 *>(&bits));
}
template <bool kBf16>
__device__ __forceinline__ uint32_t pack2f(float lo, float hi) {
  if constexpr (kBf16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
  }
}

// y[row] = round(round(x * rsqrt(mean(x^2) + eps)) * gamma): the normalised value is rounded to the storage
// type before the weight is applied, as the eager module the reference's block test runs does.
// kAdd: x is round(x + addend), stored to `sum` on the way (the residual add in front of the second norm of a layer: its
// result is not read back; as two kernels 54 + 48 us at 16384 rows x 4096 bf16, 5.9 + 5.6 us at 1000).
// A thread keeps its first kKept chunks of the row in registers, so rows of up to 8192 elements are read once.
template <bool kBf16, bool kAdd>
__global__ void __launch_bounds__(kNormThreads) rmsnorm_kernel(const uint16_t *x, const uint16_t *addend, uint16_t *sum, const uint16_t *gamma,
                                                                uint16_t *y, int dim, float eps) {
  constexpr int kKept = 4;
  pdl_wait();
  pdl_launch_dependents();
  const size_t row = static_cast<size_t>(blockIdx.x) * dim;
  const uint4 *src = reinterpret_cast<const uint4 *>(x + row);
  const int chunks = dim / 8;
  float partial = 0.f;
  uint4 kept[kKept];
  auto take = [&](int c) {
    uint4 v = src[c];
    if constexpr (kAdd) {
      const uint4 other = reinterpret_cast<const uint4 *>(addend + row)[c];
      uint32_t w[4] = {v.x, v.y, v.z, v.w};
      const uint32_t ow[4] = {other.x, other.y, other.z, other.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = unpack2<kBf16>(w[i]), g = unpack2<kBf16>(ow[i]);
        w[i] = pack2f<kBf16>(f.x + g.x, f.y + g.y);
      }
      v = make_uint4(w[0], w[1], w[2], w[3]);
      reinterpret_cast<uint4 *>(sum + row)[c] = v;
    }
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = unpack2<kBf16>(w[i]);
      partial = fmaf(f.x, f.x, partial);
      partial = fmaf(f.y, f.y, partial);
    }
    return v;
  };
#pragma unroll
  for (int i = 0; i < kKept; ++i)
    if (threadIdx.x + i * kNormThreads < chunks) kept[i] = take(threadIdx.x + i * kNormThreads);
  for (int c = threadIdx.x + kKept * kNormThreads; c < chunks; c += kNormThreads) take(c);
  __shared__ float warp_sums[kNormThreads / 32];
  __shared__ float inv_rms;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) partial += __shfl_xor_sync(0xffffffffu, partial, off);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = partial;
  __syncthreads();
  if (threadIdx.x == 0) {
    float total = 0.f;
    for (int w = 0; w < kNormThreads / 32; ++w) total += warp_sums[w];
    inv_rms = rsqrtf(total / static_cast<float>(dim) + eps);
  }
  __syncthreads();
  const float inv = inv_rms;
  const uint4 *g = reinterpret_cast<const uint4 *>(gamma);
  uint4 *dst = reinterpret_cast<uint4 *>(y + row);
  auto put = [&](int c, const uint4 &v) {
    const uint4 gv = g[c];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w}, gw[4] = {gv.x, gv.y, gv.z, gv.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = unpack2<kBf16>(w[i]);
      const float2 normalised = unpack2<kBf16>(pack2f<kBf16>(f.x * inv, f.y * inv));
      const float2 gf = unpack2<kBf16>(gw[i]);
      o[i] = pack2f<kBf16>(normalised.x * gf.x, normalised.y * gf.y);
    }
    dst[c] = make_uint4(o[0], o[1], o[2], o[3]);
  };
#pragma unroll
  for (int i = 0; i < kKept; ++i)
    if (threadIdx.x + i * kNormThreads < chunks) put(threadIdx.x + i * kNormThreads, kept[i]);
  // a sum is read back by the thread that stored it
  const uint4 *again = kAdd ? reinterpret_cast<const uint4 *>(sum + row) : src;
  for (int c = threadIdx.x + kKept * kNormThreads; c < chunks; c += kNormThreads) put(c, again[c]);
}

// qkv is the projection output, token-major: row (b * seq + s) holds [q heads | k heads | v heads] x head_dim.
// Writes head-major Q [B, Hq, S, D], K [B, Hkv, S, D], V [B, Hkv, S, D]; Q and K get the rotary embedding
// (pairs (i, i + D/2), angle = (position_offset + s) * theta^(-2i/D), f32 math, one rounding).
// One block per token: the sines and cosines of its D/2 angles are the same for every head, so they are computed once into
// shared memory; with them per head the kernel was bound by sincosf. kVec = elements of either half per thread and step:
// 8 (16-byte accesses; head_dim % 16 == 0) or 2.
// 16384 tokens x 48 heads x 128 bf16 (403 MB, 61 us at the copy rate): 178 us with the angles per head, 64 us now; 1000 tokens 16.3 -> 7.5.
constexpr int kRopeThreads = 128;
constexpr int kRopeAngles = 512;   // angles in shared memory at a time

template <bool kBf16, int kVec>
__global__ void __launch_bounds__(kRopeThreads) rope_split_kernel(const uint16_t *qkv, uint16_t *q, uint16_t *k, uint16_t *v,
                                                                   int seq, int q_heads, int kv_heads, int head_dim,
                                                                   float log2_theta, int position_offset) {
  __shared__ float2 angles[kRopeAngles];   // (sin, cos)
  const int token = blockIdx.x;
  const int b = token / seq, s = token % seq;
  const int heads = q_heads + 2 * kv_heads;
  const int half = head_dim / 2;
  const uint16_t *row = qkv + static_cast<size_t>(token) * heads * head_dim;
  const float position = static_cast<float>(position_offset + s);
  pdl_launch_dependents();
  for (int first = 0; first < half; first += kRopeAngles) {
    const int count = min(kRopeAngles, half - first);
    if (first > 0) __syncthreads();
    for (int i = threadIdx.x; i < count; i += kRopeThreads) {
      float sine, cosine;
      sincosf(position * exp2f(-2.0f * static_cast<float>(first + i) / static_cast<float>(head_dim) * log2_theta), &sine, &cosine);
      angles[i] = make_float2(sine, cosine);
    }
    __syncthreads();
    if (first == 0) pdl_wait();   // the angles need nothing of the kernel before this one
    const int groups = count / kVec;
    for (int idx = threadIdx.x; idx < heads * groups; idx += kRopeThreads) {
      const int head = idx / groups, at = (idx % groups) * kVec, i = first + at;
      const uint16_t *src = row + static_cast<size_t>(head) * head_dim + i;
      uint32_t lo[kVec / 2], hi[kVec / 2];
      if constexpr (kVec == 8) {
        *reinterpret_cast<uint4 *>(lo) = *reinterpret_cast<const uint4 *>(src);
        *reinterpret_cast<uint4 *>(hi) = *reinterpret_cast<const uint4 *>(src + half);
      } else {
        lo[0] = *reinterpret_cast<const uint32_t *>(src);
        hi[0] = *reinterpret_cast<const uint32_t *>(src + half);
      }
      uint16_t *dst;
      if (head < q_heads) dst = q + ((static_cast<size_t>(b) * q_heads + head) * seq + s) * head_dim;
      else if (head < q_heads + kv_heads) dst = k + ((static_cast<size_t>(b) * kv_heads + (head - q_heads)) * seq + s) * head_dim;
      else dst = v + ((static_cast<size_t>(b) * kv_heads + (head - q_heads - kv_heads)) * seq + s) * head_dim;
      const bool rotate = head < q_heads + kv_heads;
#pragma unroll
      for (int e = 0; e < kVec / 2; ++e) {
        const float2 a0 = angles[at + 2 * e], a1 = angles[at + 2 * e + 1];
        const float2 l = unpack2<kBf16>(lo[e]), h = unpack2<kBf16>(hi[e]);
        lo[e] = rotate ? pack2f<kBf16>(l.x * a0.y - h.x * a0.x, l.y * a1.y - h.y * a1.x) : pack2f<kBf16>(l.x, l.y);
        hi[e] = rotate ? pack2f<kBf16>(h.x * a0.y + l.x * a0.x, h.y * a1.y + l.y * a1.x) : pack2f<kBf16>(h.x, h.y);
      }
      if constexpr (kVec == 8) {
        *reinterpret_cast<uint4 *>(dst + i) = *reinterpret_cast<const uint4 *>(lo);
        *reinterpret_cast<uint4 *>(dst + i + half) = *reinterpret_cast<const uint4 *>(hi);
      } else {
        *reinterpret_cast<uint32_t *>(dst + i) = lo[0];
        *reinterpret_cast<uint32_t *>(dst + i + half) = hi[0];
      }
    }
  }
}

template <bool kBf16>
__global__ void __launch_bounds__(256) residual_add_kernel(const uint4 *a, const uint4 *b, uint4 *out, size_t chunks) {
  pdl_wait();
  pdl_launch_dependents();
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t c = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < chunks; c += stride) {
    const uint4 x = a[c], y = b[c];
    const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, yw[4] = {y.x, y.y, y.z, y.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 fx = unpack2<kBf16>(xw[i]), fy = unpack2<kBf16>(yw[i]);
      o[i] = pack2f<kBf16>(fx.x + fy.x, fx.y + fy.y);
    }
    out[c] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

wb200_status launch_rmsnorm(int format, const void *x, const void *gamma, void *y, int rows, int dim, float eps,
                            cudaStream_t stream, const void *addend, void *sum, bool beside) {
  if (format != WB200_BF16 && format != WB200_F16) return fail(WB200_ERR_UNSUPPORTED, "rmsnorm takes bf16 or f16 storage");
  if (rows <= 0 || dim <= 0 || dim % 8 != 0 || !aligned16(x) || !aligned16(gamma) || !aligned16(y) || !aligned16(addend) || !aligned16(sum))
    return fail(WB200_ERR_INVALID_ARGUMENT, "rmsnorm needs dim % 8 == 0 and 16-byte aligned buffers");
  const bool bf16 = format == WB200_BF16;
  const auto kernel = addend ? (bf16 ? rmsnorm_kernel<true, true> : rmsnorm_kernel<false, true>)
                             : (bf16 ? rmsnorm_kernel<true, false> : rmsnorm_kernel<false, false>);
  WB200_CUDA_CHECK(launch_ordered(kernel, rows, kNormThreads, 0, stream, !beside, static_cast<const uint16_t *>(x), static_cast<const uint16_t *>(addend),
                                    static_cast<uint16_t *>(sum), static_cast<const uint16_t *>(gamma), static_cast<uint16_t *>(y), dim, eps));
  return WB200_OK;
}

wb200_status launch_rope_split(int format, const void *qkv, void *q, void *k, void *v, int batch, int seq, int q_heads,
                               int kv_heads, int head_dim, float theta, int position_offset, cudaStream_t stream, bool beside) {
  if (format != WB200_BF16 && format != WB200_F16) return fail(WB200_ERR_UNSUPPORTED, "rope takes bf16 or f16 storage");
  if (batch <= 0 || seq <= 0 || q_heads <= 0 || kv_heads <= 0 || head_dim <= 0 || head_dim % 4 != 0 || !(theta > 0.f))
    return fail(WB200_ERR_INVALID_ARGUMENT, "invalid rope extents (head_dim % 4 == 0, theta > 0)");
  const int tokens = batch * seq;
  const float log2_theta = log2f(theta);
  const bool wide = head_dim % 16 == 0 && aligned16(qkv) && aligned16(q) && aligned16(k) && aligned16(v);
  const bool bf16 = format == WB200_BF16;
  const auto kernel = wide ? (bf16 ? rope_split_kernel<true, 8> : rope_split_kernel<false, 8>)
                           : (bf16 ? rope_split_kernel<true, 2> : rope_split_kernel<false, 2>);
  WB200_CUDA_CHECK(launch_ordered(kernel, tokens, kRopeThreads, 0, stream, !beside, static_cast<const uint16_t *>(qkv), static_cast<uint16_t *>(q),
                                    static_cast<uint16_t *>(k), static_cast<uint16_t *>(v), seq, q_heads, kv_heads, head_dim, log2_theta,
                                    position_offset));
  return WB200_OK;
}

wb200_status launch_residual_add(int format, const void *a, const void *b, void *out, size_t elements, cudaStream_t stream, bool beside) {
  if (format != WB200_BF16 && format != WB200_F16) return fail(WB200_ERR_UNSUPPORTED, "residual add takes bf16 or f16 storage");
  if (elements == 0 || elements % 8 != 0 || !aligned16(a) || !aligned16(b) || !aligned16(out))
    return fail(WB200_ERR_INVALID_ARGUMENT, "residual add needs a multiple of 8 elements and 16-byte aligned buffers");
  const size_t chunks = elements / 8;
  size_t blocks = (chunks + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  WB200_CUDA_CHECK(launch_ordered(format == WB200_BF16 ? residual_add_kernel<true> : residual_add_kernel<false>, static_cast<unsigned>(blocks), 256, 0,
                                    stream, !beside, static_cast<const uint4 *>(a), static_cast<const uint4 *>(b), static_cast<uint4 *>(out), chunks));
  return WB200_OK;
}

}  // namespace wb200
