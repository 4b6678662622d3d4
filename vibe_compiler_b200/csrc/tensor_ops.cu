// Managed-reference tensor commands on the device: elementwise, convert, reduce, and the physical
// tensor codec. Semantics follow lib/Wafer/Simulator/Reference/ManagedReferenceTargetModel.cpp:
// decode every operand to f32 (:137-155), apply one f32 operation (:230-299), encode with
// round-to-nearest-even (:157-185); NaN inputs or results are reported, not produced. Arithmetic
// uses the explicitly rounded intrinsics so the compiler cannot contract or reassociate.
#include "gemm_formal.cuh"
#include "kernels.h"
#include "formal_functions_f32.cuh"
#include "ptx_sm100.cuh"
#include "storage_walk.cuh"

namespace wb200 {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float apply_elementwise(int op, float x, float y) {
  switch (op) {
    case WB200_EW_ABS: return fabsf(x);
    case WB200_EW_NEG: return -x;
    case WB200_EW_RECIP: return __fdiv_rn(1.0f, x);
    case WB200_EW_SQUARE: return __fmul_rn(x, x);
    case WB200_EW_MAX: return fmaxf(x, y);
    case WB200_EW_MIN: return fminf(x, y);
    case WB200_EW_ADD: return __fadd_rn(x, y);
    case WB200_EW_SUB: return __fsub_rn(x, y);
    case WB200_EW_MUL: return __fmul_rn(x, y);
    case WB200_EW_RELU: return x < 0.0f ? 0.0f : x;
    case WB200_EW_SQRT: return __fsqrt_rn(x);
    case WB200_EW_RSQRT: return __fdiv_rn(1.0f, __fsqrt_rn(x));
    case WB200_EW_LOG2: return log2f(x);
    case WB200_EW_LN: return logf(x);
    case WB200_EW_POW2: return exp2f(x);
    case WB200_EW_EXP: return expf(x);
    case WB200_EW_EXPLP: return exp2f(__fmul_rn(x, 0x1.715476p+0f));
    case WB200_EW_SIN: return sinf(x);
    case WB200_EW_COS: return cosf(x);
    case WB200_EW_TANH: return tanhf(x);
    case WB200_EW_SIGMOID:
      if (x >= 0.0f) return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-x)));
      return __fdiv_rn(expf(x), __fadd_rn(1.0f, expf(x)));
    case WB200_EW_SOFTPLUS: return __fadd_rn(fmaxf(x, 0.0f), log1pf(expf(-fabsf(x))));
    default: return x;
  }
}

// Calls visit(src element, dst element, valid mask) for this thread's groups.
template <typename Visit>
__device__ __forceinline__ void walk_groups(const StorageWalk &w, Visit &&visit) {
  walk_groups(w, static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x, static_cast<int64_t>(gridDim.x) * blockDim.x, visit);
}
__device__ __forceinline__ void walk_load(const uint8_t *base, int64_t at, uint32_t valid, int format, uint32_t (&v)[8]) {
  if (valid == 0xffu) {
    load_group8(base, at >> 3, format == WB200_F32 ? 4 : 2, v);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = (valid >> e) & 1u ? load_element_bits(base, at + e, format) : 0u;
  }
}
__device__ __forceinline__ void walk_store(uint8_t *base, int64_t at, uint32_t valid, int format, const uint32_t (&v)[8]) {
  if (valid == 0xffu) {
    store_group8(base, at >> 3, format == WB200_F32 ? 4 : 2, v);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if ((valid >> e) & 1u) store_element_bits(base, at + e, format, v[e]);
  }
}

// Eight elements per thread with 128-bit accesses, the operation and the format fixed at compile time.
template <int kOp, int kFormat>
__global__ void __launch_bounds__(kThreads)
elementwise_walk_kernel(int input_count, const uint8_t *in0, const uint8_t *in1, uint8_t *dst, const StorageWalk walk, int *nan_flag) {
  bool saw_nan = false;
  walk_groups(walk, [&](int64_t at, int64_t, uint32_t valid) {
    uint32_t a[8], b[8], r[8];
    walk_load(in0, at, valid, kFormat, a);
    if (input_count > 1) walk_load(in1, at, valid, kFormat, b);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float x = widen_bits(a[e], kFormat), y = input_count > 1 ? widen_bits(b[e], kFormat) : 0.0f;
      const float result = apply_elementwise(kOp, x, y);
      saw_nan |= ((x != x) | (y != y) | (result != result)) && ((valid >> e) & 1u);
      r[e] = narrow_bits(result, kFormat);
    }
    walk_store(dst, at, valid, kFormat, r);
  });
  if (saw_nan) raise_status(nan_flag, 1);
}

template <int kSrc, int kDst>
__global__ void __launch_bounds__(kThreads)
convert_walk_kernel(const uint8_t *src, uint8_t *dst, const StorageWalk walk, int *nan_flag) {
  bool saw_nan = false;
  walk_groups(walk, [&](int64_t from, int64_t to, uint32_t valid) {
    uint32_t a[8], r[8];
    walk_load(src, from, valid, kSrc, a);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float x = widen_bits(a[e], kSrc);
      saw_nan |= (x != x);
      r[e] = narrow_bits(x, kDst);
    }
    walk_store(dst, to, valid, kDst, r);
  });
  if (saw_nan) raise_status(nan_flag, 1);
}

// Reduction of rank-4 NCx tensors [n, h, w, c] with many outputs, one thread per output element; the reduced coordinates
// are visited in row-major input order, which is the order the reference's running accumulator sees them (:412-447). The
// output index is split once with 32-bit divisions, and while the channel is kept the fold walks constant strides along n, h and w.
template <int kOp, int kFormat>
__global__ void __launch_bounds__(kThreads)
reduce_nhwc_kernel(const uint8_t *src, uint8_t *dst, const LayoutMap src_map, const LayoutMap dst_map, uint32_t reduced_mask, int *nan_flag) {
  const int64_t out_index = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (out_index >= dst_map.element_count) return;
  const uint32_t out_c = static_cast<uint32_t>(dst_map.shape[3]), out_w = static_cast<uint32_t>(dst_map.shape[2]), out_h = static_cast<uint32_t>(dst_map.shape[1]);
  const uint32_t index = static_cast<uint32_t>(out_index);
  const uint32_t pixel = index / out_c, c0 = index - pixel * out_c;
  const uint32_t row = pixel / out_w, w0 = pixel - row * out_w;
  const uint32_t n0 = row / out_h, h0 = row - n0 * out_h;
  const uint32_t n_count = (reduced_mask & 1u) ? static_cast<uint32_t>(src_map.shape[0]) : 1u, h_count = (reduced_mask & 2u) ? static_cast<uint32_t>(src_map.shape[1]) : 1u;
  const uint32_t w_count = (reduced_mask & 4u) ? static_cast<uint32_t>(src_map.shape[2]) : 1u, c_count = (reduced_mask & 8u) ? static_cast<uint32_t>(src_map.shape[3]) : 1u;
  const uint32_t in_w = static_cast<uint32_t>(src_map.shape[2]);
  float acc = kOp == WB200_RED_MAX ? -INFINITY : (kOp == WB200_RED_MIN ? INFINITY : 0.0f);
  bool saw_nan = false;
  auto step = [&](float value) {
    saw_nan |= (value != value);
    if (kOp == WB200_RED_SUM) {
      acc = __fadd_rn(acc, value);
    } else if (acc == 0.0f && value == 0.0f) {
      const bool negative = kOp == WB200_RED_MAX ? (signbit(acc) && signbit(value)) : (signbit(acc) || signbit(value));
      acc = negative ? -0.0f : 0.0f;
    } else {
      acc = kOp == WB200_RED_MAX ? fmaxf(acc, value) : fminf(acc, value);
    }
    saw_nan |= (acc != acc);
  };
  if (!(reduced_mask & 8u)) {
    const int64_t full_c = src_map.cx_blocks * src_map.c_block;
    const int64_t width = static_cast<int64_t>(c0) < full_c ? src_map.c_block : src_map.c0;
    const int64_t stride_h = width * in_w, stride_n = src_map.outer_slice_stride;
    const int64_t base = physical_index_nhwc(src_map, (reduced_mask & 1u) ? 0 : n0,
                                             static_cast<int64_t>((reduced_mask & 2u) ? 0u : h0) * in_w + ((reduced_mask & 4u) ? 0u : w0), c0);
    for (uint32_t n = 0; n < n_count; ++n)
      for (uint32_t h = 0; h < h_count; ++h) {
        const int64_t line = base + n * stride_n + h * stride_h;
#pragma unroll 8
        for (uint32_t w = 0; w < w_count; ++w) step(widen_bits(load_element_bits(src, line + w * width, kFormat), kFormat));
      }
  } else {
    for (uint32_t n = 0; n < n_count; ++n)
      for (uint32_t h = 0; h < h_count; ++h)
        for (uint32_t w = 0; w < w_count; ++w)
          for (uint32_t c = 0; c < c_count; ++c) {
            const int64_t in_n = (reduced_mask & 1u) ? n : n0;
            const uint32_t in_h = (reduced_mask & 2u) ? h : h0, in_wi = (reduced_mask & 4u) ? w : w0;
            step(widen_bits(load_element_bits(src, physical_index_nhwc(src_map, in_n, static_cast<int64_t>(in_h) * in_w + in_wi, c), kFormat), kFormat));
          }
  }
  store_element_bits(dst, physical_index_nhwc(dst_map, n0, static_cast<int64_t>(h0) * out_w + w0, c0), kFormat, narrow_bits(acc, kFormat));
  if (saw_nan) raise_status(nan_flag, 1);
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
codec_kernel(const T *src, T *dst, const LayoutMap map, int pack) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < map.element_count; i += stride) {
    const int64_t phys = physical_index(map, i);
    if (pack) dst[phys] = src[i];
    else dst[i] = src[phys];
  }
}
// The same in 16-byte units: with the channel count a multiple of the unit's elements, a unit never straddles a row, a
// channel block or the tail's width, so both sides are contiguous and aligned. 256 x 520 two-byte elements: 5.6 -> 2 us.
// `job` of a launch by blockIdx.y: the two operands of a GEMM travel together (both over PCIe when they lie in host memory).
struct CodecJob { const uint4 *src; uint4 *dst; LayoutMap map; uint32_t units; };
struct CodecJobs { CodecJob job[2]; };
template <int kUnit>
__global__ void __launch_bounds__(kThreads)
codec_wide_kernel(const __grid_constant__ CodecJobs jobs, int pack) {
  const CodecJob &job = jobs.job[blockIdx.y];
  const LayoutMap &map = job.map;
  const uint32_t row_units = static_cast<uint32_t>(map.shape[map.rank - 1]) / kUnit;
  const bool sliced = map.layout == WB200_LAYOUT_NCX && map.rank > 1;
  const uint32_t full_c = static_cast<uint32_t>(map.cx_blocks * map.c_block);
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < job.units; u += gridDim.x * blockDim.x) {
    uint32_t outer = u / row_units;
    const uint32_t c = (u - outer * row_units) * kUnit;
    int64_t at = 0;
    if (sliced) {
      const uint32_t slice = outer / static_cast<uint32_t>(map.block_outer_elements);
      outer -= slice * static_cast<uint32_t>(map.block_outer_elements);
      at = slice * map.outer_slice_stride;
    }
    if (c < full_c) {
      const uint32_t block = c / static_cast<uint32_t>(map.c_block);
      at += block * (map.block_outer_elements * map.c_block) + outer * map.c_block + (c - block * static_cast<uint32_t>(map.c_block));
    } else {
      at += map.cx_blocks * map.block_outer_elements * map.c_block + outer * map.c0 + (c - full_c);
    }
    if (pack) job.dst[at / kUnit] = job.src[u];
    else job.dst[u] = job.src[at / kUnit];
  }
}

// ------------------------------------------------------------------------------------------------ formal elementwise
// Bit-exact evaluation of the reference's formal elementwise family
// (lib/Wafer/Simulator/Reference/Formal/FormalNumericElementwise.cpp:23-248): arithmetic in the operand format with
// one RNE rounding, NaN results canonicalised (not rejected), relations to Bool or to 1.0 / 0.0, logic on "bits != 0",
// and the IEEE exception flags. Arithmetic runs in f32 and is narrowed once: for f16 / bf16 the double rounding is
// innocuous (24 >= 2 * 11 + 2), for f32 the hardware operation is the RNE operation. Inexactness comes from
// error-free transformations, not from a wider re-computation.
constexpr uint32_t kFlagInvalid = 1u, kFlagDivByZero = 2u, kFlagOverflow = 4u, kFlagUnderflow = 8u, kFlagInexact = 16u;

struct FormatTraits { uint32_t sign, exp_mask, mant_mask, quiet_bit, canonical_nan, one; int precision; float min_normal; };
// Folds (reduce, pooling): their chained f32 add steps take the early-return path too. Measured on 2^27 elements: NCx sum
// over w 0.418 ms with it, 0.458 ms without; 2x2 sum pooling 0.254 ms against 0.338 ms.
constexpr bool kFoldCommonCase = true;
__device__ __forceinline__ FormatTraits traits_of(int format) {
  if (format == WB200_F32) return {0x80000000u, 0x7f800000u, 0x007fffffu, 0x00400000u, 0x7fc00000u, 0x3f800000u, 24, 1.17549435e-38f};
  if (format == WB200_BF16) return {0x8000u, 0x7f80u, 0x007fu, 0x0040u, 0x7fc0u, 0x3f80u, 8, 1.17549435e-38f};
  return {0x8000u, 0x7c00u, 0x03ffu, 0x0200u, 0x7e00u, 0x3c00u, 11, 6.10351562e-05f};
}

// |value| rounded to `precision` bits with an unbounded exponent range is below the smallest normal number.
__device__ __forceinline__ bool tiny_after_rounding(double value, int precision, float min_normal) {
  if (value == 0.0) return false;
  int exponent;
  const double mantissa = frexp(fabs(value), &exponent);                 // [0.5, 1)
  const double rounded = ldexp(rint(ldexp(mantissa, precision)), exponent - precision);
  return rounded < static_cast<double>(min_normal);
}

// `common_case` false leaves out the early-return path of f32 add / sub / mul / square (see kFoldCommonCase).
__device__ __forceinline__ uint32_t formal_scalar(int op, int format, int out_format, uint32_t a, uint32_t b, uint32_t *flags_out,
                                                  bool common_case = true) {
  if (common_case && format == WB200_F32 && out_format == WB200_F32 && (op == WB200_EW_ADD || op == WB200_EW_SUB || op == WB200_EW_MUL || op == WB200_EW_SQUARE)) {
    // The common f32 case first: finite operands and a finite result that cannot be tiny. The arithmetic is the general
    // path's (same sum / product, same error-free residual), with its NaN, infinity, narrowing and underflow decisions
    // known in advance: a finite sum that is subnormal or zero is exact, and a product of at least 2^-100 is normal and
    // has a residual that one fused multiply-add yields exactly.
    const uint32_t second = op == WB200_EW_SQUARE ? a : b;
    if ((a & 0x7f800000u) != 0x7f800000u && (second & 0x7f800000u) != 0x7f800000u) {
      const float x = __uint_as_float(a);
      float r, residual;
      bool decided;
      if (op == WB200_EW_MUL || op == WB200_EW_SQUARE) {
        const float y = __uint_as_float(second);
        r = __fmul_rn(x, y);
        residual = __fmaf_rn(x, y, -r);
        decided = fabsf(r) >= 7.8886090522101181e-31f;
      } else {
        const float y = op == WB200_EW_SUB ? -__uint_as_float(second) : __uint_as_float(second);
        r = __fadd_rn(x, y);
        const float part = __fsub_rn(r, x);
        residual = __fadd_rn(__fsub_rn(x, __fsub_rn(r, part)), __fsub_rn(y, part));
        decided = true;
      }
      if (decided && fabsf(r) < __uint_as_float(0x7f800000u)) {
        *flags_out = residual != 0.f ? kFlagInexact : 0u;
        return __float_as_uint(r);
      }
    }
  }
  const FormatTraits t = traits_of(format);
  if (common_case && (format == WB200_F16 || format == WB200_BF16) && out_format == format &&
      (op == WB200_EW_ADD || op == WB200_EW_SUB || op == WB200_EW_MUL || op == WB200_EW_SQUARE)) {
    // The 16-bit common case: finite operands and a normal result. Same f32 sum / product, residual and single narrowing
    // as the general path. A small sum of two 16-bit values is exact, so only a product can be tiny after rounding, and
    // one of at least twice the smallest normal number (and at least 2^-100, for the exact residual) is not.
    const uint32_t second = op == WB200_EW_SQUARE ? a : b;
    if ((a & t.exp_mask) != t.exp_mask && (second & t.exp_mask) != t.exp_mask) {
      const float x = widen_bits(a, format);
      float r, residual;
      bool decided;
      if (op == WB200_EW_MUL || op == WB200_EW_SQUARE) {
        const float y = widen_bits(second, format);
        r = __fmul_rn(x, y);
        residual = __fmaf_rn(x, y, -r);
        decided = fabsf(r) >= 7.8886090522101181e-31f && fabsf(r) >= 2.0f * t.min_normal;
      } else {
        const float y = op == WB200_EW_SUB ? -widen_bits(second, format) : widen_bits(second, format);
        r = __fadd_rn(x, y);
        const float part = __fsub_rn(r, x);
        residual = __fadd_rn(__fsub_rn(x, __fsub_rn(r, part)), __fsub_rn(y, part));
        decided = true;
      }
      const uint32_t narrowed = narrow_bits(r, format);   // r is not a NaN: the operands are finite
      const uint32_t exponent = narrowed & t.exp_mask;
      if (decided && exponent != 0 && exponent != t.exp_mask) {
        *flags_out = (residual != 0.f || widen_bits(narrowed, format) != r) ? kFlagInexact : 0u;
        return narrowed;
      }
    }
  }
  if (op == WB200_EW_MAX || op == WB200_EW_MIN) {
    // Maximum / minimum as straight-line selects (no branch, so a fold's independent loads stay ahead of its chain):
    // a NaN operand gives the canonical NaN (invalid when it signals), two zeros give -0 only when the sign rule says
    // so, otherwise the operand the comparison picks. No rounding.
    const uint32_t magnitude_a = a & ~t.sign, magnitude_b = b & ~t.sign;
    const bool nan_a = magnitude_a > t.exp_mask, nan_b = magnitude_b > t.exp_mask;
    const bool signalling = (nan_a && !(a & t.quiet_bit)) || (nan_b && !(b & t.quiet_bit));
    const float x = widen_bits(a, format), y = widen_bits(b, format);
    const uint32_t picked = (op == WB200_EW_MAX ? x < y : x > y) ? b : a;
    const uint32_t zero = (op == WB200_EW_MAX ? (a & b) : (a | b)) & t.sign;
    *flags_out = signalling ? kFlagInvalid : 0u;
    return (nan_a || nan_b) ? t.canonical_nan : ((magnitude_a | magnitude_b) == 0 ? zero : picked);
  }
  uint32_t flags = 0;
  const bool binary = !(op == WB200_EW_ABS || op == WB200_EW_NEG || op == WB200_EW_RECIP || op == WB200_EW_SQUARE || op == WB200_EW_RELU);
  auto is_nan = [&](uint32_t v) { return (v & t.exp_mask) == t.exp_mask && (v & t.mant_mask) != 0; };
  auto is_snan = [&](uint32_t v) { return is_nan(v) && (v & t.quiet_bit) == 0; };
  auto is_zero = [&](uint32_t v) { return (v & ~t.sign) == 0; };
  auto is_inf = [&](uint32_t v) { return (v & ~t.sign) == t.exp_mask; };
  const bool nan = is_nan(a) || (binary && is_nan(b));
  if (is_snan(a) || (binary && is_snan(b))) flags |= kFlagInvalid;
  const float x = widen_bits(a, format), y = binary ? widen_bits(b, format) : 0.f;
  uint32_t result;
  if (op >= WB200_EW_EQ && op <= WB200_EW_LT) {
    bool truth;
    if (nan) truth = op == WB200_EW_NE;
    else switch (op) {
      case WB200_EW_EQ: truth = x == y; break;
      case WB200_EW_NE: truth = x != y; break;
      case WB200_EW_GE: truth = x >= y; break;
      case WB200_EW_GT: truth = x > y; break;
      case WB200_EW_LE: truth = x <= y; break;
      default: truth = x < y; break;
    }
    *flags_out = flags;
    if (out_format == WB200_BOOL) return truth ? 1u : 0u;
    return truth ? traits_of(out_format).one : 0u;
  }
  if (nan && (op == WB200_EW_ABS || op == WB200_EW_NEG || op == WB200_EW_MAX || op == WB200_EW_MIN || op == WB200_EW_RELU)) {
    *flags_out = flags;
    return t.canonical_nan;
  }
  switch (op) {
    case WB200_EW_ABS: result = a & ~t.sign; break;
    case WB200_EW_NEG: result = a ^ t.sign; break;
    case WB200_EW_RELU: result = ((a & t.sign) && !is_zero(a)) ? 0u : a; break;
    case WB200_EW_MAX:
    case WB200_EW_MIN:
      if (is_zero(a) && is_zero(b)) {
        const bool negative = op == WB200_EW_MAX ? ((a & t.sign) && (b & t.sign)) : ((a & t.sign) || (b & t.sign));
        result = negative ? t.sign : 0u;
      } else {
        const bool choose_rhs = op == WB200_EW_MAX ? x < y : x > y;
        result = choose_rhs ? b : a;
      }
      break;
    default: {
      // recip, square, add, sub, mul: one RNE rounding in the operand format
      float r32;
      double small_product = 0.0;   // the exact product where it is small enough to be tiny after rounding
      bool maybe_tiny = false;
      bool inexact32 = false, finite_inputs = !is_inf(a) && !(binary && is_inf(b)) && !nan;
      if (op == WB200_EW_RECIP) {
        r32 = __fdiv_rn(1.0f, x);
        if (!nan && is_zero(a)) flags |= kFlagDivByZero;
        // 1 / x is representable only when x is a power of two
        if (finite_inputs && !is_zero(a)) inexact32 = (__float_as_uint(fabsf(x)) & 0x007fffffu) != 0 && (__float_as_uint(fabsf(x)) & 0x7f800000u) != 0;
        if (finite_inputs && !is_zero(a) && (__float_as_uint(fabsf(x)) & 0x7f800000u) == 0)   // subnormal f32 operand: power of two iff one bit set
          inexact32 = (__float_as_uint(fabsf(x)) & (__float_as_uint(fabsf(x)) - 1u)) != 0;
      } else if (op == WB200_EW_ADD || op == WB200_EW_SUB) {
        const float yy = op == WB200_EW_SUB ? -y : y;
        r32 = __fadd_rn(x, yy);
        if (finite_inputs && isfinite(r32)) {
          const float bb = __fsub_rn(r32, x);
          const float err = __fadd_rn(__fsub_rn(x, __fsub_rn(r32, bb)), __fsub_rn(yy, bb));
          inexact32 = err != 0.f;
        }
      } else {
        const float yy = op == WB200_EW_SQUARE ? x : y;
        r32 = __fmul_rn(x, yy);
        const float magnitude = fabsf(r32);
        if (magnitude >= 7.8886090522101181e-31f && magnitude >= 2.0f * t.min_normal) {
          // |r32| >= 2^-100: the residual x * yy - r32 is a multiple of 2^-149, so one fused multiply-add yields it
          // exactly; and a product of at least twice the smallest normal number is never tiny after rounding.
          if (finite_inputs) inexact32 = __fmaf_rn(x, yy, -r32) != 0.f;
        } else {
          if (finite_inputs) inexact32 = static_cast<double>(r32) != static_cast<double>(x) * static_cast<double>(yy);
          // only a product below twice the smallest normal number can still be tiny after rounding; whether it is also
          // inexact is known once the result is narrowed (a 16-bit product is exact in f32 and inexact only after that)
          small_product = static_cast<double>(x) * static_cast<double>(yy);
          maybe_tiny = finite_inputs && fabs(small_product) < 2.0 * static_cast<double>(t.min_normal);
        }
      }
      if (r32 != r32) {
        if (!nan) flags |= kFlagInvalid;   // inf - inf, 0 * inf
        result = t.canonical_nan;
        break;
      }
      result = narrow_bits(r32, format);
      const bool inexact = inexact32 || widen_bits(result, format) != r32;
      if (finite_inputs && !(flags & kFlagDivByZero)) {
        if (is_inf(result)) flags |= kFlagOverflow | kFlagInexact;
        else if (inexact) {
          flags |= kFlagInexact;
          if ((result & t.exp_mask) == 0) flags |= kFlagUnderflow;   // subnormal or zero after rounding, and inexact
          else if (maybe_tiny && tiny_after_rounding(small_product, t.precision, t.min_normal)) flags |= kFlagUnderflow;   // rounded up to the smallest normal
        }
      }
      break;
    }
  }
  *flags_out = flags;
  return result;
}

// Correctly rounded unary functions of the reference's MPFR family for the 16-bit formats
// (lib/Wafer/Simulator/Reference/Numeric/MPFRNumeric.cpp:560-682: the function evaluated exactly, rounded once to
// nearest-even with gradual underflow; sigmoid and softplus as whole functions, :372-470). The value is computed in
// f64 (a few ulp of f64) and narrowed with a single rounding (f64 -> f32 with round-to-odd, then RNE to 11 or 8 bits);
// a misrounding needs the true value within 2^-50 of a rounding boundary of a 16-bit format, and the complete input
// space (65 536 operands per function and format) is checked against a 200-bit evaluation. binary32 and TF32 operands
// take the two-step evaluation of formal_functions_f32.cuh.
__device__ __forceinline__ uint32_t narrow_from_double(double value, int format) {
  float f = __double2float_rz(value);
  if (static_cast<double>(f) != value && isfinite(f)) f = __uint_as_float(__float_as_uint(f) | 1u);   // sticky bit: round to odd
  return narrow_bits(f, format);
}

__device__ uint32_t formal_mpfr_scalar(int op, int format, uint32_t a, uint32_t *flags_out) {
  if (format == WB200_F32 || format == WB200_TF32) {
    // binary32 and TF32 operands: binary64 evaluation with a rounding test and a double-double second step
    // (formal_functions_f32.cuh). TF32 keeps its 19 significant bits in storage bits 31..13; the low bits are ignored.
    int function;
    switch (op) {
      case WB200_EW_SQRT: function = ff32::kSqrt; break;
      case WB200_EW_RSQRT: function = ff32::kRsqrt; break;
      case WB200_EW_LOG2: function = ff32::kLog2; break;
      case WB200_EW_LN: function = ff32::kLn; break;
      case WB200_EW_POW2: function = ff32::kPow2; break;
      case WB200_EW_EXP: function = ff32::kExp; break;
      case WB200_EW_SIN: function = ff32::kSin; break;
      case WB200_EW_COS: function = ff32::kCos; break;
      case WB200_EW_TANH: function = ff32::kTanh; break;
      case WB200_EW_SIGMOID: function = ff32::kSigmoid; break;
      default: function = ff32::kSoftplus; break;
    }
    const bool tf32 = format == WB200_TF32;
    return ff32::correctly_rounded(function, tf32, tf32 ? (a & 0xffffe000u) : a, flags_out, nullptr);
  }
  const FormatTraits t = traits_of(format);
  uint32_t flags = 0;
  const bool nan = (a & t.exp_mask) == t.exp_mask && (a & t.mant_mask) != 0;
  if (nan) {
    *flags_out = (a & t.quiet_bit) ? 0u : kFlagInvalid;
    return t.canonical_nan;
  }
  const bool negative = (a & t.sign) != 0, zero = (a & ~t.sign) == 0, inf = (a & ~t.sign) == t.exp_mask;
  const double x = static_cast<double>(widen_bits(a, format));
  const uint32_t pos_inf = t.exp_mask, neg_inf = t.exp_mask | t.sign;
  auto finish = [&](uint32_t bits, uint32_t f) { *flags_out = f; return bits; };
  double value;
  bool exact = false;
  switch (op) {
    case WB200_EW_SQRT:
      if (zero) return finish(a, 0);                                   // sqrt(-0) = -0
      if (negative) return finish(t.canonical_nan, kFlagInvalid);
      if (inf) return finish(pos_inf, 0);
      value = sqrt(x);
      exact = fma(value, value, -x) == 0.0;
      break;
    case WB200_EW_RSQRT:
      if (zero) return finish(negative ? neg_inf : pos_inf, kFlagDivByZero);
      if (negative) return finish(t.canonical_nan, kFlagInvalid);
      if (inf) return finish(0u, 0);
      value = 1.0 / sqrt(x);
      { int e; exact = frexp(x, &e) == 0.5 && ((e - 1) & 1) == 0; }      // x = 4^k
      break;
    case WB200_EW_LOG2:
    case WB200_EW_LN:
      if (zero) return finish(neg_inf, kFlagDivByZero);
      if (negative) return finish(t.canonical_nan, kFlagInvalid);
      if (inf) return finish(pos_inf, 0);
      if (op == WB200_EW_LOG2) { int e; const bool power = frexp(x, &e) == 0.5; value = power ? static_cast<double>(e - 1) : log2(x); exact = power; }
      else { value = log(x); exact = x == 1.0; }
      break;
    case WB200_EW_POW2:
    case WB200_EW_EXP:
      if (inf) return finish(negative ? 0u : pos_inf, 0);
      value = op == WB200_EW_POW2 ? exp2(x) : exp(x);
      exact = op == WB200_EW_POW2 ? (x == rint(x)) : zero;
      break;
    case WB200_EW_SIN:
    case WB200_EW_COS:
      if (inf) return finish(t.canonical_nan, kFlagInvalid);
      if (zero) return finish(op == WB200_EW_SIN ? a : t.one, 0);
      value = op == WB200_EW_SIN ? sin(x) : cos(x);
      break;
    case WB200_EW_TANH:
      if (zero) return finish(a, 0);
      if (inf) return finish(negative ? (t.one | t.sign) : t.one, 0);
      value = tanh(x);
      break;
    case WB200_EW_SIGMOID:
      if (inf) return finish(negative ? 0u : t.one, 0);
      if (zero) return finish(narrow_bits(0.5f, format), 0);
      value = x >= 0.0 ? 1.0 / (1.0 + exp(-x)) : exp(x) / (1.0 + exp(x));
      break;
    default:   // softplus = ln(1 + e^x)
      if (inf) return finish(negative ? 0u : pos_inf, 0);
      value = x > 0.0 ? x + log1p(exp(-x)) : log1p(exp(x));
      break;
  }
  const uint32_t bits = narrow_from_double(value, format);
  // Every exactly infinite result was returned above, so an infinite result here is an overflow; 2^x, e^x, sigmoid
  // and softplus are never exactly zero, so a zero result of theirs is an underflow (this also covers an f64
  // evaluation that saturated, e.g. 2^1904 or 2^-2000 with an integer operand).
  const bool never_zero = op == WB200_EW_POW2 || op == WB200_EW_EXP || op == WB200_EW_SIGMOID || op == WB200_EW_SOFTPLUS;
  if ((bits & ~t.sign) == t.exp_mask) flags |= kFlagOverflow | kFlagInexact;
  else if ((bits & ~t.sign) == 0 && never_zero) flags |= kFlagUnderflow | kFlagInexact;
  else if (!exact || static_cast<double>(widen_bits(bits, format)) != value) {
    flags |= kFlagInexact;
    if (tiny_after_rounding(value, t.precision, t.min_normal)) flags |= kFlagUnderflow;
  }
  return finish(bits, flags);
}

__device__ __forceinline__ uint32_t formal_load(const uint8_t *base, int format, const LayoutMap &map, int64_t i) {
  if (format == WB200_BOOL) return (base[i >> 3] >> (i & 7)) & 1u;   // bit-packed, least significant bit first
  return load_element_bits(base, physical_index(map, i), format);
}

// One thread per 8 consecutive logical elements, so that a bit-packed Bool destination byte has a single writer.
// kLinear: every tensor is in Tensor / NTensor layout (physical index == logical index); with `vector` set (all
// pointers 16-byte aligned) full groups then move with 128-bit accesses and no layout arithmetic at all.
// kOp >= 0 fixes the operation and the operand format at compile time (the arithmetic and relation families in linear
// layout): the generic evaluator then folds to a few dozen instructions instead of its whole decision tree.
// The groups first_group, first_group + group_stride, ... of one command; returns the OR of the elements' flags. The
// command's own kernel walks the groups with its whole grid, a command run (formal_run_kernel) with one block.
template <bool kLinear, int kOp, int kFormat>
__device__ __forceinline__ uint32_t
formal_elementwise_groups(int runtime_op, int runtime_format, int out_format, int input_count, const uint8_t *in0, const uint8_t *in1, uint8_t *dst,
                          const LayoutMap &in_map, const LayoutMap &out_map, const RhsBroadcast rhs, int vector, int64_t first_group,
                          int64_t group_stride) {
  const int op = kOp >= 0 ? kOp : runtime_op, in_format = kOp >= 0 ? kFormat : runtime_format;
  const int64_t total = out_map.element_count;
  const int64_t groups = (total + 7) / 8;
  const int64_t stride = group_stride;
  uint32_t flags = 0;
  const bool logic = op >= WB200_EW_LOGIC_NOT && op <= WB200_EW_LOGIC_XOR;
  const bool mpfr_family = op == WB200_EW_SQRT || op == WB200_EW_RSQRT || (op >= WB200_EW_LOG2 && op <= WB200_EW_EXP) ||
                           (op >= WB200_EW_SIN && op <= WB200_EW_SIGMOID) || op == WB200_EW_SOFTPLUS;
  const int in_bytes = format_bits(in_format) / 8, out_bytes = format_bits(out_format) / 8;   // 0 for Bool
  const bool same_rhs = input_count > 1 && rhs.mode == WB200_RHS_SAME;
  const bool scalar_rhs = input_count > 1 && rhs.mode == WB200_RHS_SCALAR;   // decided once, not per element
  if (kOp < 0 && mpfr_family) {
    // The correctly rounded functions cost hundreds to thousands of instructions per element: one element per thread
    // and step (first_group / group_stride are then the thread's index and the thread count), so that a short vector
    // spreads over as many threads as it has elements. Unary, float in and out: no Bool packing to respect.
    for (int64_t i = first_group; i < total; i += stride) {
      const uint32_t a = kLinear ? load_element_bits(in0, i, in_format) : formal_load(in0, in_format, in_map, i);
      uint32_t element_flags = 0;
      const uint32_t value = formal_mpfr_scalar(op, in_format, a, &element_flags);
      flags |= element_flags;
      store_element_bits(dst, kLinear ? i : physical_index(out_map, i), out_format, value);
    }
    return flags;
  }
  for (int64_t g = first_group; g < groups; g += stride) {
    const int64_t first = g * 8;
    const int count = total - first < 8 ? static_cast<int>(total - first) : 8;
    const bool wide = kLinear && vector && count == 8;
    uint32_t a[8], b[8], value[8];
    if (wide && in_bytes) {
      load_group8(in0, g, in_bytes, a);
      if (same_rhs) load_group8(in1, g, in_bytes, b);
    } else if (wide) {   // packed Bool operands: one byte holds the group
      const uint32_t byte_a = in0[g], byte_b = same_rhs ? in1[g] : 0u;
#pragma unroll
      for (int e = 0; e < 8; ++e) { a[e] = (byte_a >> e) & 1u; b[e] = (byte_b >> e) & 1u; }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (e >= count) break;
      const int64_t i = first + e;
      if (!wide) a[e] = kLinear ? (in_format == WB200_BOOL ? (in0[i >> 3] >> (i & 7)) & 1u : load_element_bits(in0, i, in_format))
                                : formal_load(in0, in_format, in_map, i);
      if (scalar_rhs) {
        b[e] = rhs.parameter;
      } else if (input_count > 1 && !(wide && same_rhs)) {
        // Second-operand forms of lib/Wafer/Simulator/Kernel/TargetModelTensorNumeric.cpp:347-372.
        int64_t j = i;
        if (rhs.mode == WB200_RHS_UNIT) j = i % rhs.parameter;
        else if (rhs.mode == WB200_RHS_GROUP) j = i / rhs.parameter * 64 + i % 64;
        b[e] = kLinear ? (in_format == WB200_BOOL ? (in1[j >> 3] >> (j & 7)) & 1u : load_element_bits(in1, j, in_format))
                       : formal_load(in1, in_format, in_map, j);
      } else if (input_count <= 1) {
        b[e] = 0u;
      }
      uint32_t element_flags = 0;
      if (logic) {
        const bool lhs = a[e] != 0, rhs_bit = b[e] != 0;
        value[e] = op == WB200_EW_LOGIC_NOT ? !lhs : op == WB200_EW_LOGIC_AND ? (lhs && rhs_bit) : op == WB200_EW_LOGIC_OR ? (lhs || rhs_bit) : (lhs != rhs_bit);
      } else if (mpfr_family) {
        value[e] = formal_mpfr_scalar(op, in_format, a[e], &element_flags);
      } else {
        value[e] = formal_scalar(op, in_format, out_format, a[e], b[e], &element_flags);
      }
      flags |= element_flags;
    }
    if (out_format == WB200_BOOL) {
      uint32_t packed = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (e < count) packed |= (value[e] & 1u) << e;
      const uint32_t keep = count == 8 ? 0u : (0xffu << count) & 0xffu;   // bits past the tensor keep the template's value
      dst[g] = static_cast<uint8_t>(keep ? ((dst[g] & keep) | packed) : packed);
    } else if (wide) {
      store_group8(dst, g, out_bytes, value);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (e < count) store_element_bits(dst, kLinear ? first + e : physical_index(out_map, first + e), out_format, value[e]);
    }
  }
  return flags;
}

template <bool kLinear, int kOp, int kFormat>
__global__ void __launch_bounds__(kThreads)
formal_elementwise_kernel(int runtime_op, int runtime_format, int out_format, int input_count, const uint8_t *in0, const uint8_t *in1, uint8_t *dst,
                          const LayoutMap in_map, const LayoutMap out_map, const RhsBroadcast rhs, int vector, uint32_t *flags_word) {
  const uint32_t flags = formal_elementwise_groups<kLinear, kOp, kFormat>(
      runtime_op, runtime_format, out_format, input_count, in0, in1, dst, in_map, out_map, rhs, vector,
      static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x, static_cast<int64_t>(gridDim.x) * blockDim.x);
  merge_block_flags(flags_word, flags);
}

// Short vectors in linear layouts: one element per thread in blocks of 128, 32-bit indexes. With eight elements per thread a
// Tile-sized vector runs on a handful of warps that evaluate their elements one after the other (4096 f32: 3.7 -> 2 us; a
// repeated-unit operand also lost its 64-bit remainders). Bool operands and results stay with the group kernel.
constexpr int kShortVector = 1 << 15, kShortThreads = 128;
__device__ __forceinline__ uint32_t rhs_bits(const uint8_t *in1, const RhsBroadcast &rhs, uint32_t i, int format) {
  if (rhs.mode == WB200_RHS_SCALAR) return rhs.parameter;
  if (rhs.mode == WB200_RHS_UNIT) i %= rhs.parameter;
  else if (rhs.mode == WB200_RHS_GROUP) i = i / rhs.parameter * 64u + i % 64u;
  return load_element_bits(in1, i, format);
}
template <int kOp, int kFormat>
__global__ void __launch_bounds__(kShortThreads)
formal_elementwise_short_kernel(int out_format, int input_count, const uint8_t *in0, const uint8_t *in1, uint8_t *dst, uint32_t count,
                                const RhsBroadcast rhs, uint64_t tile_stride, uint32_t *flags_word) {
  const uint32_t i = blockIdx.x * kShortThreads + threadIdx.x;
  uint32_t flags = 0;
  const uint64_t tile_offset = blockIdx.z * tile_stride;
  in0 += tile_offset;
  in1 += tile_offset;   // read only where there is one
  dst += tile_offset;
  pdl_launch_dependents();
  pdl_wait();
  if (i < count) {
    const uint32_t a = load_element_bits(in0, i, kFormat), b = input_count > 1 ? rhs_bits(in1, rhs, i, kFormat) : 0u;
    store_element_bits(dst, i, out_format, formal_scalar(kOp, kFormat, out_format, a, b, &flags));
  }
  merge_block_flags(flags_word, flags);
}

// The correctly rounded functions in linear layouts, one element per thread, the function fixed at compile time: one
// evaluator instead of eleven behind a switch, so a block's code fits the instruction cache. kSingle: binary32 and TF32.
template <int kOp, bool kSingle>
__global__ void __launch_bounds__(kShortThreads)
formal_function_kernel(int format, const uint8_t *in0, uint8_t *dst, int64_t count, uint64_t tile_stride, uint32_t *flags_word) {
  uint32_t flags = 0;
  in0 += blockIdx.z * tile_stride;
  dst += blockIdx.z * tile_stride;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kShortThreads;
  const int fixed = kSingle ? (format == WB200_TF32 ? WB200_TF32 : WB200_F32) : (format == WB200_BF16 ? WB200_BF16 : WB200_F16);
  pdl_launch_dependents();
  pdl_wait();
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * kShortThreads + threadIdx.x; i < count; i += stride) {
    uint32_t element_flags = 0;
    const uint32_t value = formal_mpfr_scalar(kOp, fixed, load_element_bits(in0, i, fixed), &element_flags);
    flags |= element_flags;
    store_element_bits(dst, i, fixed, value);
  }
  merge_block_flags(flags_word, flags);
}

// One step of a chain on a thread's kPer (8 or 1) values. The switch gives every arithmetic operation its own copy of the scalar
// evaluator with the operation and format fixed at compile time (a few dozen instructions each); only the cases a chain
// uses are ever fetched. The correctly rounded function family is one out-of-line call.
template <int kFormat, int kPer>
__device__ __forceinline__ void chain_step(int op, uint32_t (&value)[kPer], const uint32_t (&b)[kPer], int count, uint32_t &flags) {
#define WB200_CHAIN_CASE(OP)                                                             \
  case OP:                                                                               \
    _Pragma("unroll") for (int e = 0; e < kPer; ++e) {                                   \
      if (e < count) {                                                                   \
        uint32_t element_flags = 0;                                                      \
        value[e] = formal_scalar(OP, kFormat, kFormat, value[e], b[e], &element_flags);  \
        flags |= element_flags;                                                          \
      }                                                                                  \
    }                                                                                    \
    break;
  switch (op) {
    WB200_CHAIN_CASE(WB200_EW_ABS) WB200_CHAIN_CASE(WB200_EW_NEG) WB200_CHAIN_CASE(WB200_EW_RELU) WB200_CHAIN_CASE(WB200_EW_RECIP)
    WB200_CHAIN_CASE(WB200_EW_SQUARE) WB200_CHAIN_CASE(WB200_EW_MAX) WB200_CHAIN_CASE(WB200_EW_MIN) WB200_CHAIN_CASE(WB200_EW_ADD)
    WB200_CHAIN_CASE(WB200_EW_SUB) WB200_CHAIN_CASE(WB200_EW_MUL)
    default:
#pragma unroll 1
      for (int e = 0; e < count; ++e) {
        uint32_t element_flags = 0;
        value[e] = formal_mpfr_scalar(op, kFormat, value[e], &element_flags);
        flags |= element_flags;
      }
      break;
  }
#undef WB200_CHAIN_CASE
}

// A chain of formal elementwise commands (see ElementwiseChain): the running value stays in registers, every step's
// destination is still written, second operands are read where the step names one. A thread owns the same kPer
// elements of every vector, so a step may read what an earlier step of the chain wrote at the same address. One element
// per thread where the vector is short or the chain holds a correctly rounded function (whose eight evaluations in a row
// made a 64-element subtract - exp - multiply chain take 67 us; it takes 4).
template <int kFormat, int kPer>
__global__ void __launch_bounds__(kPer == 1 ? kShortThreads : kThreads)
formal_chain_kernel(const ElementwiseChain chain, int vector, uint64_t tile_stride, uint32_t *flags_word) {
  pdl_launch_dependents();
  pdl_wait();
  const uint64_t tile_offset = blockIdx.z * tile_stride;
  constexpr int format = kFormat, bytes = kFormat == WB200_F32 ? 4 : 2;
  const int64_t total = chain.count, groups = (total + kPer - 1) / kPer;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  uint32_t flags = 0;
  for (int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; g < groups; g += stride) {
    const int64_t first = g * kPer;
    const int count = total - first < kPer ? static_cast<int>(total - first) : kPer;
    const bool wide = kPer == 8 && vector && count == 8;
    uint32_t value[kPer], b[kPer];
#pragma unroll 1
    for (int s = 0; s < chain.steps; ++s) {
      if (chain.step[s].lhs) {
        const uint8_t *lhs = chain.step[s].lhs + tile_offset;
        if (wide) {
          if constexpr (kPer == 8) load_group8(lhs, g, bytes, value);
        } else {
#pragma unroll
          for (int e = 0; e < kPer; ++e) value[e] = e < count ? load_element_bits(lhs, first + e, format) : 0u;
        }
      }
      const uint8_t *rhs = chain.step[s].rhs + tile_offset;   // read only where there is one
      uint8_t *dst = chain.step[s].dst + tile_offset;
      if (chain.step[s].rhs_mode == WB200_RHS_SAME) {
        if (wide) {
          if constexpr (kPer == 8) load_group8(rhs, g, bytes, b);
        } else {
#pragma unroll
          for (int e = 0; e < kPer; ++e) b[e] = e < count ? load_element_bits(rhs, first + e, format) : 0u;
        }
      } else if (chain.step[s].rhs_mode == WB200_RHS_UNIT) {
#pragma unroll
        for (int e = 0; e < kPer; ++e)   // a command has fewer than 2^32 elements
          b[e] = e < count ? load_element_bits(rhs, static_cast<uint32_t>(first + e) % chain.step[s].scalar, format) : 0u;
      } else {
#pragma unroll
        for (int e = 0; e < kPer; ++e) b[e] = chain.step[s].scalar;
      }
      chain_step<kFormat, kPer>(chain.step[s].op, value, b, count, flags);
      if (wide) {
        if constexpr (kPer == 8) store_group8(dst, g, bytes, value);
      } else {
#pragma unroll
        for (int e = 0; e < kPer; ++e)
          if (e < count) store_element_bits(dst, first + e, format, value[e]);
      }
    }
  }
  merge_block_flags(flags_word, flags);
}

// The same fold for rank-4 NCx tensors [n, h, w, c] (every TargetCall-level reduce): coordinates are carried as loop
// counters, so the only divisions are the three that split the output index.
template <int kCombine, int kFormat>
__device__ __forceinline__ uint32_t formal_reduce_nhwc_output(const uint8_t *src, uint8_t *dst, const LayoutMap &src_map, const LayoutMap &dst_map,
                                                              uint32_t reduced_mask, int64_t out_index) {
  constexpr int format = kFormat, combine = kCombine;
  uint32_t block_flags_in = 0;
  if (out_index < dst_map.element_count) {
  const uint32_t out_c = static_cast<uint32_t>(dst_map.shape[3]), out_w = static_cast<uint32_t>(dst_map.shape[2]), out_h = static_cast<uint32_t>(dst_map.shape[1]);
  const uint32_t index = static_cast<uint32_t>(out_index);    // the launcher admits at most 2^32 - 1 outputs
  const uint32_t pixel = index / out_c, c0 = index - pixel * out_c;
  const uint32_t row = pixel / out_w, w0 = pixel - row * out_w;
  const uint32_t n0 = row / out_h, h0 = row - n0 * out_h;
  // dimension d is bit d of the mask; a reduced dimension runs over its whole input extent from 0
  const uint32_t n_count = (reduced_mask & 1u) ? static_cast<uint32_t>(src_map.shape[0]) : 1u, h_count = (reduced_mask & 2u) ? static_cast<uint32_t>(src_map.shape[1]) : 1u;
  const uint32_t w_count = (reduced_mask & 4u) ? static_cast<uint32_t>(src_map.shape[2]) : 1u, c_count = (reduced_mask & 8u) ? static_cast<uint32_t>(src_map.shape[3]) : 1u;
  const uint32_t in_w = static_cast<uint32_t>(src_map.shape[2]);
  const uint32_t infinity = format == WB200_F32 ? 0x7f800000u : format == WB200_BF16 ? 0x7f80u : 0x7c00u;
  const uint32_t sign = format == WB200_F32 ? 0x80000000u : 0x8000u;
  uint32_t accumulator = combine == WB200_EW_ADD ? 0u : combine == WB200_EW_MAX ? (infinity | sign) : infinity;
  uint32_t flags = 0;
  if (!(reduced_mask & 8u)) {
    // The channel is kept: along n, h and w the physical address moves by constant strides (one channel block is
    // `width` elements wide), so the fold is three strided loops whose loads do not depend on one another.
    const int64_t full_c = src_map.cx_blocks * src_map.c_block;
    const int64_t width = static_cast<int64_t>(c0) < full_c ? src_map.c_block : src_map.c0;
    const int64_t stride_w = width, stride_h = width * in_w, stride_n = src_map.outer_slice_stride;
    const int64_t base = physical_index_nhwc(src_map, (reduced_mask & 1u) ? 0 : n0,
                                             static_cast<int64_t>((reduced_mask & 2u) ? 0u : h0) * in_w + ((reduced_mask & 4u) ? 0u : w0), c0);
    for (uint32_t n = 0; n < n_count; ++n)
      for (uint32_t h = 0; h < h_count; ++h) {
        const int64_t row = base + n * stride_n + h * stride_h;
#pragma unroll 8
        for (uint32_t w = 0; w < w_count; ++w) {
          uint32_t step_flags = 0;
          accumulator = formal_scalar(combine, format, format, accumulator, load_element_bits(src, row + w * stride_w, format), &step_flags, kFoldCommonCase);
          flags |= step_flags;
        }
      }
  } else {
    for (uint32_t n = 0; n < n_count; ++n)
      for (uint32_t h = 0; h < h_count; ++h)
        for (uint32_t w = 0; w < w_count; ++w)
          for (uint32_t c = 0; c < c_count; ++c) {
            const int64_t in_n = (reduced_mask & 1u) ? n : n0;
            const uint32_t in_h = (reduced_mask & 2u) ? h : h0, in_wi = (reduced_mask & 4u) ? w : w0;
            uint32_t step_flags = 0;
            const uint32_t value = load_element_bits(src, physical_index_nhwc(src_map, in_n, static_cast<int64_t>(in_h) * in_w + in_wi, c), format);
            accumulator = formal_scalar(combine, format, format, accumulator, value, &step_flags, kFoldCommonCase);
            flags |= step_flags;
          }
  }
  store_element_bits(dst, physical_index_nhwc(dst_map, n0, static_cast<int64_t>(h0) * out_w + w0, c0), format, accumulator);
  block_flags_in = flags;
  }
  return block_flags_in;
}
template <int kCombine, int kFormat>
__global__ void __launch_bounds__(kThreads)
formal_reduce_nhwc_kernel(const uint8_t *src, uint8_t *dst, const LayoutMap src_map, const LayoutMap dst_map,
                          uint32_t reduced_mask, uint32_t *flags_word) {
  const uint32_t flags = formal_reduce_nhwc_output<kCombine, kFormat>(src, dst, src_map, dst_map, reduced_mask,
                                                                     static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x);
  merge_block_flags(flags_word, flags);
}

// Reductions with few outputs, and those of any rank and layout. The fold of an output is a chain in row-major input order
// (managed: ManagedReferenceTargetModel.cpp:412-447; formal: lib/Wafer/Simulator/Reference/Numeric/FormalTensorNumeric.cpp:
// 363-425 with the step of Reference/Formal/FormalNumericReduce.cpp:12-67: from +0 (sum) or -inf / +inf (max / min), NaNs
// canonicalised, IEEE flags of every step collected), so parallelism is over outputs only, and a thread that also fetches
// its own inputs waits for memory once per unrolled batch. Here a block folds 32 outputs: its 256 threads fetch 64 inputs of
// each ahead of the fold (registers, then one of two shared-memory panels), and one warp runs the chains from shared memory.
// A chunk is first folded without any branch - plain additions with the error-free residual OR-ed up, or integer maxima of
// order-preserving keys (-0 below +0, as the step's zero rule has it) - and repeated with the full step only if it met a NaN
// or an infinity. Measured (device time, f32 sum): 520 chains of 256 274 -> 4 us; formal, 64 chains of 64: 18.6 -> 3 us.
struct FoldPlan {
  LayoutMap src, dst;
  uint32_t reduced_mask, steps;
  int count;                  // reduced dimensions, slowest first
  uint32_t size[3];
  int kind[3];                // 0 NCx slice, 1 outer (row-major index over the dimensions before the channel), 2 channel
  int64_t outer_step[3];
  int along_steps;            // consecutive steps are neighbours in memory (the channel is reduced)
};
constexpr int kFoldOutputs = 32, kFoldChunk = 64, kFoldPerThread = kFoldOutputs * kFoldChunk / kThreads;

__device__ __forceinline__ int64_t fold_address(const LayoutMap &m, int64_t slice, int64_t outer, int64_t c) {
  if (m.layout == WB200_LAYOUT_TENSOR || m.layout == WB200_LAYOUT_NTENSOR) return outer * m.shape[m.rank - 1] + c;
  return physical_index_nhwc(m, slice, outer, c);
}

// Address arithmetic and the rare full step are out of line: these kernels run for a few microseconds between others, so the
// instructions they fetch count as much as those they execute.
__device__ __noinline__ void fold_kept_coordinates(const FoldPlan &plan, int64_t output, int64_t *slice_out, int64_t *outer_out, int64_t *c_out, int64_t *dst_at) {
  // coordinates the output keeps (the reduced ones are zero), and where it is stored; 64-bit divisions only where needed
  int64_t remaining = output, outer = 0, slice = 0, c = 0, scale = 1, dst_outer = 0, dst_scale = 1;
  const int rank = plan.src.rank;
  const bool sliced = plan.src.layout == WB200_LAYOUT_NCX && rank > 1, narrow = plan.dst.element_count < (1ll << 31);
#pragma unroll 1
  for (int d = rank - 1; d >= 0; --d) {
    const bool reduced = (plan.reduced_mask >> d) & 1u;
    const int64_t extent = plan.src.shape[d];
    int64_t coord = 0;
    if (!reduced) {
      const int64_t quotient = narrow ? static_cast<uint32_t>(remaining) / static_cast<uint32_t>(extent) : remaining / extent;
      coord = remaining - quotient * extent;
      remaining = quotient;
    }
    if (d == rank - 1) c = coord;
    else if (d == 0 && sliced) slice = coord;
    else {
      outer += coord * scale;
      scale *= extent;
      dst_outer += coord * dst_scale;
      if (!reduced) dst_scale *= extent;
    }
  }
  *slice_out = slice; *outer_out = outer; *c_out = c;
  *dst_at = fold_address(plan.dst, slice, dst_outer, c);
}
__device__ __noinline__ int64_t fold_element(const FoldPlan &plan, int64_t slice, int64_t outer, int64_t c, uint32_t step) {
#pragma unroll 1
  for (int d = plan.count - 1; d >= 0; --d) {
    const uint32_t quotient = step / plan.size[d], coord = step - quotient * plan.size[d];
    step = quotient;
    if (plan.kind[d] == 2) c += coord;
    else if (plan.kind[d] == 1) outer += coord * plan.outer_step[d];
    else slice += coord;
  }
  return fold_address(plan.src, slice, outer, c);
}
template <int kCombine, int kFormat>
__device__ __noinline__ uint32_t fold_full_steps(const uint32_t *column, int stride, int count, uint32_t acc, uint32_t *flags) {
#pragma unroll 1
  for (int s = 0; s < count; ++s) {
    uint32_t step_flags = 0;
    acc = formal_scalar(kCombine, kFormat, kFormat, acc, column[s * stride], &step_flags, kFoldCommonCase);
    *flags |= step_flags;
  }
  return acc;
}

// The chains of a block: `fetch(base, v)` loads this thread's inputs of the chunk at step `base`, `place(i, out, step)` says
// which output and step element i is. The result of output `tid` is returned in threads tid < outputs.
template <bool kFormal, int kCombine, int kFormat, typename Fetch, typename Place>
__device__ __forceinline__ uint32_t fold_block(uint32_t steps, int outputs, Fetch &&fetch, Place &&place, uint32_t &flags, bool &saw_nan) {
  static_assert(kCombine != WB200_EW_ADD || kFormat == WB200_F32, "sums are f32");
  __shared__ uint32_t panel[2][kFoldChunk][kFoldOutputs + 1];
  const int tid = threadIdx.x;
  auto stage = [&](int which, const uint32_t (&v)[kFoldPerThread]) {
#pragma unroll
    for (int i = 0; i < kFoldPerThread; ++i) {
      int out;
      uint32_t step;
      place(i, out, step);
      panel[which][step][out] = v[i];
    }
  };
  constexpr uint32_t infinity = kFormat == WB200_F32 ? 0x7f800000u : kFormat == WB200_BF16 ? 0x7f80u : 0x7c00u;
  constexpr uint32_t sign = kFormat == WB200_F32 ? 0x80000000u : 0x8000u;
  auto key_of = [](uint32_t bits) {   // order-preserving signed key of a non-NaN value
    const int v = kFormat == WB200_F32 ? static_cast<int>(bits) : static_cast<int>(static_cast<int16_t>(bits));
    return v ^ ((v >> 31) & (kFormat == WB200_F32 ? 0x7fffffff : 0x7fff));
  };
  auto bits_of = [](int key) {
    const int v = key ^ ((key >> 31) & (kFormat == WB200_F32 ? 0x7fffffff : 0x7fff));
    return static_cast<uint32_t>(v) & (kFormat == WB200_F32 ? 0xffffffffu : 0xffffu);
  };
  uint32_t acc = kCombine == WB200_EW_ADD ? 0u : kCombine == WB200_EW_MAX ? (infinity | sign) : infinity;
  auto fold = [&](int which, int count) {
    const uint32_t (*column)[kFoldOutputs + 1] = panel[which];
    uint32_t top = 0, residual = 0, result;
    if constexpr (kCombine == WB200_EW_ADD) {
      float a = __uint_as_float(acc);
#pragma unroll 8
      for (int s = 0; s < count; ++s) {
        const uint32_t bits = column[s][tid];
        const float v = __uint_as_float(bits), r = __fadd_rn(a, v);
        if constexpr (kFormal) {
          top = max(top, bits & 0x7fffffffu);
          const float part = __fsub_rn(r, a);
          residual |= __float_as_uint(__fadd_rn(__fsub_rn(a, __fsub_rn(r, part)), __fsub_rn(v, part))) & 0x7fffffffu;
        } else {
          saw_nan |= (v != v) | (r != r);
        }
        a = r;
      }
      result = __float_as_uint(a);
      top = max(top, result & 0x7fffffffu);
    } else {
      int a = key_of(acc);
      top = acc & ~sign;
#pragma unroll 8
      for (int s = 0; s < count; ++s) {
        const uint32_t bits = column[s][tid];
        top = max(top, bits & ~sign);
        a = kCombine == WB200_EW_MAX ? max(a, key_of(bits)) : min(a, key_of(bits));
      }
      result = bits_of(a);
    }
    const bool exceptional = kCombine == WB200_EW_ADD ? top >= infinity : top > infinity;
    if constexpr (kFormal) {
      if (exceptional) {
        acc = fold_full_steps<kCombine, kFormat>(&column[0][tid], kFoldOutputs + 1, count, acc, &flags);
        return;
      }
      if (residual) flags |= kFlagInexact;
    } else if constexpr (kCombine != WB200_EW_ADD) {
      saw_nan |= exceptional;
    }
    acc = result;
  };
  uint32_t v[kFoldPerThread];
  fetch(0, v);
  stage(0, v);
  __syncthreads();
  int which = 0;
  for (uint32_t base = 0; base < steps; base += kFoldChunk, which ^= 1) {
    const bool more = base + kFoldChunk < steps;
    if (more) fetch(base + kFoldChunk, v);
    if (tid < outputs) fold(which, static_cast<int>(min(static_cast<uint32_t>(kFoldChunk), steps - base)));
    if (more) stage(which ^ 1, v);
    __syncthreads();
  }
  return acc;
}

// Any rank, layout and set of reduced dimensions.
template <bool kFormal, int kCombine, int kFormat>
__global__ void __launch_bounds__(kThreads)
fold_staged_kernel(const uint8_t *src, uint8_t *dst, const __grid_constant__ FoldPlan plan, uint64_t tile_stride, int *nan_flag,
                   uint32_t *flags_word) {
  src += blockIdx.z * tile_stride;
  dst += blockIdx.z * tile_stride;
  __shared__ int64_t kept_slice[kFoldOutputs], kept_outer[kFoldOutputs], kept_c[kFoldOutputs], kept_dst[kFoldOutputs];
  const int tid = threadIdx.x;
  const int64_t first_output = static_cast<int64_t>(blockIdx.x) * kFoldOutputs;
  const int outputs = static_cast<int>(min(static_cast<int64_t>(kFoldOutputs), plan.dst.element_count - first_output));
  if (tid < outputs) fold_kept_coordinates(plan, first_output + tid, &kept_slice[tid], &kept_outer[tid], &kept_c[tid], &kept_dst[tid]);
  __syncthreads();
  pdl_launch_dependents();
  pdl_wait();
  auto place = [&](int i, int &out, uint32_t &step) {
    if (plan.along_steps) { step = (tid & 31) + 32 * (i & 1); out = (tid >> 5) + 8 * (i >> 1); }
    else { out = tid & 31; step = (tid >> 5) + 8 * i; }
  };
  auto fetch = [&](uint32_t base, uint32_t (&v)[kFoldPerThread]) {
#pragma unroll
    for (int i = 0; i < kFoldPerThread; ++i) {
      int out;
      uint32_t step;
      place(i, out, step);
      step += base;
      v[i] = 0;
      if (out < outputs && step < plan.steps)
        v[i] = load_element_bits(src, fold_element(plan, kept_slice[out], kept_outer[out], kept_c[out], step), kFormat);
    }
  };
  uint32_t flags = 0;
  bool saw_nan = false;
  const uint32_t acc = fold_block<kFormal, kCombine, kFormat>(plan.steps, outputs, fetch, place, flags, saw_nan);
  if (tid < outputs) store_element_bits(dst, kept_dst[tid], kFormat, acc);
  if constexpr (kFormal) merge_block_flags(flags_word, flags);
  else if (saw_nan) raise_status(nan_flag, 1);
}

// One reduced dimension that is not the channel, tensors of fewer than 2^31 elements: the address is linear in the step, and
// the placement fits a few 32-bit words (a launch of a microsecond or two waits for every line of its parameters).
struct LinearFold {
  uint32_t outputs, steps;
  uint32_t channels;          // outputs are [.., kept outer, channel]
  uint32_t kept_per_slice;    // kept outer extents of a leading slice (all of them where there are no slices)
  uint32_t inner;             // extents between the reduced dimension and the channel
  uint32_t full;              // channels in 64-wide blocks; the others lie `tail` wide behind them (Tensor: 0 and `channels`)
  uint32_t tail, src_block, src_tail, src_slice, dst_block, dst_tail, dst_slice;   // elements: block pitch, tail start, slice pitch
  uint32_t reduced_outer;     // extent of the reduced dimension within the outer index (1 when slices are reduced)
  uint32_t slice_step;        // slices are reduced: elements between steps, else 0
};
template <bool kFormal, int kCombine, int kFormat>
__global__ void __launch_bounds__(kThreads)
fold_linear_kernel(const uint8_t *src, uint8_t *dst, const __grid_constant__ LinearFold f, uint64_t tile_stride, int *nan_flag,
                   uint32_t *flags_word) {
  src += blockIdx.z * tile_stride;
  dst += blockIdx.z * tile_stride;
  const int tid = threadIdx.x, lane = tid & 31;
  const uint32_t output = blockIdx.x * kFoldOutputs + lane;
  const int outputs = static_cast<int>(min(static_cast<uint32_t>(kFoldOutputs), f.outputs - blockIdx.x * kFoldOutputs));
  const uint32_t rest = output / f.channels, c = output - rest * f.channels;
  const uint32_t slice = rest / f.kept_per_slice, kept = rest - slice * f.kept_per_slice;
  const uint32_t hi = kept / f.inner, outer = hi * f.inner * f.reduced_outer + (kept - hi * f.inner);
  const bool blocked = c < f.full;
  const uint32_t width = blocked ? 64u : f.tail;
  const uint32_t in_row = blocked ? c & 63u : c - f.full;
  const uint32_t line = slice * f.src_slice + (blocked ? (c >> 6) * f.src_block : f.src_tail) + outer * width + in_row;
  const uint32_t line_step = f.slice_step ? f.slice_step : f.inner * width;
  const uint32_t dst_at = slice * f.dst_slice + (blocked ? (c >> 6) * f.dst_block : f.dst_tail) + kept * width + in_row;
  pdl_launch_dependents();
  pdl_wait();
  auto place = [&](int i, int &out, uint32_t &step) { out = lane; step = (tid >> 5) + 8 * i; };
  auto fetch = [&](uint32_t base, uint32_t (&v)[kFoldPerThread]) {
    const uint32_t first = base + (tid >> 5);
#pragma unroll
    for (int i = 0; i < kFoldPerThread; ++i) {
      v[i] = 0;
      if (lane < outputs && first + 8 * i < f.steps) v[i] = load_element_bits(src, line + (first + 8 * i) * line_step, kFormat);
    }
  };
  uint32_t flags = 0;
  bool saw_nan = false;
  const uint32_t acc = fold_block<kFormal, kCombine, kFormat>(f.steps, outputs, fetch, place, flags, saw_nan);
  if (tid < outputs) store_element_bits(dst, dst_at, kFormat, acc);
  if constexpr (kFormal) merge_block_flags(flags_word, flags);
  else if (saw_nan) raise_status(nan_flag, 1);
}

// ------------------------------------------------------------------------------------------------ command runs
// One launch for a run of formal commands of one Tile (FormalRun). A cluster of kRunCtas thread blocks of kRunThreads
// threads executes the commands in issue order with a cluster barrier (release / acquire at cluster scope) after each,
// so a command reads what earlier commands of the run wrote, whichever block wrote it. A cluster is co-scheduled by the
// hardware, so its blocks may wait for one another. Elementwise commands and reductions go through the very device
// functions of their own kernels, spread over the cluster's threads; the GEMM is the formal chain of gemm_formal.cu written for one thread per output:
//   acc = +0; for k ascending: acc = fma(widen(lhs), widen(rhs), acc); [acc = acc + psum;] dst = narrow(acc)
// (lib/Wafer/Simulator/Reference/Numeric/FormalTensorNumeric.cpp:271-361) through the tile function of gemm_formal.cuh, so
// every destination gets the bits the command-by-command replay gives it.
constexpr int kRunThreads = 512;   // 128 registers per thread: the formal evaluators need them
constexpr int kRunCtas = 8;        // one cluster (the portable maximum)
__device__ __forceinline__ uint32_t run_cta_rank() {
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  return rank;
}
__device__ __forceinline__ void run_cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The GEMM of a run: 64 x 64 output tiles, sixteen at a time (one per group of 256 threads of the cluster, each group with
// shared-memory panels of its own), through the tile function of the command's own kernel, so every output sees the same k-ascending
// chain. `variant` was chosen on the host (gemm_formal_variant).
struct RunPanels {
  float lhs[kRunThreads / 256][kPanelK][kBlockM + 4];
  float rhs[kRunThreads / 256][kPanelK][kBlockN + 4];
};
__device__ __forceinline__ void run_gemm(const GemmFormalArgs &a, int variant, RunPanels &panels) {
  const int group = threadIdx.x >> 8, tid = threadIdx.x & 255;
  const int cluster_group = static_cast<int>(run_cta_rank()) * (kRunThreads / 256) + group;
  const int tiles_n = (a.n + kBlockN - 1) / kBlockN, tiles = ((a.m + kBlockM - 1) / kBlockM) * tiles_n;
  for (int first = 0; first < tiles; first += kRunCtas * (kRunThreads / 256)) {
    const int tile = first + cluster_group;
    const bool active = tile < tiles;
    const int row0 = active ? (tile / tiles_n) * kBlockM : 0, col0 = active ? (tile % tiles_n) * kBlockN : 0;
    if (variant == 3) gemm_formal_tile<true, true, true>(a, 0, row0, col0, tid, active, panels.lhs[group], panels.rhs[group]);
    else if (variant == 2) gemm_formal_tile<true, true, false>(a, 0, row0, col0, tid, active, panels.lhs[group], panels.rhs[group]);
    else gemm_formal_tile<false, false, false>(a, 0, row0, col0, tid, active, panels.lhs[group], panels.rhs[group]);
  }
}

// An elementwise command of a run. The arithmetic family on float operands takes the instantiation with the operation
// and format fixed at compile time, as in the command's own kernel (a few dozen instructions per element instead of the
// generic evaluator's decision tree); everything else takes the generic one.
template <int kOp>
__device__ __noinline__ uint32_t run_elementwise_op(const RunElementwise &e, int vector) {
  if (e.in_format == WB200_F32)
    return formal_elementwise_groups<true, kOp, WB200_F32>(e.op, e.in_format, e.out_format, e.input_count, e.in0, e.in1, e.dst, e.in_map, e.out_map,
                                                           e.rhs, vector, run_cta_rank() * kRunThreads + threadIdx.x, kRunCtas * kRunThreads);
  if (e.in_format == WB200_BF16)
    return formal_elementwise_groups<true, kOp, WB200_BF16>(e.op, e.in_format, e.out_format, e.input_count, e.in0, e.in1, e.dst, e.in_map, e.out_map,
                                                            e.rhs, vector, run_cta_rank() * kRunThreads + threadIdx.x, kRunCtas * kRunThreads);
  return formal_elementwise_groups<true, kOp, WB200_F16>(e.op, e.in_format, e.out_format, e.input_count, e.in0, e.in1, e.dst, e.in_map, e.out_map,
                                                         e.rhs, vector, run_cta_rank() * kRunThreads + threadIdx.x, kRunCtas * kRunThreads);
}
__device__ __noinline__ uint32_t run_elementwise_generic(const RunElementwise &e, int vector) {
  return formal_elementwise_groups<true, -1, 0>(e.op, e.in_format, e.out_format, e.input_count, e.in0, e.in1, e.dst, e.in_map, e.out_map, e.rhs,
                                                vector, run_cta_rank() * kRunThreads + threadIdx.x, kRunCtas * kRunThreads);
}
__device__ __forceinline__ uint32_t run_elementwise(const RunElementwise &e, int vector) {
  if (is_float_format(e.in_format)) {
    switch (e.op) {
      case WB200_EW_MAX: return run_elementwise_op<WB200_EW_MAX>(e, vector);
      case WB200_EW_MIN: return run_elementwise_op<WB200_EW_MIN>(e, vector);
      case WB200_EW_ADD: return run_elementwise_op<WB200_EW_ADD>(e, vector);
      case WB200_EW_SUB: return run_elementwise_op<WB200_EW_SUB>(e, vector);
      case WB200_EW_MUL: return run_elementwise_op<WB200_EW_MUL>(e, vector);
      default: break;
    }
  }
  return run_elementwise_generic(e, vector);
}

__device__ __forceinline__ uint32_t run_reduce(const RunReduce &r) {
  uint32_t flags = 0;
  const bool nhwc = r.src_map.layout == WB200_LAYOUT_NCX && r.dst_map.layout == WB200_LAYOUT_NCX && r.src_map.rank == 4 && r.dst_map.rank == 4;
  if (!nhwc) return flags;   // formal_run_admits lets nothing else in
  for (int64_t out = run_cta_rank() * kRunThreads + threadIdx.x; out < r.dst_map.element_count; out += kRunCtas * kRunThreads) {
#define WB200_RUN_REDUCE(COMBINE)                                                                                                  \
    if (r.format == WB200_F32) flags |= formal_reduce_nhwc_output<COMBINE, WB200_F32>(r.src, r.dst, r.src_map, r.dst_map, r.reduced_mask, out);   \
    else if (r.format == WB200_BF16) flags |= formal_reduce_nhwc_output<COMBINE, WB200_BF16>(r.src, r.dst, r.src_map, r.dst_map, r.reduced_mask, out); \
    else flags |= formal_reduce_nhwc_output<COMBINE, WB200_F16>(r.src, r.dst, r.src_map, r.dst_map, r.reduced_mask, out)
    if (r.op == WB200_RED_SUM) { WB200_RUN_REDUCE(WB200_EW_ADD); }
    else if (r.op == WB200_RED_MAX) { WB200_RUN_REDUCE(WB200_EW_MAX); }
    else { WB200_RUN_REDUCE(WB200_EW_MIN); }
#undef WB200_RUN_REDUCE
  }
  return flags;
}

__global__ void __cluster_dims__(kRunCtas, 1, 1) __launch_bounds__(kRunThreads) formal_run_kernel(const __grid_constant__ FormalRun run, uint32_t *flags_word) {
  __shared__ __align__(16) RunPanels panels;
  // The command being executed, copied from the parameter space: its fields are read inside the inner loops, and a
  // dynamically indexed kernel parameter costs a constant-bank load per use.
  __shared__ __align__(16) unsigned char command_storage[sizeof(RunCommand)];
  const RunCommand &command = *reinterpret_cast<const RunCommand *>(command_storage);
  static_assert(sizeof(RunCommand) % 4 == 0, "copied as 32-bit words");
  uint32_t flags = 0;
#pragma unroll 1
  for (int c = 0; c < run.count; ++c) {
    {
      const uint32_t *from = reinterpret_cast<const uint32_t *>(&run.command[c]);
      uint32_t *to = reinterpret_cast<uint32_t *>(command_storage);
      for (int w = threadIdx.x; w < static_cast<int>(sizeof(RunCommand) / 4); w += kRunThreads) to[w] = from[w];
    }
    __syncthreads();
    if (command.kind == WB200_RUN_ELEMENTWISE) {
      const RunElementwise &e = command.u.elementwise;
      const int vector = ((reinterpret_cast<uintptr_t>(e.in0) | reinterpret_cast<uintptr_t>(e.in1) | reinterpret_cast<uintptr_t>(e.dst)) & 15) == 0;
      flags |= run_elementwise(e, vector);
    } else if (command.kind == WB200_RUN_REDUCE) {
      flags |= run_reduce(command.u.reduce);
    } else {
      run_gemm(command.u.gemm, command.variant, panels);
    }
    run_cluster_barrier();   // the next command may read anything this one wrote, in any block
  }
  merge_block_flags(flags_word, flags);
}

// Plain pooling (lib/Wafer/Simulator/Kernel/TargetModelTensorNumeric.cpp:466-583): every output folds its window in
// (kh, kw) order with the formal max / min / add, so the roundings and the raised flags are those of the reference's
// window-by-window elementwise passes. Sum starts from +0 and adds every tap; max / min start from the first tap.
// kVec consecutive channels per thread (1 or 4): with 4 the taps move as one 16-byte (f32) or 8-byte (16-bit) access and
// the index arithmetic is shared; the launcher picks it when channel counts, strides and pointers allow it.
template <int kVec>
__device__ __forceinline__ void load_channels(const uint8_t *base, int64_t index, int format, uint32_t (&v)[kVec]) {
  if (kVec == 1) {
    v[0] = load_element_bits(base, index, format);
  } else if (format == WB200_F32) {
    const uint4 w = *reinterpret_cast<const uint4 *>(base + index * 4);
    v[0] = w.x; v[1 % kVec] = w.y; v[2 % kVec] = w.z; v[3 % kVec] = w.w;
  } else {
    const uint2 w = *reinterpret_cast<const uint2 *>(base + index * 2);
    v[0] = w.x & 0xffffu; v[1 % kVec] = w.x >> 16; v[2 % kVec] = w.y & 0xffffu; v[3 % kVec] = w.y >> 16;
  }
}
template <int kVec>
__device__ __forceinline__ void store_channels(uint8_t *base, int64_t index, int format, const uint32_t (&v)[kVec]) {
  if (kVec == 1) {
    store_element_bits(base, index, format, v[0]);
  } else if (format == WB200_F32) {
    *reinterpret_cast<uint4 *>(base + index * 4) = make_uint4(v[0], v[1 % kVec], v[2 % kVec], v[3 % kVec]);
  } else {
    *reinterpret_cast<uint2 *>(base + index * 2) = make_uint2((v[0] & 0xffffu) | (v[1 % kVec] << 16), (v[2 % kVec] & 0xffffu) | (v[3 % kVec] << 16));
  }
}

template <int kCombine, int kFormat, int kVec>
__global__ void __launch_bounds__(kThreads)
formal_pool_kernel(const uint8_t *src, uint8_t *dst, const LayoutMap src_map, const LayoutMap dst_map,
                   const PoolWindow window, uint32_t *flags_word) {
  constexpr int combine = kCombine, format = kFormat;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  uint32_t flags = 0;
  const uint32_t out_h = static_cast<uint32_t>(dst_map.shape[1]), out_w = static_cast<uint32_t>(dst_map.shape[2]);
  const uint32_t channel_groups = static_cast<uint32_t>(dst_map.shape[3]) / kVec, in_w = static_cast<uint32_t>(src_map.shape[2]);
  const int64_t total = dst_map.element_count / kVec;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
    const uint32_t index = static_cast<uint32_t>(i);          // the launcher admits at most 2^32 - 1 outputs
    const uint32_t pixel = index / channel_groups, c = (index - pixel * channel_groups) * kVec;
    const uint32_t row = pixel / out_w, w = pixel - row * out_w;
    const uint32_t n = row / out_h, h = row - n * out_h;
    uint32_t result[kVec];
    const int64_t full_c = src_map.cx_blocks * src_map.c_block;
    const int64_t width = static_cast<int64_t>(c) < full_c ? src_map.c_block : src_map.c0;   // taps of one channel move by constant strides
    const int64_t corner = physical_index_nhwc(src_map, n, static_cast<int64_t>(h * window.stride_h) * in_w + w * window.stride_w, c);
    for (uint32_t kh = 0; kh < window.kernel_h; ++kh)
      for (uint32_t kw = 0; kw < window.kernel_w; ++kw) {
        uint32_t tap[kVec];
        load_channels<kVec>(src, corner + (static_cast<int64_t>(kh) * in_w + kw) * width, format, tap);
#pragma unroll
        for (int v = 0; v < kVec; ++v) {
          if (kh == 0 && kw == 0) {
            if (combine != WB200_EW_ADD) { result[v] = tap[v]; continue; }
            result[v] = 0u;
          }
          uint32_t element_flags = 0;
          result[v] = formal_scalar(combine, format, format, result[v], tap[v], &element_flags, kFoldCommonCase);
          flags |= element_flags;
        }
      }
    store_channels<kVec>(dst, physical_index_nhwc(dst_map, n, static_cast<int64_t>(h) * out_w + w, c), format, result);
  }
  merge_block_flags(flags_word, flags);
}

int grid_for(int64_t elements) {
  int64_t blocks = (elements + kThreads - 1) / kThreads;
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 16) blocks = 148 * 16;
  return static_cast<int>(blocks);
}

bool codec_takes_units(const uint8_t *src, const uint8_t *dst, const LayoutMap &map, int element_bytes) {
  const bool blocked = map.layout == WB200_LAYOUT_CX || map.layout == WB200_LAYOUT_NCX;
  return (element_bytes == 2 || element_bytes == 4) && blocked && map.shape[map.rank - 1] % (16 / element_bytes) == 0 && all_aligned16(src, dst) &&
         map.physical_elements < (1ll << 31);
}
CodecJob codec_job(const uint8_t *src, uint8_t *dst, const LayoutMap &map, int element_bytes) {
  return {reinterpret_cast<const uint4 *>(src), reinterpret_cast<uint4 *>(dst), map, static_cast<uint32_t>(map.element_count * element_bytes / 16)};
}

wb200_status launch_codec(const uint8_t *src, uint8_t *dst, const LayoutMap &map, int element_bytes, int pack,
                          cudaStream_t stream) {
  if (codec_takes_units(src, dst, map, element_bytes)) {
    CodecJobs jobs{};
    jobs.job[0] = codec_job(src, dst, map, element_bytes);
    const int grid = grid_for(jobs.job[0].units);
    if (element_bytes == 2) codec_wide_kernel<8><<<grid, kThreads, 0, stream>>>(jobs, pack);
    else codec_wide_kernel<4><<<grid, kThreads, 0, stream>>>(jobs, pack);
    WB200_CUDA_CHECK(cudaGetLastError());
    return WB200_OK;
  }
  const int grid = grid_for(map.element_count);
  switch (element_bytes) {
    case 1: codec_kernel<uint8_t><<<grid, kThreads, 0, stream>>>(src, dst, map, pack); break;
    case 2: codec_kernel<uint16_t><<<grid, kThreads, 0, stream>>>(reinterpret_cast<const uint16_t *>(src), reinterpret_cast<uint16_t *>(dst), map, pack); break;
    case 4: codec_kernel<uint32_t><<<grid, kThreads, 0, stream>>>(reinterpret_cast<const uint32_t *>(src), reinterpret_cast<uint32_t *>(dst), map, pack); break;
    case 8: codec_kernel<uint64_t><<<grid, kThreads, 0, stream>>>(reinterpret_cast<const uint64_t *>(src), reinterpret_cast<uint64_t *>(dst), map, pack); break;
    default: return fail(WB200_ERR_UNSUPPORTED, "codec supports byte-addressable element types only");
  }
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

// Few outputs cannot fill the machine with one thread each; the staged fold spreads their loads over 8 threads per output.
constexpr int64_t kManyOutputs = 65536;
template <bool kFormal>
wb200_status launch_fold_staged(int op, int format, const uint8_t *src, uint8_t *dst, const LayoutMap &src_map, const LayoutMap &dst_map,
                                uint32_t reduced_mask, int *nan_flag, uint32_t *flags_word, cudaStream_t stream, TileBatch tiles = TileBatch()) {
  FoldPlan plan{};
  plan.src = src_map; plan.dst = dst_map; plan.reduced_mask = reduced_mask;
  const int rank = src_map.rank;
  const bool sliced = src_map.layout == WB200_LAYOUT_NCX && rank > 1;
  int64_t steps = 1;
  for (int d = 0; d < rank; ++d) {
    if (!(reduced_mask & (1u << d))) continue;
    if (plan.count == 3) return fail(WB200_ERR_UNSUPPORTED, "a reduction has at most three dimensions");
    plan.size[plan.count] = static_cast<uint32_t>(src_map.shape[d]);
    plan.kind[plan.count] = d == rank - 1 ? 2 : (d == 0 && sliced) ? 0 : 1;
    int64_t outer_step = 1;
    for (int e = d + 1; e < rank - 1; ++e) outer_step *= src_map.shape[e];
    plan.outer_step[plan.count] = outer_step;
    steps *= src_map.shape[d];
    ++plan.count;
  }
  if (steps >= (1ll << 31)) return fail(WB200_ERR_LIMIT, "a reduction folds at most 2^31 - 1 inputs per output");
  plan.steps = static_cast<uint32_t>(steps);
  plan.along_steps = (reduced_mask >> (rank - 1)) & 1u;
  const int64_t blocks = (dst_map.element_count + kFoldOutputs - 1) / kFoldOutputs;
  if (blocks >= (1ll << 31)) return fail(WB200_ERR_LIMIT, "reduction output too large");
  const dim3 grid(static_cast<unsigned>(blocks < 1 ? 1 : blocks), 1, tiles.tiles);
  LinearFold linear{};
  const bool is_linear = plan.count == 1 && plan.kind[0] != 2 && dst_map.element_count > 0 && steps > 0 && src_map.physical_elements < (1ll << 31);
  if (is_linear) {
    const bool blocked = src_map.layout == WB200_LAYOUT_CX || src_map.layout == WB200_LAYOUT_NCX;
    linear.outputs = static_cast<uint32_t>(dst_map.element_count);
    linear.steps = plan.steps;
    linear.channels = static_cast<uint32_t>(src_map.shape[rank - 1]);
    const int64_t slices = sliced ? dst_map.shape[0] : 1;
    linear.kept_per_slice = static_cast<uint32_t>(dst_map.element_count / linear.channels / slices);
    linear.inner = plan.kind[0] == 1 ? static_cast<uint32_t>(plan.outer_step[0]) : linear.kept_per_slice;
    linear.reduced_outer = plan.kind[0] == 1 ? plan.size[0] : 1u;
    linear.slice_step = plan.kind[0] == 0 ? static_cast<uint32_t>(src_map.outer_slice_stride) : 0u;
    linear.full = blocked ? static_cast<uint32_t>(src_map.cx_blocks * src_map.c_block) : 0u;
    linear.tail = blocked ? static_cast<uint32_t>(src_map.c0) : linear.channels;
    if (blocked) {
      linear.src_block = static_cast<uint32_t>(src_map.block_outer_elements * src_map.c_block);
      linear.src_tail = static_cast<uint32_t>(src_map.cx_blocks) * linear.src_block;
      linear.src_slice = static_cast<uint32_t>(src_map.outer_slice_stride);
      linear.dst_block = static_cast<uint32_t>(dst_map.block_outer_elements * dst_map.c_block);
      linear.dst_tail = static_cast<uint32_t>(dst_map.cx_blocks) * linear.dst_block;
      linear.dst_slice = static_cast<uint32_t>(dst_map.outer_slice_stride);
    }
  }
#define WB200_FOLD(COMBINE, FORMAT)                                                                                                      \
  do {                                                                                                                                  \
    if (is_linear) WB200_CUDA_CHECK(launch_dependent(fold_linear_kernel<kFormal, COMBINE, FORMAT>, grid, kThreads, 0, stream, src, dst, linear, tiles.stride, nan_flag, flags_word)); \
    else WB200_CUDA_CHECK(launch_dependent(fold_staged_kernel<kFormal, COMBINE, FORMAT>, grid, kThreads, 0, stream, src, dst, plan, tiles.stride, nan_flag, flags_word));             \
  } while (0)
#define WB200_FOLD_FORMATS(COMBINE)                                   \
  if (format == WB200_F32) WB200_FOLD(COMBINE, WB200_F32);            \
  else if (format == WB200_BF16) WB200_FOLD(COMBINE, WB200_BF16);     \
  else WB200_FOLD(COMBINE, WB200_F16)
  if (op == WB200_RED_SUM) {
    if (format != WB200_F32) return fail(WB200_ERR_UNSUPPORTED, "sum reductions are F32");
    WB200_FOLD(WB200_EW_ADD, WB200_F32);
  } else if (op == WB200_RED_MAX) { WB200_FOLD_FORMATS(WB200_EW_MAX); }
  else { WB200_FOLD_FORMATS(WB200_EW_MIN); }
#undef WB200_FOLD_FORMATS
#undef WB200_FOLD
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}
bool reduce_one_thread_per_output(const LayoutMap &src_map, const LayoutMap &dst_map) {
  return src_map.layout == WB200_LAYOUT_NCX && dst_map.layout == WB200_LAYOUT_NCX && src_map.rank == 4 && dst_map.rank == 4 &&
         dst_map.element_count >= kManyOutputs && dst_map.element_count < (1ll << 32);
}

}  // namespace

wb200_status launch_elementwise(int op, int format, int input_count, const uint8_t *in0, const uint8_t *in1,
                                uint8_t *dst, const LayoutMap &map, int *nan_flag, cudaStream_t stream) {
  if (!all_aligned16(in0, in1, dst)) return fail(WB200_ERR_INVALID_ARGUMENT, "elementwise storage must be 16-byte aligned on the device");
  const StorageWalk walk = storage_walk(map, map);
  const int grid = walk_blocks(walk, kThreads);
#define WB200_MEW(OP)                                                                                                                     \
  case OP:                                                                                                                                \
    if (format == WB200_F32) elementwise_walk_kernel<OP, WB200_F32><<<grid, kThreads, 0, stream>>>(input_count, in0, in1, dst, walk, nan_flag);        \
    else if (format == WB200_BF16) elementwise_walk_kernel<OP, WB200_BF16><<<grid, kThreads, 0, stream>>>(input_count, in0, in1, dst, walk, nan_flag); \
    else elementwise_walk_kernel<OP, WB200_F16><<<grid, kThreads, 0, stream>>>(input_count, in0, in1, dst, walk, nan_flag);                          \
    break;
  switch (op) {
    WB200_MEW(WB200_EW_ABS) WB200_MEW(WB200_EW_NEG) WB200_MEW(WB200_EW_RECIP) WB200_MEW(WB200_EW_SQUARE) WB200_MEW(WB200_EW_MAX)
    WB200_MEW(WB200_EW_MIN) WB200_MEW(WB200_EW_ADD) WB200_MEW(WB200_EW_SUB) WB200_MEW(WB200_EW_MUL) WB200_MEW(WB200_EW_RELU)
    WB200_MEW(WB200_EW_SQRT) WB200_MEW(WB200_EW_RSQRT) WB200_MEW(WB200_EW_LOG2) WB200_MEW(WB200_EW_LN) WB200_MEW(WB200_EW_POW2)
    WB200_MEW(WB200_EW_EXP) WB200_MEW(WB200_EW_EXPLP) WB200_MEW(WB200_EW_SIN) WB200_MEW(WB200_EW_COS) WB200_MEW(WB200_EW_TANH)
    WB200_MEW(WB200_EW_SIGMOID) WB200_MEW(WB200_EW_SOFTPLUS)
    default: return fail(WB200_ERR_UNSUPPORTED, "elementwise operation is not in the managed domain");
  }
#undef WB200_MEW
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

static bool is_function(int op) {
  return op == WB200_EW_SQRT || op == WB200_EW_RSQRT || (op >= WB200_EW_LOG2 && op <= WB200_EW_EXP) ||
         (op >= WB200_EW_SIN && op <= WB200_EW_SIGMOID) || op == WB200_EW_SOFTPLUS;
}

wb200_status launch_elementwise_formal(int op, int in_format, int out_format, int input_count, const uint8_t *in0, const uint8_t *in1,
                                       uint8_t *dst, const LayoutMap &in_map, const LayoutMap &out_map, uint32_t *flags_word,
                                       cudaStream_t stream, RhsBroadcast rhs, TileBatch tiles) {
  auto linear_layout = [](const LayoutMap &m) { return m.layout == WB200_LAYOUT_TENSOR || m.layout == WB200_LAYOUT_NTENSOR; };
  const bool function_family = is_function(op);
  if (function_family && linear_layout(in_map) && linear_layout(out_map)) {
    int64_t blocks = (out_map.element_count + kShortThreads - 1) / kShortThreads;
    const dim3 grid(static_cast<unsigned>(blocks < 1 ? 1 : blocks > 148 * 16 ? 148 * 16 : blocks), 1, tiles.tiles);
    const bool single = in_format == WB200_F32 || in_format == WB200_TF32;
#define WB200_FUNCTION(OP)                                                                                                              \
  case OP:                                                                                                                              \
    if (single) WB200_CUDA_CHECK(launch_dependent(formal_function_kernel<OP, true>, grid, kShortThreads, 0, stream, in_format, in0, dst, out_map.element_count, tiles.stride, flags_word)); \
    else WB200_CUDA_CHECK(launch_dependent(formal_function_kernel<OP, false>, grid, kShortThreads, 0, stream, in_format, in0, dst, out_map.element_count, tiles.stride, flags_word));      \
    break;
    switch (op) {
      WB200_FUNCTION(WB200_EW_SQRT) WB200_FUNCTION(WB200_EW_RSQRT) WB200_FUNCTION(WB200_EW_LOG2) WB200_FUNCTION(WB200_EW_LN)
      WB200_FUNCTION(WB200_EW_POW2) WB200_FUNCTION(WB200_EW_EXP) WB200_FUNCTION(WB200_EW_SIN) WB200_FUNCTION(WB200_EW_COS)
      WB200_FUNCTION(WB200_EW_TANH) WB200_FUNCTION(WB200_EW_SIGMOID) WB200_FUNCTION(WB200_EW_SOFTPLUS)
      default: return fail(WB200_ERR_UNSUPPORTED, "elementwise operation has no formal evaluation");
    }
#undef WB200_FUNCTION
    WB200_CUDA_CHECK(cudaGetLastError());
    return WB200_OK;
  }
  const bool short_vector = out_map.element_count > 0 && out_map.element_count <= kShortVector && linear_layout(in_map) && linear_layout(out_map) &&
                            is_float_format(in_format) && is_float_format(out_format);
  if (short_vector) {
    const uint32_t count = static_cast<uint32_t>(out_map.element_count);
    const dim3 grid((count + kShortThreads - 1) / kShortThreads, 1, tiles.tiles);
#define WB200_SHORT_LAUNCH(OP, FORMAT) \
  WB200_CUDA_CHECK(launch_dependent(formal_elementwise_short_kernel<OP, FORMAT>, grid, kShortThreads, 0, stream, out_format, input_count, in0, in1, dst, count, rhs, tiles.stride, flags_word))
#define WB200_SHORT(OP)                                             \
  case OP:                                                          \
    if (in_format == WB200_F32) WB200_SHORT_LAUNCH(OP, WB200_F32);  \
    else if (in_format == WB200_BF16) WB200_SHORT_LAUNCH(OP, WB200_BF16); \
    else WB200_SHORT_LAUNCH(OP, WB200_F16);                         \
    WB200_CUDA_CHECK(cudaGetLastError());                           \
    return WB200_OK;
    switch (op) {
      WB200_SHORT(WB200_EW_ABS) WB200_SHORT(WB200_EW_NEG) WB200_SHORT(WB200_EW_RELU) WB200_SHORT(WB200_EW_RECIP) WB200_SHORT(WB200_EW_SQUARE)
      WB200_SHORT(WB200_EW_MAX) WB200_SHORT(WB200_EW_MIN) WB200_SHORT(WB200_EW_ADD) WB200_SHORT(WB200_EW_SUB) WB200_SHORT(WB200_EW_MUL)
      WB200_SHORT(WB200_EW_EQ) WB200_SHORT(WB200_EW_NE) WB200_SHORT(WB200_EW_GE) WB200_SHORT(WB200_EW_GT) WB200_SHORT(WB200_EW_LE)
      WB200_SHORT(WB200_EW_LT)
      default: break;
    }
#undef WB200_SHORT
#undef WB200_SHORT_LAUNCH
  }
  if (tiles.tiles > 1) return fail(WB200_ERR_UNSUPPORTED, "no elementwise kernel for several Tiles at these sizes and formats");
  // a thread takes eight consecutive elements, or one at a time for the correctly rounded functions
  const int64_t groups = function_family ? out_map.element_count : (out_map.element_count + 7) / 8;
  int64_t blocks = (groups + kThreads - 1) / kThreads;
  blocks = blocks < 1 ? 1 : blocks > 148 * 32 ? 148 * 32 : blocks;
  const int grid = static_cast<int>(blocks);
#define WB200_EW_LAUNCH(LINEAR, OP, FORMAT)                                                                                              \
  formal_elementwise_kernel<LINEAR, OP, FORMAT><<<grid, kThreads, 0, stream>>>(op, in_format, out_format, input_count, in0, in1, dst, in_map, \
                                                                              out_map, rhs, vector, flags_word)
#define WB200_EW_FORMATS(OP)                                            \
  case OP:                                                              \
    if (in_format == WB200_F32) WB200_EW_LAUNCH(true, OP, WB200_F32);   \
    else if (in_format == WB200_BF16) WB200_EW_LAUNCH(true, OP, WB200_BF16); \
    else WB200_EW_LAUNCH(true, OP, WB200_F16);                          \
    break;
  if (linear_layout(in_map) && linear_layout(out_map)) {
    const int vector = all_aligned16(in0, in1, dst);
    const bool specialised = is_float_format(in_format);
    switch (specialised ? op : -1) {
      WB200_EW_FORMATS(WB200_EW_ABS) WB200_EW_FORMATS(WB200_EW_NEG) WB200_EW_FORMATS(WB200_EW_RELU) WB200_EW_FORMATS(WB200_EW_RECIP)
      WB200_EW_FORMATS(WB200_EW_SQUARE) WB200_EW_FORMATS(WB200_EW_MAX) WB200_EW_FORMATS(WB200_EW_MIN) WB200_EW_FORMATS(WB200_EW_ADD)
      WB200_EW_FORMATS(WB200_EW_SUB) WB200_EW_FORMATS(WB200_EW_MUL) WB200_EW_FORMATS(WB200_EW_EQ) WB200_EW_FORMATS(WB200_EW_NE)
      WB200_EW_FORMATS(WB200_EW_GE) WB200_EW_FORMATS(WB200_EW_GT) WB200_EW_FORMATS(WB200_EW_LE) WB200_EW_FORMATS(WB200_EW_LT)
      default: WB200_EW_LAUNCH(true, -1, 0); break;
    }
  } else {
    const int vector = 0;
    WB200_EW_LAUNCH(false, -1, 0);
  }
#undef WB200_EW_FORMATS
#undef WB200_EW_LAUNCH
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

wb200_status launch_elementwise_chain(const ElementwiseChain &chain, uint32_t *flags_word, cudaStream_t stream, TileBatch tiles) {
  if (chain.steps < 1 || chain.steps > kMaxChainSteps || chain.count < 1 || !is_float_format(chain.format))
    return fail(WB200_ERR_INVALID_ARGUMENT, "malformed elementwise chain");
  if (!chain.step[0].lhs) return fail(WB200_ERR_INVALID_ARGUMENT, "malformed elementwise chain");
  uintptr_t low_bits = tiles.tiles > 1 ? static_cast<uintptr_t>(tiles.stride) : 0;
  for (int s = 0; s < chain.steps; ++s)
    low_bits |= reinterpret_cast<uintptr_t>(chain.step[s].dst) | reinterpret_cast<uintptr_t>(chain.step[s].lhs) | (chain.step[s].rhs_mode == WB200_RHS_SAME ? reinterpret_cast<uintptr_t>(chain.step[s].rhs) : 0);
  bool one_each = chain.count <= kShortVector;
  for (int s = 0; s < chain.steps; ++s) one_each |= is_function(chain.step[s].op);
  const int per = one_each ? 1 : 8, threads = one_each ? kShortThreads : kThreads;
  int64_t blocks = ((chain.count + per - 1) / per + threads - 1) / threads;
  blocks = blocks < 1 ? 1 : blocks > 148 * 32 ? 148 * 32 : blocks;
  const dim3 grid(static_cast<unsigned>(blocks), 1, tiles.tiles);
  const int vector = (low_bits & 15) == 0;
#define WB200_CHAIN(FORMAT)                                                                                          \
  do {                                                                                                               \
    if (one_each) WB200_CUDA_CHECK(launch_dependent(formal_chain_kernel<FORMAT, 1>, grid, threads, 0, stream, chain, vector, tiles.stride, flags_word));           \
    else WB200_CUDA_CHECK(launch_dependent(formal_chain_kernel<FORMAT, 8>, grid, threads, 0, stream, chain, vector, tiles.stride, flags_word));                    \
  } while (0)
  if (chain.format == WB200_F32) WB200_CHAIN(WB200_F32);
  else if (chain.format == WB200_BF16) WB200_CHAIN(WB200_BF16);
  else WB200_CHAIN(WB200_F16);
#undef WB200_CHAIN
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

// Commands small enough for one thread block: one block is 1 / 148 of the machine, so a large command is faster in its
// own kernel. Elementwise: linear 1-D vectors of at most 2^17 elements; reduce: NCx rank 4 with at most 2^18 inputs;
// GEMM: one matrix of at most 2^20 multiply-adds.
bool formal_run_admits(const RunCommand &command) {
  auto linear = [](const LayoutMap &m) { return m.layout == WB200_LAYOUT_TENSOR || m.layout == WB200_LAYOUT_NTENSOR; };
  if (command.kind == WB200_RUN_ELEMENTWISE) {
    const RunElementwise &e = command.u.elementwise;
    return linear(e.in_map) && linear(e.out_map) && e.out_map.element_count <= (1 << 17);
  }
  if (command.kind == WB200_RUN_REDUCE) {
    const RunReduce &r = command.u.reduce;
    return r.src_map.layout == WB200_LAYOUT_NCX && r.dst_map.layout == WB200_LAYOUT_NCX && r.src_map.rank == 4 && r.dst_map.rank == 4 &&
           r.src_map.element_count <= (1 << 18);
  }
  const GemmFormalArgs &g = command.u.gemm;
  return g.batch == 1 && static_cast<int64_t>(g.m) * g.n * g.k <= (1 << 20) && is_float_format(g.in_format) && is_float_format(g.out_format);
}

wb200_status launch_formal_run(const FormalRun &run, uint32_t *flags_word, cudaStream_t stream) {
  if (run.count < 1 || run.count > kMaxRunCommands) return fail(WB200_ERR_INVALID_ARGUMENT, "malformed command run");
  for (int c = 0; c < run.count; ++c)
    if (!formal_run_admits(run.command[c])) return fail(WB200_ERR_INVALID_ARGUMENT, "command outside the domain of a command run");
  formal_run_kernel<<<kRunCtas, kRunThreads, 0, stream>>>(run, flags_word);
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

wb200_status launch_reduce_formal(int op, int format, const uint8_t *src, uint8_t *dst, const LayoutMap &src_map, const LayoutMap &dst_map,
                                  uint32_t reduced_mask, uint32_t *flags_word, cudaStream_t stream, TileBatch tiles) {
  if (!reduce_one_thread_per_output(src_map, dst_map))
    return launch_fold_staged<true>(op, format, src, dst, src_map, dst_map, reduced_mask, nullptr, flags_word, stream, tiles);
  if (tiles.tiles > 1) return fail(WB200_ERR_UNSUPPORTED, "no reduction of several Tiles with so many outputs");
  const int grid = static_cast<int>((dst_map.element_count + kThreads - 1) / kThreads);
#define WB200_RED_LAUNCH(COMBINE, FORMAT) formal_reduce_nhwc_kernel<COMBINE, FORMAT><<<grid, kThreads, 0, stream>>>(src, dst, src_map, dst_map, reduced_mask, flags_word)
#define WB200_RED_FORMATS(COMBINE)                                              \
    if (format == WB200_F32) WB200_RED_LAUNCH(COMBINE, WB200_F32);              \
    else if (format == WB200_BF16) WB200_RED_LAUNCH(COMBINE, WB200_BF16);       \
    else WB200_RED_LAUNCH(COMBINE, WB200_F16)
    if (op == WB200_RED_SUM) { WB200_RED_FORMATS(WB200_EW_ADD); }
    else if (op == WB200_RED_MAX) { WB200_RED_FORMATS(WB200_EW_MAX); }
    else { WB200_RED_FORMATS(WB200_EW_MIN); }
#undef WB200_RED_FORMATS
#undef WB200_RED_LAUNCH
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

wb200_status launch_pool_formal(int combine, int format, const uint8_t *src, uint8_t *dst, const LayoutMap &src_map,
                                const LayoutMap &dst_map, PoolWindow window, uint32_t *flags_word, cudaStream_t stream) {
  if (dst_map.element_count >= (1ll << 32)) return fail(WB200_ERR_LIMIT, "pooling output has more than 2^32 - 1 elements");
  // Four channels per thread need every channel run, block and slice to start on a multiple of four elements.
  auto by_four = [](const LayoutMap &m) {
    return m.shape[3] % 4 == 0 && m.c_block % 4 == 0 && m.c0 % 4 == 0 && m.outer_slice_stride % 4 == 0;
  };
  const bool vec4 = by_four(src_map) && by_four(dst_map) && all_aligned16(src, dst);
  const int grid = grid_for(dst_map.element_count / (vec4 ? 4 : 1));
#define WB200_POOL_LAUNCH(COMBINE, FORMAT)                                                                                      \
  do {                                                                                                                          \
    if (vec4) formal_pool_kernel<COMBINE, FORMAT, 4><<<grid, kThreads, 0, stream>>>(src, dst, src_map, dst_map, window, flags_word); \
    else formal_pool_kernel<COMBINE, FORMAT, 1><<<grid, kThreads, 0, stream>>>(src, dst, src_map, dst_map, window, flags_word);     \
  } while (0)
#define WB200_POOL_FORMATS(COMBINE)                                             \
  if (format == WB200_F32) WB200_POOL_LAUNCH(COMBINE, WB200_F32);               \
  else if (format == WB200_BF16) WB200_POOL_LAUNCH(COMBINE, WB200_BF16);        \
  else WB200_POOL_LAUNCH(COMBINE, WB200_F16)
  if (combine == WB200_EW_ADD) { WB200_POOL_FORMATS(WB200_EW_ADD); }
  else if (combine == WB200_EW_MAX) { WB200_POOL_FORMATS(WB200_EW_MAX); }
  else { WB200_POOL_FORMATS(WB200_EW_MIN); }
#undef WB200_POOL_FORMATS
#undef WB200_POOL_LAUNCH
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

wb200_status launch_convert(int src_format, int dst_format, const uint8_t *src, uint8_t *dst,
                            const LayoutMap &src_map, const LayoutMap &dst_map, int *nan_flag, cudaStream_t stream) {
  if (!is_float_format(src_format) || !is_float_format(dst_format) || src_map.layout != dst_map.layout || !all_aligned16(src, dst))
    return fail(WB200_ERR_INVALID_ARGUMENT, "convert takes float formats of one layout, 16-byte aligned on the device");
  const StorageWalk walk = storage_walk(src_map, dst_map);
  const int grid = walk_blocks(walk, kThreads);
#define WB200_MCV(SRC, DST) convert_walk_kernel<SRC, DST><<<grid, kThreads, 0, stream>>>(src, dst, walk, nan_flag)
#define WB200_MCV_TO(SRC)                                        \
  if (dst_format == WB200_F32) WB200_MCV(SRC, WB200_F32);        \
  else if (dst_format == WB200_BF16) WB200_MCV(SRC, WB200_BF16); \
  else WB200_MCV(SRC, WB200_F16)
  if (src_format == WB200_F32) { WB200_MCV_TO(WB200_F32); }
  else if (src_format == WB200_BF16) { WB200_MCV_TO(WB200_BF16); }
  else { WB200_MCV_TO(WB200_F16); }
#undef WB200_MCV_TO
#undef WB200_MCV
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

wb200_status launch_reduce(int op, int format, const uint8_t *src, uint8_t *dst, const LayoutMap &src_map,
                           const LayoutMap &dst_map, uint32_t reduced_mask, int *nan_flag, cudaStream_t stream) {
  if (!reduce_one_thread_per_output(src_map, dst_map))
    return launch_fold_staged<false>(op, format, src, dst, src_map, dst_map, reduced_mask, nan_flag, nullptr, stream);
  const int grid = static_cast<int>((dst_map.element_count + kThreads - 1) / kThreads);
#define WB200_MRED(OP, FORMAT) reduce_nhwc_kernel<OP, FORMAT><<<grid, kThreads, 0, stream>>>(src, dst, src_map, dst_map, reduced_mask, nan_flag)
#define WB200_MRED_FORMATS(OP)                                 \
  if (format == WB200_F32) WB200_MRED(OP, WB200_F32);          \
  else if (format == WB200_BF16) WB200_MRED(OP, WB200_BF16);   \
  else WB200_MRED(OP, WB200_F16)
  if (op == WB200_RED_SUM) { WB200_MRED_FORMATS(WB200_RED_SUM); }
  else if (op == WB200_RED_MAX) { WB200_MRED_FORMATS(WB200_RED_MAX); }
  else { WB200_MRED_FORMATS(WB200_RED_MIN); }
#undef WB200_MRED_FORMATS
#undef WB200_MRED
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

wb200_status launch_unpack(const uint8_t *storage, uint8_t *compact, const LayoutMap &map, int element_bytes, cudaStream_t stream) {
  return launch_codec(storage, compact, map, element_bytes, 0, stream);
}
wb200_status launch_unpack_pair(const uint8_t *storage0, uint8_t *compact0, const LayoutMap &map0, const uint8_t *storage1, uint8_t *compact1,
                                const LayoutMap &map1, int element_bytes, int *launches, cudaStream_t stream) {
  if (!codec_takes_units(storage0, compact0, map0, element_bytes) || !codec_takes_units(storage1, compact1, map1, element_bytes)) {
    *launches = 2;
    wb200_status st = launch_unpack(storage0, compact0, map0, element_bytes, stream);
    return st != WB200_OK ? st : launch_unpack(storage1, compact1, map1, element_bytes, stream);
  }
  *launches = 1;
  CodecJobs jobs;
  jobs.job[0] = codec_job(storage0, compact0, map0, element_bytes);
  jobs.job[1] = codec_job(storage1, compact1, map1, element_bytes);
  const dim3 grid(grid_for(jobs.job[0].units > jobs.job[1].units ? jobs.job[0].units : jobs.job[1].units), 2);
  if (element_bytes == 2) codec_wide_kernel<8><<<grid, kThreads, 0, stream>>>(jobs, 0);
  else codec_wide_kernel<4><<<grid, kThreads, 0, stream>>>(jobs, 0);
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}
wb200_status launch_pack(const uint8_t *compact, uint8_t *storage, const LayoutMap &map, int element_bytes, cudaStream_t stream) {
  return launch_codec(compact, storage, map, element_bytes, 1, stream);
}

}  // namespace wb200
