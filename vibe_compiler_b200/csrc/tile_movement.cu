// Movement commands of the TargetCall ABI on device-resident memory images: strided DMA (DDR <-> scratch-pad),
// gather / scatter inside a scratch-pad, element fill. A strided byte layout is {inner_bytes, strides[3],
// iterations[3]}; its segments are enumerated with dimension 0 fastest and the payload is their concatenation
// (lib/Wafer/Simulator/Memory/TargetModelStridedMemory.cpp:121-152). A copy pairs payload byte p of the source
// layout with payload byte p of the destination layout (lib/Wafer/Simulator/Kernel/TargetModelMovement.cpp:52-146).
// HBM-bound byte work: algorithmic bytes = payload read once + written once.
#include <algorithm>

#include "kernels.h"
#include "ptx_sm100.cuh"

namespace wb200 {
namespace {

// blockIdx.y = copy, blockIdx.z = Tile.
template <int kJobs>
struct CopyJobs {
  CopyJob job[kJobs];
};
template <typename Unit, int kJobs>
__global__ void __launch_bounds__(256) strided_copy_kernel(const __grid_constant__ CopyJobs<kJobs> jobs) {
  const CopyJob &job = jobs.job[kJobs == 1 ? 0 : blockIdx.y];
  const StridedLayout &from = job.from, &to = job.to;
  const uint32_t units_per_segment = job.units_per_segment;
  pdl_launch_dependents();
  pdl_wait();
  const uint8_t *src = job.src + blockIdx.z * job.src_step;
  uint8_t *dst = job.dst + blockIdx.z * job.dst_step;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t u = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; u < job.total_units; u += stride) {
    // a command moves at most 4 GiB, so 32-bit division is enough (64-bit division is several times slower)
    const uint32_t unit = static_cast<uint32_t>(u);
    const uint32_t segment = unit / units_per_segment;
    const uint64_t within = static_cast<uint64_t>(unit - segment * units_per_segment) * sizeof(Unit);
    uint32_t s = segment, t = segment;
    uint64_t from_offset = within, to_offset = within;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const uint32_t s_next = s / from.iterations[d], t_next = t / to.iterations[d];
      from_offset += static_cast<uint64_t>(s - s_next * from.iterations[d]) * from.strides[d];
      to_offset += static_cast<uint64_t>(t - t_next * to.iterations[d]) * to.strides[d];
      s = s_next;
      t = t_next;
    }
    *reinterpret_cast<Unit *>(dst + to_offset) = *reinterpret_cast<const Unit *>(src + from_offset);
  }
}

template <typename Element>
__global__ void __launch_bounds__(256) fill_kernel(Element *dst, Element value, uint64_t count, uint64_t tile_stride) {
  pdl_launch_dependents();
  pdl_wait();
  dst += blockIdx.z * (tile_stride / sizeof(Element));
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride) dst[i] = value;
}

// wafer_tx81_bit2fp (lib/Wafer/Simulator/Kernel/TargetModelTensorNumeric.cpp:198-236): bit i of the packed Bool source
// (least significant bit first) becomes 1.0 or +0 of the destination format.
template <typename T>
__global__ void __launch_bounds__(256) bit2fp_kernel(const uint8_t *src, T *dst, uint32_t count, T one) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) dst[i] = ((src[i >> 3] >> (i & 7)) & 1u) ? one : static_cast<T>(0);
}

// wafer_tx81_mask_move (:238-286): destination elements whose mask element is exactly 1.0 take the source element, a
// zero mask keeps them; any other mask value refuses the command. `store` = 0 only validates; the smallest refused
// element is reported as (element << 8 | 4).
template <typename T>
__global__ void __launch_bounds__(256) mask_move_kernel(const T *src, const T *mask, T *dst, uint32_t count, T one, int store,
                                                        unsigned long long *first_refused) {
  const uint32_t stride = gridDim.x * blockDim.x;
  unsigned long long refused = ~0ull;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    const T predicate = mask[i];
    if (predicate == one) {
      if (store) dst[i] = src[i];
    } else if (predicate != 0) {
      const unsigned long long key = (static_cast<unsigned long long>(i) << 8) | 4ull;
      refused = key < refused ? key : refused;
    }
  }
  if (refused != ~0ull) atomicMin(first_refused, refused);
}

int grid_for(uint64_t items) {
  uint64_t blocks = (items + 255) / 256;
  if (blocks > 148u * 8u) blocks = 148u * 8u;
  return blocks == 0 ? 1 : static_cast<int>(blocks);
}

bool layout_aligned(const StridedLayout &layout, uint32_t unit) {
  if (layout.inner_bytes % unit) return false;
  for (int d = 0; d < 3; ++d)
    if (layout.iterations[d] > 1 && layout.strides[d] % unit) return false;
  return true;
}

}  // namespace

uint64_t strided_segments(const StridedLayout &layout) {
  return static_cast<uint64_t>(layout.iterations[0]) * layout.iterations[1] * layout.iterations[2];
}

uint64_t strided_span(const StridedLayout &layout) {
  uint64_t span = layout.inner_bytes;
  for (int d = 0; d < 3; ++d)
    if (layout.iterations[d] > 1) span += static_cast<uint64_t>(layout.iterations[d] - 1) * layout.strides[d];
  return span;
}

wb200_status make_copy_job(const uint8_t *src, const StridedLayout &from, uint8_t *dst, const StridedLayout &to, uint32_t tiles, int64_t src_step,
                           int64_t dst_step, CopyJob *job) {
  if (from.inner_bytes == 0 || from.inner_bytes != to.inner_bytes)
    return fail(WB200_ERR_INVALID_ARGUMENT, "strided copy needs equal, non-zero inner byte counts");
  for (int d = 0; d < 3; ++d)
    if (from.iterations[d] == 0 || to.iterations[d] == 0) return fail(WB200_ERR_INVALID_ARGUMENT, "strided copy iteration counts must be positive");
  const uint64_t segments = strided_segments(from);
  if (segments != strided_segments(to)) return fail(WB200_ERR_INVALID_ARGUMENT, "source and destination segment counts differ");
  // every Tile's addresses have to allow the unit
  const uintptr_t bases = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst) |
                          (tiles > 1 ? static_cast<uintptr_t>(src_step) | static_cast<uintptr_t>(dst_step) : 0);
  const uint32_t unit = bases % 16 == 0 && layout_aligned(from, 16) && layout_aligned(to, 16) ? 16
                        : bases % 4 == 0 && layout_aligned(from, 4) && layout_aligned(to, 4)  ? 4
                                                                                              : 1;
  *job = {src, dst, from, to, from.inner_bytes / unit, unit, segments * from.inner_bytes / unit, src_step, dst_step};
  return WB200_OK;
}

namespace {
template <int kJobs>
cudaError_t launch_copies(const CopyJob *jobs, int count, uint32_t tiles, cudaStream_t stream) {
  CopyJobs<kJobs> args{};
  uint64_t longest = 0;
  for (int i = 0; i < count; ++i) {
    args.job[i] = jobs[i];
    longest = std::max(longest, jobs[i].total_units);
  }
  const dim3 grid(grid_for(longest), count, tiles);
  if (jobs[0].unit == 16) return launch_dependent(strided_copy_kernel<uint4, kJobs>, grid, 256, 0, stream, args);
  if (jobs[0].unit == 4) return launch_dependent(strided_copy_kernel<uint32_t, kJobs>, grid, 256, 0, stream, args);
  return launch_dependent(strided_copy_kernel<uint8_t, kJobs>, grid, 256, 0, stream, args);
}
}  // namespace

wb200_status launch_copy_jobs(const CopyJob *jobs, int count, uint32_t tiles, cudaStream_t stream) {
  if (count < 1 || count > kMaxCopyJobs) return fail(WB200_ERR_INVALID_ARGUMENT, "unsupported number of copies");
  for (int i = 1; i < count; ++i)
    if (jobs[i].unit != jobs[0].unit) return fail(WB200_ERR_INVALID_ARGUMENT, "copies of one launch have one unit");
  if (count == 1) WB200_CUDA_CHECK(launch_copies<1>(jobs, count, tiles, stream));
  else WB200_CUDA_CHECK(launch_copies<kMaxCopyJobs>(jobs, count, tiles, stream));
  return WB200_OK;
}

wb200_status launch_strided_copy(const uint8_t *src, const StridedLayout &from, uint8_t *dst, const StridedLayout &to,
                                 cudaStream_t stream, uint32_t tiles, int64_t src_step, int64_t dst_step) {
  CopyJob job;
  const wb200_status st = make_copy_job(src, from, dst, to, tiles, src_step, dst_step, &job);
  return st != WB200_OK ? st : launch_copy_jobs(&job, 1, tiles, stream);
}

wb200_status launch_fill(uint8_t *dst, uint32_t value_bits, uint64_t count, int element_bytes, cudaStream_t stream, TileBatch tiles) {
  if (count == 0) return WB200_OK;
  if (reinterpret_cast<uintptr_t>(dst) % element_bytes || (tiles.tiles > 1 && tiles.stride % element_bytes)) return fail(WB200_ERR_INVALID_ARGUMENT, "fill destination is not element aligned");
  switch (element_bytes) {
    case 1: WB200_CUDA_CHECK(launch_dependent(fill_kernel<uint8_t>, dim3(grid_for(count), 1, tiles.tiles), 256, 0, stream, dst, static_cast<uint8_t>(value_bits), count, tiles.stride)); break;
    case 2: WB200_CUDA_CHECK(launch_dependent(fill_kernel<uint16_t>, dim3(grid_for(count), 1, tiles.tiles), 256, 0, stream, reinterpret_cast<uint16_t *>(dst), static_cast<uint16_t>(value_bits), count, tiles.stride)); break;
    case 4: WB200_CUDA_CHECK(launch_dependent(fill_kernel<uint32_t>, dim3(grid_for(count), 1, tiles.tiles), 256, 0, stream, reinterpret_cast<uint32_t *>(dst), value_bits, count, tiles.stride)); break;
    default: return fail(WB200_ERR_UNSUPPORTED, "fill takes 1, 2 or 4 byte elements");
  }
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

wb200_status launch_bit2fp(const uint8_t *src, uint8_t *dst, uint32_t count, int format, cudaStream_t stream) {
  if (count == 0) return WB200_OK;
  const int grid = grid_for(count);
  if (format == WB200_F32) bit2fp_kernel<uint32_t><<<grid, 256, 0, stream>>>(src, reinterpret_cast<uint32_t *>(dst), count, 0x3f800000u);
  else if (format == WB200_BF16) bit2fp_kernel<uint16_t><<<grid, 256, 0, stream>>>(src, reinterpret_cast<uint16_t *>(dst), count, static_cast<uint16_t>(0x3f80));
  else if (format == WB200_F16) bit2fp_kernel<uint16_t><<<grid, 256, 0, stream>>>(src, reinterpret_cast<uint16_t *>(dst), count, static_cast<uint16_t>(0x3c00));
  else return fail(WB200_ERR_UNSUPPORTED, "Bit2FP requires F16, BF16 or F32 output");
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

wb200_status launch_mask_move(const uint8_t *src, const uint8_t *mask, uint8_t *dst, uint32_t count, int format, int store,
                              unsigned long long *first_refused, cudaStream_t stream) {
  if (count == 0) return WB200_OK;
  const int grid = grid_for(count);
  if (format == WB200_F32)
    mask_move_kernel<uint32_t><<<grid, 256, 0, stream>>>(reinterpret_cast<const uint32_t *>(src), reinterpret_cast<const uint32_t *>(mask),
                                                         reinterpret_cast<uint32_t *>(dst), count, 0x3f800000u, store, first_refused);
  else if (format == WB200_BF16 || format == WB200_F16)
    mask_move_kernel<uint16_t><<<grid, 256, 0, stream>>>(reinterpret_cast<const uint16_t *>(src), reinterpret_cast<const uint16_t *>(mask),
                                                         reinterpret_cast<uint16_t *>(dst), count,
                                                         static_cast<uint16_t>(format == WB200_BF16 ? 0x3f80 : 0x3c00), store, first_refused);
  else return fail(WB200_ERR_UNSUPPORTED, "MaskMove requires F16, BF16 or F32");
  WB200_CUDA_CHECK(cudaGetLastError());
  return WB200_OK;
}

}  // namespace wb200
