// Host storage in and out of one command call. The reference hands commands over as pageable host vectors; a pageable
// cudaMemcpyAsync costs 10-40 us each (driver staging and, for results, a synchronisation of its own), more than the
// commands themselves. Storage goes through one pinned, device-mapped area of the backend instead:
//   up to kMappedBytes per operand (or result) the kernel reads (writes) the area directly over PCIe, where it
//   touches a byte once and in whole groups, so there is no copy command at all;
//   storage in device memory (operands read several times, results stored element by element, anything larger) is copied
//   through the area up to kPieceBytes, larger operands by the driver; larger results come back through the area in pieces, so
//   that the CPU copy of a piece overlaps the DMA of the next.
// Storage that is page-locked already (the results the Python layer hands out, see ResultPool; a caller's own pinned
// memory) is read and written where it lies, so a chain of commands copies nothing between its calls.
// One synchronisation ends the call. A result is copied to the caller only after the call's status words are known.
#pragma once

#include "backend.h"

namespace wb200 {

class CommandIO {
 public:
  static constexpr size_t kMappedBytes = size_t(1) << 20;
  static constexpr size_t kPieceBytes = size_t(1) << 20;
  static constexpr int64_t kScattered = 4 << 10;

  // `expected` bytes of host storage will pass through the call (sizes the pinned area, up to its limit).
  CommandIO(wb200_backend *backend, size_t expected) : backend_(backend), stream_(backend->stream) {
    status_ = backend->stage_reserve(expected);
  }
  // A call that fails half way leaves copies in flight out of the area the next call will fill.
  ~CommandIO() {
    if (!finished_) cudaStreamSynchronize(stream_);
  }
  CommandIO(const CommandIO &) = delete;
  CommandIO &operator=(const CommandIO &) = delete;
  wb200_status status() const { return status_; }

  // An operand. `reread`: the kernels read it more than once, so it belongs in device memory (slot `slot`).
  wb200_status input(size_t slot, const uint8_t *host, size_t bytes, const uint8_t **device, bool reread = false) {
    const bool pinned = page_locked(host, bytes);
    held_[held_count_] = host;   // it may be read by the kernels or by a copy in flight after output() has run
    held_bytes_[held_count_++] = bytes;
    if (pinned && !reread) {
      *device = host;
      return WB200_OK;
    }
    if (!reread && bytes <= kMappedBytes) {
      uint8_t *area = take(bytes);
      if (area) {
        memcpy(area, host, bytes);
        *device = area;
        return WB200_OK;
      }
    }
    void *buffer;
    wb200_status st = backend_->buffer(slot, bytes, &buffer);
    if (st != WB200_OK) return st;
    *device = static_cast<uint8_t *>(buffer);
    if (pinned) {
      WB200_CUDA_CHECK(cudaMemcpyAsync(buffer, host, bytes, cudaMemcpyHostToDevice, stream_));
      return WB200_OK;
    }
    return upload(buffer, host, bytes);
  }

  // The result, after all operands. `padded`: its layout has bytes that are no element, which keep the template's values.
  // `host` is where deliver() puts it. `scattered`: elements the kernel stores one by one, at about 1.3 ns each over PCIe, so that
  // a larger result goes through device memory and one copy from there (bit-exact GEMM, 1001 x 1003 bf16: 1783 against 619 us
  // in all, 256 x 520 f32 429 against 290; a formal convert of 2 x 5 x 7 x 97 83 against 70; 64 x 64 f32 GEMM 38 against 44).
  wb200_status output(size_t slot, const uint8_t *storage_template, uint8_t *host, size_t bytes, bool padded, uint8_t **device, int64_t scattered = 0) {
    bytes_ = bytes;
    if (scattered > kScattered) {
      wb200_status st = device_output(slot, storage_template, bytes, padded, device);
      if (st != WB200_OK) return st;
      if (page_locked(host, bytes)) {   // the copy reaches it in stream order, behind everything that reads the operands
        in_place_result_ = true;
        copied_result_ = host;
      } else if (bytes <= kMappedBytes && (mapped_ = take(bytes)) != nullptr) {
        copied_result_ = mapped_;
        device_ = nullptr;
      }
      return WB200_OK;
    }
    bool overlaps = false;
    for (int i = 0; i < held_count_; ++i) overlaps |= host < held_[i] + held_bytes_[i] && held_[i] < host + bytes;
    if (!overlaps && page_locked(host, bytes)) {
      if (padded && host != storage_template) memmove(host, storage_template, bytes);
      *device = host;
      in_place_result_ = true;
      return WB200_OK;
    }
    if (bytes <= kMappedBytes && (mapped_ = take(bytes)) != nullptr) {
      if (padded) memcpy(mapped_, storage_template, bytes);
      *device = mapped_;
      return WB200_OK;
    }
    return device_output(slot, storage_template, bytes, padded, device);
  }

  // Host storage into device memory of the caller's.
  wb200_status copy_in(void *device, const uint8_t *host, size_t bytes) {
    if (!page_locked(host, bytes)) return upload(device, host, bytes);
    WB200_CUDA_CHECK(cudaMemcpyAsync(device, host, bytes, cudaMemcpyHostToDevice, stream_));
    return WB200_OK;
  }
  // Device memory of the caller's to host storage that is written by deliver_copies() alone, after the caller has accepted what
  // finish() brought: storage that is not page-locked is fetched into the area ahead of it, the rest is copied then.
  wb200_status copy_out(uint8_t *host, const void *device, size_t bytes) {
    const uint8_t *from = static_cast<const uint8_t *>(device);
    if (page_locked(host, bytes)) {
      direct_.push_back({host, from, bytes});
      return WB200_OK;
    }
    uint8_t *area = take(bytes);
    if (!area) {   // larger than the area: piece by piece after the rest
      late_.push_back({host, from, bytes});
      return WB200_OK;
    }
    copies_.push_back({host, area, bytes});
    WB200_CUDA_CHECK(cudaMemcpyAsync(area, device, bytes, cudaMemcpyDeviceToHost, stream_));
    return WB200_OK;
  }
  wb200_status deliver_copies() {
    for (const Copy &copy : direct_) WB200_CUDA_CHECK(cudaMemcpyAsync(copy.host, copy.from, copy.bytes, cudaMemcpyDeviceToHost, stream_));
    for (const Copy &copy : copies_) memcpy(copy.host, copy.from, copy.bytes);
    for (const Copy &copy : late_) {
      device_ = copy.from;
      bytes_ = copy.bytes;
      wb200_status st = deliver(copy.host);
      if (st != WB200_OK) return st;
    }
    if (!direct_.empty()) WB200_CUDA_CHECK(cudaStreamSynchronize(stream_));
    return WB200_OK;
  }

  // The device words (flags, refusals) a call reads back with its result: at most kStageWordBytes, once per call. Their place
  // lies behind the operands' area, which uploads may have filled to the last byte.
  wb200_status read_back(const void *device_word, size_t bytes, const uint8_t **host) {
    uint8_t *area = backend_->stage + backend_->stage_bytes;
    WB200_CUDA_CHECK(cudaMemcpyAsync(area, device_word, bytes, cudaMemcpyDeviceToHost, stream_));
    *host = area;
    return WB200_OK;
  }

  // Ends the device part: everything enqueued has run, the status words are read (and cleared), words of read_back() are
  // there. *nan_flag as in read_device_status().
  wb200_status finish(int *nan_flag) {
    if (copied_result_) WB200_CUDA_CHECK(cudaMemcpyAsync(copied_result_, result_, bytes_, cudaMemcpyDeviceToHost, stream_));
    finished_ = true;
    return read_device_status(backend_, stream_, nan_flag);
  }

  // Copies the result to the caller (after finish(), and after the caller has accepted the status).
  wb200_status deliver(uint8_t *host) {
    if (in_place_result_) return WB200_OK;
    if (!device_) {
      memcpy(host, mapped_, bytes_);
      return WB200_OK;
    }
    // two halves of the area alternate: the DMA of a piece overlaps the CPU copy of the one before
    const size_t piece = kPieceBytes < backend_->stage_bytes / 2 ? kPieceBytes : backend_->stage_bytes / 2;
    wb200_status st = backend_->auxiliary_streams();   // for the events
    if (st != WB200_OK) return st;
    const size_t pieces = (bytes_ + piece - 1) / piece;
    auto size_of = [&](size_t i) { return i + 1 < pieces ? piece : bytes_ - (pieces - 1) * piece; };
    auto issue = [&](size_t i) -> wb200_status {
      WB200_CUDA_CHECK(cudaMemcpyAsync(backend_->stage + (i & 1) * piece, device_ + i * piece, size_of(i), cudaMemcpyDeviceToHost, stream_));
      WB200_CUDA_CHECK(cudaEventRecord(backend_->aux_event[i & 1], stream_));
      return WB200_OK;
    };
    for (size_t i = 0; i < pieces && i < 2; ++i)
      if ((st = issue(i)) != WB200_OK) return st;
    for (size_t i = 0; i < pieces; ++i) {
      WB200_CUDA_CHECK(cudaEventSynchronize(backend_->aux_event[i & 1]));
      memcpy(host + i * piece, backend_->stage + (i & 1) * piece, size_of(i));
      if (i + 2 < pieces && (st = issue(i + 2)) != WB200_OK) return st;
    }
    return WB200_OK;
  }

 private:
  // Page-locked from the first byte to the last (a caller may have registered only a part) and 16-byte aligned. Small
  // operands are not worth the query.
  static bool page_locked(const void *host, size_t bytes) {
    return bytes >= 16384 && (reinterpret_cast<uintptr_t>(host) & 15u) == 0 && page_locked_range(host, bytes);
  }
  // What kernels access in place lies at the end of the area, pieces on their way to device memory at its start.
  uint8_t *take(size_t bytes) {
    const size_t rounded = (bytes + 255) / 256 * 256;
    if (backend_->stage_low + rounded > backend_->stage_high) return nullptr;
    backend_->stage_high -= rounded;
    return backend_->stage + backend_->stage_high;
  }
  wb200_status device_output(size_t slot, const uint8_t *storage_template, size_t bytes, bool padded, uint8_t **device) {
    void *buffer;
    wb200_status st = backend_->buffer(slot, bytes, &buffer);
    if (st != WB200_OK) return st;
    *device = static_cast<uint8_t *>(buffer);
    device_ = result_ = *device;
    return padded ? upload(buffer, storage_template, bytes) : WB200_OK;
  }
  // Through the area up to kPieceBytes; beyond, the driver's own copy of pageable memory is faster (reduce of 8 / 32 MB 422 / 1423
  // us in all against 540 / 2060 in pieces of 1 MB; 64 KB 99 against 65). Either has read pageable
  // `host` when it returns.
  wb200_status upload(void *device, const uint8_t *host, size_t bytes) {
    if (bytes > kPieceBytes) {
      WB200_CUDA_CHECK(cudaMemcpyAsync(device, host, bytes, cudaMemcpyHostToDevice, stream_));
      return WB200_OK;
    }
    if (backend_->stage_low + bytes > backend_->stage_high) {
      WB200_CUDA_CHECK(cudaStreamSynchronize(stream_));   // the pieces have left the area
      backend_->stage_low = 0;
      if (bytes > backend_->stage_high) return fail(WB200_ERR_LIMIT, "command staging area exhausted");
    }
    uint8_t *piece = backend_->stage + backend_->stage_low;
    backend_->stage_low += bytes;
    memcpy(piece, host, bytes);
    WB200_CUDA_CHECK(cudaMemcpyAsync(device, piece, bytes, cudaMemcpyHostToDevice, stream_));
    return WB200_OK;
  }

  wb200_backend *backend_;
  cudaStream_t stream_;
  wb200_status status_;
  struct Copy { uint8_t *host; const uint8_t *from; size_t bytes; };
  std::vector<Copy> direct_, copies_, late_;
  uint8_t *mapped_ = nullptr;                              // the result in the area,
  const uint8_t *device_ = nullptr;                        // or in device memory, to be brought in pieces
  const uint8_t *result_ = nullptr;                        // where the kernels put a result of device_output(),
  uint8_t *copied_result_ = nullptr;                       // and where finish() copies it
  bool in_place_result_ = false, finished_ = false;
  const uint8_t *held_[4];      // the operands: a page-locked result that overlaps one is written only after they have been read
  size_t held_bytes_[4];
  int held_count_ = 0;
  size_t bytes_ = 0;
};

}  // namespace wb200
