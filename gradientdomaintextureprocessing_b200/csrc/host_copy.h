// Copies between the caller's host vectors and device buffers.
//
// Pageable memory (what callers usually hold) goes through two pinned chunks of this
// object: several host threads move a chunk while the copy engine moves the other.
// A plain copy of pageable memory is one driver thread's, and a fresh destination is
// faulted in page by page by that thread: 64 geodesic sources at 1024^2 (182 MB of
// distances) took 63.3 ms, now 40.8, the difference all here.  Pinned memory, and copies too
// small to gain from threads, are plain copies.
//
// One object per stream user (not for concurrent calls); the chunks are allocated on
// the first staged copy and freed with the object.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace gdtp {

class HostCopy {
 public:
  HostCopy() = default;
  HostCopy(const HostCopy&) = delete;
  HostCopy& operator=(const HostCopy&) = delete;
  ~HostCopy();
  // device <- host, queued on s; the host memory may change once this returns
  // unless it is pinned (then once the stream has passed the copy)
  cudaError_t upload(void* device, const void* host, size_t bytes, cudaStream_t s);
  // host <- device after the work queued on s; complete when this returns
  cudaError_t download(void* host, const void* device, size_t bytes, cudaStream_t s);

 private:
  static constexpr size_t kChunk = size_t(4) << 20;
  static constexpr size_t kStagedMin = size_t(1) << 20;
  static constexpr int kSlots = 2;
  bool staged(const void* host, size_t bytes);
  unsigned char* chunks_ = nullptr;  // kSlots x kChunk, pinned
  cudaEvent_t done_[kSlots] = {};
  bool failed_ = false;              // no pinned memory to be had: plain copies
};

}  // namespace gdtp
