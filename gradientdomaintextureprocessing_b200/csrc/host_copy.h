// Copies between the caller's host vectors and device buffers.
//
// Pageable memory (what callers usually hold) goes through two pinned chunks of this
// object: several host threads move a chunk while the copy engine moves the other.
// A plain copy of pageable memory is one driver thread's, and a fresh destination is
// faulted in page by page by that thread: 64 geodesic sources at 1024^2 (182 MB of
// distances) took 63.3 ms, now 40.8, the difference all here.  A vector there and
// back (an operator call), plain against staged: 8.6 MB 1.02 / 0.65 ms, 22.8 MB 2.6 /
// 1.2, 91 MB 27 / 8.2, 183 MB 55 / 16.6 (chunks of 2 and 4 MB 29 and 23; 10 or 14
// threads the same: fresh pages bound it); a V-cycle on 3.4 MB vectors 1.24 / 0.86.
// Below 2 MB waking the threads costs what the copy gains,
// so those, and pinned memory, are plain copies.  The threads sleep between transfers:
// an OpenMP team's idle spin cost the caller's next host operation 0.2 ms and more
// (drawing 1 of 512^2 sources 0.53 -> 2.46 ms after a solve; with these 0.41 on both).
//
// One object per device, shared by its systems (each with its own held 16 MB of pinned
// memory and 5 threads per model that ever saw a large vector).  Calls may overlap, from
// several threads and on several streams: each takes a set of chunks and threads for its
// whole length, one that is free; at most kMaxSets are made, and a call that finds none
// makes a plain copy.  A set costs more than a copy gains (pinned memory: 2 MB 2.9 to
// 5.8 ms, 4 MB 2.2 to 6.4, 16 MB 7.5 to 22; a vector there and back 0.15 ms at 2.5 MB, 0.9
// at 17), so one is made once plain copies have moved kPayback bytes, of the size that the
// copy at hand needs: a program of a few calls makes none.  The sets go with the last
// system of the device.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <memory>
#include <mutex>
#include <vector>

namespace gdtp {

class HostCopy {
 public:
  // the device's object, made here when no system has it
  static std::shared_ptr<HostCopy> of_device(int device);
  // payback: plain copies before a set is made, bytes
  explicit HostCopy(size_t payback = kPayback);
  HostCopy(const HostCopy&) = delete;
  HostCopy& operator=(const HostCopy&) = delete;
  ~HostCopy();
  // device <- host, queued on s; the host memory may change once this returns
  // unless it is pinned (then once the stream has passed the copy)
  cudaError_t upload(void* device, const void* host, size_t bytes, cudaStream_t s);
  // host <- device after the work queued on s; complete when this returns
  cudaError_t download(void* host, const void* device, size_t bytes, cudaStream_t s);

 private:
  class Workers;
  struct Set;
  struct Transfer;
  static constexpr size_t kPayback = size_t(64) << 20;
  static constexpr size_t kChunkMax = size_t(8) << 20;
  static constexpr size_t kChunkMin = size_t(1) << 20;
  static constexpr size_t kStagedMin = size_t(2) << 20;
  static constexpr int kSlots = 2;
  static constexpr size_t kMaxSets = 4;
  // a set for one copy on s, null for a plain copy; the caller returns it
  Set* take(const void* host, size_t bytes, cudaStream_t s);
  void give(Set* set);
  static size_t piece(size_t bytes);
  const size_t payback_;
  std::mutex m_;                            // guards the rest
  std::vector<std::unique_ptr<Set>> sets_;
  size_t plain_ = 0;                        // moved by plain copies since the last set was made
  bool failed_ = false;                     // no pinned memory to be had: plain copies
};

}  // namespace gdtp
