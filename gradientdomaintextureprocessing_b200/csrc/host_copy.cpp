// Copies between the caller's host vectors and device buffers (host_copy.h).
#include "host_copy.h"

#include <omp.h>

#include <algorithm>
#include <cstring>

namespace gdtp {
namespace {

// memcpy by up to kThreads threads, at least kPiece bytes each
constexpr size_t kPiece = size_t(512) << 10;
constexpr int kThreads = 8;
void copy_parallel(void* dst, const void* src, size_t bytes) {
  const int threads = int(std::min<size_t>(std::min(kThreads, omp_get_max_threads()), bytes / kPiece));
  if (threads <= 1) {
    std::memcpy(dst, src, bytes);
    return;
  }
  const size_t part = ((bytes + threads - 1) / threads + 4095) & ~size_t(4095);
#pragma omp parallel for num_threads(threads) schedule(static, 1)
  for (int t = 0; t < threads; t++) {
    const size_t at = part * size_t(t);
    if (at < bytes) std::memcpy(static_cast<char*>(dst) + at, static_cast<const char*>(src) + at, std::min(part, bytes - at));
  }
}

}  // namespace

HostCopy::~HostCopy() {
  for (cudaEvent_t e : done_)
    if (e) cudaEventDestroy(e);
  if (chunks_) cudaFreeHost(chunks_);
}

// the copy goes through the pinned chunks (allocated here on first use)
bool HostCopy::staged(const void* host, size_t bytes) {
  if (failed_ || bytes < kStagedMin) return false;
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (at.type != cudaMemoryTypeUnregistered) return false;
  if (chunks_) return true;
  void* p = nullptr;
  bool ok = cudaHostAlloc(&p, kSlots * kChunk, cudaHostAllocDefault) == cudaSuccess;
  for (cudaEvent_t& e : done_) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    if (p) cudaFreeHost(p);
    failed_ = true;
    return false;
  }
  chunks_ = static_cast<unsigned char*>(p);
  return true;
}

cudaError_t HostCopy::upload(void* device, const void* host, size_t bytes, cudaStream_t s) {
  if (!staged(host, bytes)) return cudaMemcpyAsync(device, host, bytes, cudaMemcpyHostToDevice, s);
  int slot = 0;
  for (size_t at = 0; at < bytes; at += kChunk, slot ^= 1) {
    const size_t len = std::min(kChunk, bytes - at);
    unsigned char* chunk = chunks_ + slot * kChunk;
    // the chunk's last copy (of this call or an earlier one) has left it
    cudaError_t e = cudaEventSynchronize(done_[slot]);
    if (e != cudaSuccess) return e;
    copy_parallel(chunk, static_cast<const char*>(host) + at, len);
    e = cudaMemcpyAsync(static_cast<char*>(device) + at, chunk, len, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaEventRecord(done_[slot], s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t HostCopy::download(void* host, const void* device, size_t bytes, cudaStream_t s) {
  if (!staged(host, bytes)) {
    const cudaError_t e = cudaMemcpyAsync(host, device, bytes, cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
  }
  // stream order keeps these copies behind an upload that still reads a chunk
  auto queue = [&](size_t at, int slot) -> cudaError_t {
    const cudaError_t e = cudaMemcpyAsync(chunks_ + slot * kChunk, static_cast<const char*>(device) + at, std::min(kChunk, bytes - at),
                                          cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaEventRecord(done_[slot], s) : e;
  };
  cudaError_t e = queue(0, 0);
  int slot = 0;
  for (size_t at = 0; at < bytes && e == cudaSuccess; at += kChunk, slot ^= 1) {
    if (at + kChunk < bytes) e = queue(at + kChunk, slot ^ 1);
    if (e == cudaSuccess) e = cudaEventSynchronize(done_[slot]);
    if (e == cudaSuccess) copy_parallel(static_cast<char*>(host) + at, chunks_ + slot * kChunk, std::min(kChunk, bytes - at));
  }
  if (e != cudaSuccess) cudaStreamSynchronize(s);  // nothing is left writing the chunks
  return e;
}

}  // namespace gdtp
