// Copies between the caller's host vectors and device buffers (host_copy.h).
#include "host_copy.h"

#include <sched.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace gdtp {

// memcpy by the caller and a few workers.  The workers sleep between transfers (an
// OpenMP team spins for some milliseconds after its work, which slowed the caller's own
// threads: 0.2 ms and more on the next host operation) and poll within one, since its
// chunks follow one another in tens of microseconds.
class HostCopy::Workers {
 public:
  Workers() {
    cpu_set_t set;
    CPU_ZERO(&set);
    threads_.reserve(kThreads);
    const int cpus = sched_getaffinity(0, sizeof(set), &set) == 0 ? CPU_COUNT(&set) : 1;
    try {
      for (int t = 1; t < std::min(kThreads, cpus); t++) threads_.emplace_back([this] { work(); });
    } catch (const std::system_error&) {  // fewer, or none: the caller copies by itself
    }
  }
  ~Workers() {
    {
      std::lock_guard<std::mutex> l(m_);
      stop_ = true;
    }
    wake_.notify_all();
    for (std::thread& t : threads_) t.join();
  }
  // begin() wakes the workers for a transfer, end() sends them back to sleep
  void begin() {
    {
      std::lock_guard<std::mutex> l(m_);
      active_ = true;
    }
    wake_.notify_all();
  }
  void end() {
    std::lock_guard<std::mutex> l(m_);
    active_ = false;
    turn_.fetch_add(1);
  }
  void copy(void* dst, const void* src, size_t bytes) {
    std::unique_lock<std::mutex> l(m_);
    dst_ = static_cast<char*>(dst);
    src_ = static_cast<const char*>(src);
    bytes_ = bytes;
    at_ = 0;
    turn_.fetch_add(1);
    while (take(l)) {}
    while (busy_ > 0) {  // a worker is in its last piece
      l.unlock();
      std::this_thread::yield();
      l.lock();
    }
  }

 private:
  static constexpr size_t kPiece = size_t(128) << 10;
  static constexpr int kThreads = 6;
  // copies the next piece with the lock released; false when none is left
  bool take(std::unique_lock<std::mutex>& l) {
    if (at_ >= bytes_) return false;
    const size_t at = at_, len = std::min(kPiece, bytes_ - at);
    at_ += len;
    busy_++;
    char* d = dst_ + at;
    const char* s = src_ + at;
    l.unlock();
    std::memcpy(d, s, len);
    l.lock();
    busy_--;
    return true;
  }
  void work() {
    std::unique_lock<std::mutex> l(m_);
    for (;;) {
      wake_.wait(l, [this] { return stop_ || active_; });
      if (stop_) return;
      while (active_) {
        while (take(l)) {}
        const unsigned turn = turn_.load();
        if (!active_) break;
        l.unlock();
        while (turn_.load() == turn) std::this_thread::yield();
        l.lock();
      }
    }
  }
  std::mutex m_;
  std::condition_variable wake_;
  std::atomic<unsigned> turn_{0};  // a new chunk, or the transfer's end
  bool active_ = false, stop_ = false;
  char* dst_ = nullptr;
  const char* src_ = nullptr;
  size_t bytes_ = 0, at_ = 0;
  int busy_ = 0;
  std::vector<std::thread> threads_;
};

// the workers are awake while this is in scope
struct HostCopy::Transfer {
  explicit Transfer(Workers& w) : w(w) { w.begin(); }
  ~Transfer() { w.end(); }
  Workers& w;
};

HostCopy::HostCopy() = default;

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
  workers_ = std::make_unique<Workers>();
  return true;
}

// a quarter of the vector, so that the two sides overlap, within the chunk's size
size_t HostCopy::piece(size_t bytes) { return std::min(kChunk, std::max(kChunkMin, bytes / 4)); }

cudaError_t HostCopy::upload(void* device, const void* host, size_t bytes, cudaStream_t s) {
  if (!staged(host, bytes)) return cudaMemcpyAsync(device, host, bytes, cudaMemcpyHostToDevice, s);
  const size_t step = piece(bytes);
  Transfer transfer(*workers_);
  int slot = 0;
  for (size_t at = 0; at < bytes; at += step, slot ^= 1) {
    const size_t len = std::min(step, bytes - at);
    unsigned char* chunk = chunks_ + slot * kChunk;
    // the chunk's last copy (of this call or an earlier one) has left it
    cudaError_t e = cudaEventSynchronize(done_[slot]);
    if (e != cudaSuccess) return e;
    workers_->copy(chunk, static_cast<const char*>(host) + at, len);
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
  const size_t step = piece(bytes);
  Transfer transfer(*workers_);
  // stream order keeps these copies behind an upload that still reads a chunk
  auto queue = [&](size_t at, int slot) -> cudaError_t {
    const cudaError_t e = cudaMemcpyAsync(chunks_ + slot * kChunk, static_cast<const char*>(device) + at, std::min(step, bytes - at),
                                          cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaEventRecord(done_[slot], s) : e;
  };
  cudaError_t e = queue(0, 0);
  int slot = 0;
  for (size_t at = 0; at < bytes && e == cudaSuccess; at += step, slot ^= 1) {
    if (at + step < bytes) e = queue(at + step, slot ^ 1);
    if (e == cudaSuccess) e = cudaEventSynchronize(done_[slot]);
    if (e == cudaSuccess) workers_->copy(static_cast<char*>(host) + at, chunks_ + slot * kChunk, std::min(step, bytes - at));
  }
  if (e != cudaSuccess) cudaStreamSynchronize(s);  // nothing is left writing the chunks
  return e;
}

}  // namespace gdtp
