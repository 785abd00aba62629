// Copies between the caller's host vectors and device buffers (host_copy.h).
#include "host_copy.h"

#include <sched.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace gdtp {

// memcpy by the caller and a few workers.  The workers sleep between transfers (an
// OpenMP team spins for some milliseconds after its work, which slowed the caller's own
// threads: 0.2 ms and more on the next host operation) and poll within one for up to
// kPoll after a chunk, since chunks follow one another in tens of microseconds; then
// they sleep until the next (a chunk may wait for all the work queued before it).
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
    if (asleep_ > 0) wake_.notify_all();
  }
  void copy(void* dst, const void* src, size_t bytes) {
    std::unique_lock<std::mutex> l(m_);
    dst_ = static_cast<char*>(dst);
    src_ = static_cast<const char*>(src);
    bytes_ = bytes;
    at_ = 0;
    turn_.fetch_add(1);
    if (asleep_ > 0) wake_.notify_all();
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
  static constexpr std::chrono::microseconds kPoll{500};
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
        const auto until = std::chrono::steady_clock::now() + kPoll;
        while (turn_.load() == turn && std::chrono::steady_clock::now() < until) std::this_thread::yield();
        l.lock();
        asleep_++;
        wake_.wait(l, [this, turn] { return turn_.load() != turn; });
        asleep_--;
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
  int busy_ = 0, asleep_ = 0;
  std::vector<std::thread> threads_;
};

// Two pinned chunks, the events after their last copies, and the threads
struct HostCopy::Set {
  unsigned char* chunks = nullptr;  // kSlots x size
  size_t size = 0;
  size_t small = 0;                 // moved in steps that the chunks' size limited
  cudaEvent_t done[kSlots] = {};
  cudaStream_t last = nullptr;      // stream of the last copy
  Workers workers;
  bool taken = true;
  // both chunks have been left
  bool idle() const {
    for (cudaEvent_t e : done)
      if (cudaEventQuery(e) != cudaSuccess) {
        if (cudaPeekAtLastError() == cudaErrorNotReady) cudaGetLastError();  // not an error of the caller's
        return false;
      }
    return true;
  }
  // (new) chunks of this size, once the old ones are left
  bool make(size_t bytes) {
    void* p = nullptr;
    if (cudaHostAlloc(&p, kSlots * bytes, cudaHostAllocDefault) != cudaSuccess) return false;
    for (cudaEvent_t& e : done) {
      if (e) cudaEventSynchronize(e);
      else if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        e = nullptr;
        cudaFreeHost(p);
        return false;
      }
    }
    if (chunks) cudaFreeHost(chunks);
    chunks = static_cast<unsigned char*>(p);
    size = bytes;
    small = 0;
    return true;
  }
  ~Set() {
    for (cudaEvent_t e : done)
      if (e) {
        cudaEventSynchronize(e);
        cudaEventDestroy(e);
      }
    if (chunks) cudaFreeHost(chunks);
  }
};

// a set in use by one copy; its workers are awake while this is in scope (they are woken
// while the first chunk is on its way: waking them when it is there costs a V-cycle of
// 640 x 480 RGB vectors 0.15 ms)
struct HostCopy::Transfer {
  Transfer(HostCopy& owner, Set* set) : owner(owner), set(set) { set->workers.begin(); }
  ~Transfer() {
    set->workers.end();
    owner.give(set);
  }
  HostCopy& owner;
  Set* set;
};

std::shared_ptr<HostCopy> HostCopy::of_device(int device) {
  static std::mutex m;
  static std::vector<std::weak_ptr<HostCopy>> objects;
  std::lock_guard<std::mutex> l(m);
  if (size_t(device) >= objects.size()) objects.resize(size_t(device) + 1);
  std::shared_ptr<HostCopy> c = objects[device].lock();
  if (!c) objects[device] = c = std::make_shared<HostCopy>();
  return c;
}

HostCopy::HostCopy(size_t payback) : payback_(payback) {}
HostCopy::~HostCopy() = default;

// A free set whose chunks are idle, or are left in the order of s: another stream's
// pending work is not waited for.  None: a new set, up to kMaxSets, once it is paid for.
HostCopy::Set* HostCopy::take(const void* host, size_t bytes, cudaStream_t s) {
  if (bytes < kStagedMin) return nullptr;
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (at.type != cudaMemoryTypeUnregistered) return nullptr;
  Set* set = nullptr;
  const size_t want = (piece(bytes) + kChunkMin - 1) / kChunkMin * kChunkMin;
  bool made = false;
  {
    std::lock_guard<std::mutex> l(m_);
    for (std::unique_ptr<Set>& q : sets_)
      if (!set && !q->taken && (q->last == s || q->idle())) set = q.get();
    if (!set) {
      plain_ += bytes;
      if (failed_ || sets_.size() >= kMaxSets || plain_ < payback_) return nullptr;
      plain_ = 0;
      made = true;
      sets_.push_back(std::make_unique<Set>());
      set = sets_.back().get();
    }
    set->taken = true;
    set->last = s;
    if (!made && set->size < want) set->small += bytes;
  }
  // (allocations go on beside other copies)
  if (!made) {
    if (set->size < want && set->small >= payback_ && !set->make(std::min(kChunkMax, std::max(want, 2 * set->size)))) {
      cudaGetLastError();  // none of that size: the chunks stay as they are
      set->small = 0;
    }
    return set;
  }
  if (set->make(want)) return set;
  cudaGetLastError();
  std::lock_guard<std::mutex> l(m_);
  failed_ = true;
  sets_.erase(std::find_if(sets_.begin(), sets_.end(), [set](const std::unique_ptr<Set>& q) { return q.get() == set; }));
  return nullptr;
}

void HostCopy::give(Set* set) {
  std::lock_guard<std::mutex> l(m_);
  set->taken = false;
}

// a quarter of the vector, so that the two sides overlap, within a chunk's size
size_t HostCopy::piece(size_t bytes) { return std::min(kChunkMax, std::max(kChunkMin, bytes / 4)); }

cudaError_t HostCopy::upload(void* device, const void* host, size_t bytes, cudaStream_t s) {
  Set* set = take(host, bytes, s);
  if (!set) return cudaMemcpyAsync(device, host, bytes, cudaMemcpyHostToDevice, s);
  const size_t step = std::min(set->size, piece(bytes));
  Transfer transfer(*this, set);
  int slot = 0;
  for (size_t at = 0; at < bytes; at += step, slot ^= 1) {
    const size_t len = std::min(step, bytes - at);
    unsigned char* chunk = set->chunks + slot * set->size;
    // the chunk's last copy (of this call or an earlier one) has left it
    cudaError_t e = cudaEventSynchronize(set->done[slot]);
    if (e == cudaSuccess) {
      set->workers.copy(chunk, static_cast<const char*>(host) + at, len);
      e = cudaMemcpyAsync(static_cast<char*>(device) + at, chunk, len, cudaMemcpyHostToDevice, s);
      if (e == cudaSuccess) e = cudaEventRecord(set->done[slot], s);
    }
    if (e != cudaSuccess) {
      cudaStreamSynchronize(s);  // nothing is left reading the chunks
      return e;
    }
  }
  return cudaSuccess;
}

cudaError_t HostCopy::download(void* host, const void* device, size_t bytes, cudaStream_t s) {
  Set* set = take(host, bytes, s);
  if (!set) {
    const cudaError_t e = cudaMemcpyAsync(host, device, bytes, cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
  }
  const size_t step = std::min(set->size, piece(bytes));
  Transfer transfer(*this, set);
  // after the chunk's last copy, also one of another stream
  auto queue = [&](size_t at, int slot) -> cudaError_t {
    cudaError_t e = cudaStreamWaitEvent(s, set->done[slot], 0);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(set->chunks + slot * set->size, static_cast<const char*>(device) + at, std::min(step, bytes - at),
                          cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaEventRecord(set->done[slot], s) : e;
  };
  cudaError_t e = queue(0, 0);
  int slot = 0;
  for (size_t at = 0; at < bytes && e == cudaSuccess; at += step, slot ^= 1) {
    if (at + step < bytes) e = queue(at + step, slot ^ 1);
    if (e == cudaSuccess) e = cudaEventSynchronize(set->done[slot]);
    if (e == cudaSuccess) set->workers.copy(static_cast<char*>(host) + at, set->chunks + slot * set->size, std::min(step, bytes - at));
  }
  if (e != cudaSuccess) cudaStreamSynchronize(s);  // nothing is left writing the chunks
  return e;
}

}  // namespace gdtp
