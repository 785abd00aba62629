// The CUDA runtime calls of csrc/host_copy.cpp on host memory: a stream is a thread
// that runs its copies and waits in order, each after a settable delay, so that copies
// are as asynchronous as a device's.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>

namespace fake {

// one record of an event; waits are for the record that is the latest when they are made
struct Mark {
  std::mutex m;
  std::condition_variable cv;
  bool done = false;
  void set() {
    std::lock_guard<std::mutex> l(m);
    done = true;
    cv.notify_all();
  }
  void wait() {
    std::unique_lock<std::mutex> l(m);
    cv.wait(l, [this] { return done; });
  }
};
struct Event {
  std::mutex m;
  std::shared_ptr<Mark> last;
  std::shared_ptr<Mark> latest() {
    std::lock_guard<std::mutex> l(m);
    return last;
  }
};

struct Stream {
  std::mutex m;
  std::condition_variable cv;
  std::deque<std::function<void()>> work;
  bool busy = false, stop = false;
  std::atomic<int> delayUs{0};
  std::thread t{[this] { run(); }};
  void run() {
    std::unique_lock<std::mutex> l(m);
    for (;;) {
      cv.wait(l, [this] { return stop || !work.empty(); });
      if (work.empty()) return;
      auto f = std::move(work.front());
      work.pop_front();
      busy = true;
      l.unlock();
      f();
      l.lock();
      busy = false;
      cv.notify_all();
    }
  }
  void push(std::function<void()> f) {
    std::lock_guard<std::mutex> l(m);
    work.push_back(std::move(f));
    cv.notify_all();
  }
  void drain() {
    std::unique_lock<std::mutex> l(m);
    cv.wait(l, [this] { return work.empty() && !busy; });
  }
  void sleep(int us) {
    push([us] { std::this_thread::sleep_for(std::chrono::microseconds(us)); });
  }
  ~Stream() {
    drain();
    {
      std::lock_guard<std::mutex> l(m);
      stop = true;
    }
    cv.notify_all();
    t.join();
  }
  cudaStream_t handle() { return reinterpret_cast<cudaStream_t>(this); }
};

inline std::atomic<long long> pinnedBytes{0}, pinnedPeak{0}, pinnedCalls{0}, copies{0};
inline std::atomic<int> events{0};

}  // namespace fake

extern "C" {
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  *a = cudaPointerAttributes();
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  size_t* q = static_cast<size_t*>(std::malloc(n + 64));
  q[0] = n;
  *p = reinterpret_cast<char*>(q) + 64;
  fake::pinnedCalls++;
  const long long now = fake::pinnedBytes += (long long)n;
  if (now > fake::pinnedPeak) fake::pinnedPeak = now;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  size_t* q = reinterpret_cast<size_t*>(static_cast<char*>(p) - 64);
  fake::pinnedBytes -= (long long)q[0];
  std::free(q);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  fake::events++;
  *e = reinterpret_cast<cudaEvent_t>(new fake::Event());
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  fake::events--;
  delete reinterpret_cast<fake::Event*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  fake::Event* ev = reinterpret_cast<fake::Event*>(e);
  auto mark = std::make_shared<fake::Mark>();
  {
    std::lock_guard<std::mutex> l(ev->m);
    ev->last = mark;
  }
  reinterpret_cast<fake::Stream*>(s)->push([mark] { mark->set(); });
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  if (auto mark = reinterpret_cast<fake::Event*>(e)->latest()) mark->wait();
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  auto mark = reinterpret_cast<fake::Event*>(e)->latest();
  if (!mark) return cudaSuccess;
  std::lock_guard<std::mutex> l(mark->m);
  return mark->done ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  if (auto mark = reinterpret_cast<fake::Event*>(e)->latest()) reinterpret_cast<fake::Stream*>(s)->push([mark] { mark->wait(); });
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  reinterpret_cast<fake::Stream*>(s)->drain();
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
  fake::Stream* st = reinterpret_cast<fake::Stream*>(s);
  fake::copies++;
  st->push([d, src, n, st] {
    if (const int us = st->delayUs) std::this_thread::sleep_for(std::chrono::microseconds(us));
    std::memcpy(d, src, n);
  });
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
}
