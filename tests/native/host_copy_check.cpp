// Staged host copies (csrc/host_copy.cpp) over a CUDA runtime on host memory
// (fake_cuda_copies.h): copies that overlap in time.
//
//   host_copy_check threads   round trips of several threads through one object
//   host_copy_check streams   a copy on one stream while another's still reads its chunks
//   host_copy_check first     when chunks are made, and how large
//   host_copy_check idle      copies that wait for the work queued before them
//   host_copy_check shared    one object per device, whose memory goes with its last owner
#include <cstdio>
#include <ctime>
#include <random>
#include <string>
#include <thread>
#include <vector>

#include "fake_cuda_copies.h"
#include "host_copy.h"

namespace {

using Data = std::vector<unsigned char>;

Data random_data(size_t n, unsigned seed) {
  Data v(n);
  std::mt19937 rng(seed);
  for (size_t i = 0; i + 4 <= n; i += 4) {
    const unsigned r = rng();
    std::memcpy(&v[i], &r, 4);
  }
  return v;
}

// every thread uploads its own vector and reads it back, streams shared or not
int threads(int nThreads, bool oneStream) {
  gdtp::HostCopy copier(0);  // staged from the first copy on
  fake::Stream shared;
  std::atomic<int> wrong{0};
  std::vector<std::thread> ts;
  for (int t = 0; t < nThreads; t++)
    ts.emplace_back([&, t] {
      fake::Stream own;
      fake::Stream& s = oneStream ? shared : own;
      for (int r = 0; r < 12; r++) {
        const size_t n = (size_t(3) << 20) + size_t(t) * 700001 + size_t(r) * 4097;
        const Data in = random_data(n, unsigned(100 * t + r));
        Data device(n), out(n);
        if (copier.upload(device.data(), in.data(), n, s.handle()) != cudaSuccess ||
            copier.download(out.data(), device.data(), n, s.handle()) != cudaSuccess || out != in)
          wrong++;
        cudaStreamSynchronize(s.handle());
      }
    });
  for (std::thread& t : ts) t.join();
  if (wrong) std::printf("%d of %d round trips differ (%d threads, %s)\n", int(wrong), 12 * nThreads, nThreads,
                         oneStream ? "one stream" : "a stream each");
  return wrong;
}

// stream a still reads the chunks of an upload when a copy on stream b begins
int streams() {
  gdtp::HostCopy copier(0);  // staged from the first copy on
  fake::Stream a, b;
  int wrong = 0;
  const size_t n = size_t(4) << 20;
  for (int r = 0; r < 6; r++) {
    const Data in = random_data(n, unsigned(r)), other = random_data(n, unsigned(50 + r));
    Data dev(n), dev2 = other, out(n), out2(n), up(n);
    a.delayUs = 30000;
    if (copier.upload(dev.data(), in.data(), n, a.handle()) != cudaSuccess) wrong++;
    if (copier.download(out2.data(), dev2.data(), n, b.handle()) != cudaSuccess || out2 != other) wrong++;
    if (copier.upload(up.data(), other.data(), n, b.handle()) != cudaSuccess) wrong++;
    cudaStreamSynchronize(b.handle());
    if (up != other) wrong++;
    cudaStreamSynchronize(a.handle());
    if (dev != in) wrong++;
    if (copier.download(out.data(), dev.data(), n, a.handle()) != cudaSuccess || out != in) wrong++;
  }
  if (wrong) std::printf("%d copies differ between two streams\n", wrong);
  return wrong;
}

// few copies make no chunks; many, or one large enough, make them of the size they need
int first() {
  int wrong = 0;
  fake::Stream s;
  auto trips = [&](gdtp::HostCopy& copier, size_t n, int count) {
    const Data in = random_data(n, unsigned(n));
    Data device(n), out(n);
    for (int r = 0; r < count; r++) {
      copier.upload(device.data(), in.data(), n, s.handle());
      copier.download(out.data(), device.data(), n, s.handle());
      if (out != in) wrong++;
    }
  };
  auto expect = [&](const char* what, long long low, long long high) {
    if (fake::pinnedBytes >= low && fake::pinnedBytes <= high) return;
    std::printf("%s: %lld pinned bytes\n", what, (long long)fake::pinnedBytes);
    wrong++;
  };
  const long long MB = 1 << 20;
  {
    gdtp::HostCopy copier;
    trips(copier, 5 * MB, 6);
    expect("60 MB moved", 0, 0);
    trips(copier, 5 * MB, 1);
    expect("70 MB moved", 2 * MB, 4 * MB);
    trips(copier, 21 * MB, 1);
    expect("one larger vector", 2 * MB, 4 * MB);
    trips(copier, 21 * MB, 1);
    expect("larger vectors", 12 * MB, 12 * MB);
    trips(copier, 50 * MB, 2);
    expect("the largest", 16 * MB, 16 * MB);
    trips(copier, 5 * MB, 2);
    expect("as before", 16 * MB, 16 * MB);
  }
  {
    gdtp::HostCopy copier;
    trips(copier, 70 * MB, 1);
    expect("one vector of 70 MB", 16 * MB, 16 * MB);
  }
  expect("all gone", 0, 0);
  return wrong;
}

// copies behind 0.3 s of queued work: the host threads sleep meanwhile
int idle() {
  gdtp::HostCopy copier(0);
  fake::Stream s;
  const size_t n = size_t(12) << 20;
  const Data in = random_data(n, 3);
  Data device(n), out(n);
  copier.upload(device.data(), in.data(), n, s.handle());
  cudaStreamSynchronize(s.handle());
  int wrong = 0;
  auto cpu = [&](const char* what, auto&& copy) {
    s.sleep(300000);
    const std::clock_t c0 = std::clock();
    copy();
    cudaStreamSynchronize(s.handle());
    const double t = double(std::clock() - c0) / CLOCKS_PER_SEC;
    if (t > 0.15) {
      std::printf("%s: %.2f s of processor time\n", what, t);
      wrong++;
    }
  };
  cpu("download", [&] { copier.download(out.data(), device.data(), n, s.handle()); });
  if (out != in) wrong++;
  std::fill(device.begin(), device.end(), 0);
  cpu("upload", [&] { copier.upload(device.data(), in.data(), n, s.handle()); });
  if (device != in) wrong++;
  return wrong;
}

// eight owners on a device, one after another and nested: one set's memory, all given back
int shared() {
  int wrong = 0;
  const size_t n = size_t(5) << 20;
  const Data in = random_data(n, 1);
  {
    fake::Stream s;
    std::vector<std::shared_ptr<gdtp::HostCopy>> owners{gdtp::HostCopy::of_device(0)};
    Data large(size_t(64) << 20), device(large.size());
    owners[0]->upload(device.data(), large.data(), large.size(), s.handle());  // staged from here on
    cudaStreamSynchronize(s.handle());
    for (int i = 0; i < 8; i++) {
      owners.push_back(gdtp::HostCopy::of_device(0));
      Data device(n), out(n);
      owners.back()->upload(device.data(), in.data(), n, s.handle());
      owners.back()->download(out.data(), device.data(), n, s.handle());
      if (out != in) wrong++;
    }
    if (gdtp::HostCopy::of_device(1) == owners[0]) wrong++;
    const long long one = fake::pinnedBytes;
    if (one <= 0 || one > (16 << 20) || fake::pinnedPeak != one) {
      std::printf("pinned memory of 8 owners: %lld bytes\n", one);
      wrong++;
    }
    owners.erase(owners.begin() + 1, owners.end());
    if (fake::pinnedBytes != one) wrong++;
  }
  if (fake::pinnedBytes != 0 || fake::events != 0) {
    std::printf("%lld pinned bytes and %d events left\n", (long long)fake::pinnedBytes, int(fake::events));
    wrong++;
  }
  return wrong;
}

}  // namespace

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  int wrong = -1;
  if (what == "threads") {
    wrong = 0;
    for (int n : {2, 3, 7})
      for (bool oneStream : {false, true}) wrong += threads(n, oneStream);
  } else if (what == "streams") {
    wrong = streams();
  } else if (what == "idle") {
    wrong = idle();
  } else if (what == "first") {
    wrong = first();
  } else if (what == "shared") {
    wrong = shared();
  }
  if (wrong == 0) std::printf("ok\n");
  return wrong == 0 ? 0 : 1;
}
