// Host threads for one call's copies (they end with it).  Plain C++: the
// device side of the copies is in cf1_hostio.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <exception>
#include <functional>
#include <thread>
#include <vector>

namespace cf1 {

// f(0) .. f(n - 1), each on a thread of its own; those no thread (or no memory
// for one) can be had for run on the calling one.  f does not throw.
template <class F>
void on_threads(unsigned n, F &&f) {
  std::vector<std::thread> threads;
  unsigned t = 1;
  try {
    threads.reserve(n);
    for (; t < n; t++) threads.emplace_back(std::ref(f), t);
  } catch (const std::exception &) {
  }
  if (n) f(0u);
  for (; t < n; t++) f(t);
  for (auto &x : threads) x.join();
}

// Copies split over several threads, the calling one among them; fewer are
// used when they cannot be had.  Between copies the others look for the next
// one, giving way to whoever else wants their core: a call waits ~75 us for the
// DMA of a chunk, and threads that slept after 100 us made queries of 2 to 4 M
// k-mers 1.1 to 1.6 times as long.
class HostCopier {
 public:
  explicit HostCopier(size_t total_bytes) {
    // a thread per 4 MB up to eight: one copies ~10 GB/s, PCIe takes ~55, and
    // starting one costs ~100 us (a thread per 512 KB made 5 Mbp slower)
    const size_t hw = std::max(1u, std::thread::hardware_concurrency());
    const size_t want = std::min({(size_t)8, hw, total_bytes >> 22});
    try {
      threads_.reserve(want);
      for (size_t i = 1; i < want; i++) threads_.emplace_back([this, i] { serve(i); });
    } catch (const std::exception &) {
    }
  }
  ~HostCopier() {
    stop_.store(true, std::memory_order_relaxed);
    next();
    for (auto &t : threads_) t.join();
  }
  HostCopier(const HostCopier &) = delete;
  HostCopier &operator=(const HostCopier &) = delete;

  void copy(void *dst, const void *src, size_t n) {
    if (threads_.empty() || n < (64u << 10)) {
      std::memcpy(dst, src, n);
      return;
    }
    dst_ = static_cast<char *>(dst);
    src_ = static_cast<const char *>(src);
    n_ = n;
    left_.store(threads_.size(), std::memory_order_relaxed);
    next();
    part(0);
    while (left_.load(std::memory_order_acquire)) std::this_thread::yield();
  }

 private:
  void next() { epoch_.fetch_add(1, std::memory_order_release); }
  void serve(size_t i) {
    for (uint64_t seen = 0;;) {
      while (epoch_.load(std::memory_order_acquire) == seen) std::this_thread::yield();
      seen++;
      if (stop_.load(std::memory_order_relaxed)) return;
      part(i);
      left_.fetch_sub(1, std::memory_order_release);
    }
  }
  void part(size_t i) const {
    const size_t k = threads_.size() + 1, step = ((n_ + k - 1) / k + 63) & ~(size_t)63;
    const size_t b = std::min(n_, i * step), e = std::min(n_, b + step);
    if (e > b) std::memcpy(dst_ + b, src_ + b, e - b);
  }

  std::vector<std::thread> threads_;
  std::atomic<uint64_t> epoch_{0};
  std::atomic<size_t> left_{0};
  std::atomic<bool> stop_{false};
  char *dst_ = nullptr;
  const char *src_ = nullptr;
  size_t n_ = 0;
};

}  // namespace cf1
