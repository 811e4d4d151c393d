// Staged copies between the device and pageable host memory (cf1_hostio.cuh).
#include <algorithm>
#include <cstring>
#include <system_error>

#include "cf1_hostio.cuh"

namespace cf1 {

bool pageable(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

HostCopier::HostCopier(size_t total_bytes) {
  // a thread per 4 MB up to eight: one copies ~10 GB/s, PCIe takes ~55, and
  // starting one costs ~100 us (a thread per 512 KB made 5 Mbp slower)
  const size_t hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t want = std::min({(size_t)8, hw, total_bytes >> 22});
  try {
    for (size_t i = 1; i < want; i++)
      threads_.emplace_back([this, i] {
        for (uint64_t seen = 0;;) {
          while (epoch_.load(std::memory_order_acquire) == seen) std::this_thread::yield();
          seen++;
          if (stop_.load(std::memory_order_relaxed)) return;
          part(i);
          left_.fetch_sub(1, std::memory_order_release);
        }
      });
  } catch (const std::system_error &) {  // no more threads to be had
  }
}

HostCopier::~HostCopier() {
  stop_.store(true, std::memory_order_relaxed);
  epoch_.fetch_add(1, std::memory_order_release);
  for (auto &t : threads_) t.join();
}

void HostCopier::part(size_t i) const {
  const size_t k = threads_.size() + 1, step = ((n_ + k - 1) / k + 63) & ~(size_t)63;
  const size_t b = std::min(n_, i * step), e = std::min(n_, b + step);
  if (e > b) std::memcpy(dst_ + b, src_ + b, e - b);
}

void HostCopier::copy(void *dst, const void *src, size_t n) {
  dst_ = static_cast<char *>(dst);
  src_ = static_cast<const char *>(src);
  n_ = n;
  if (threads_.empty() || n < (64u << 10)) {
    std::memcpy(dst, src, n);
    return;
  }
  left_.store(threads_.size(), std::memory_order_relaxed);
  epoch_.fetch_add(1, std::memory_order_release);
  part(0);
  while (left_.load(std::memory_order_acquire)) std::this_thread::yield();
}

void copy_out(cf1gpu_ctx *c, void *dst, const void *dev, size_t bytes) {
  cudaStream_t s = c->stream;
  if (bytes < IO_STAGE_MIN || !pageable(dst)) {
    if (bytes) CF1_CUDA(cudaMemcpyAsync(dst, dev, bytes, cudaMemcpyDeviceToHost, s));
    CF1_CUDA(cudaStreamSynchronize(s));
    return;
  }
  c->stage_out.reserve(2 * std::min(bytes, IO_CHUNK), 0);
  HostCopier cp(bytes);
  const size_t half = c->stage_out.cap / 2, step = std::min(half, IO_CHUNK);
  const size_t n = (bytes + step - 1) / step;
  auto drain = [&](size_t i) {  // chunk i is on its way: wait for it and hand it over
    CF1_CUDA(cudaEventSynchronize(c->io_ev[2 + (i & 1)]));
    cp.copy(static_cast<char *>(dst) + i * step, c->stage_out.p + (i & 1) * half, std::min(step, bytes - i * step));
  };
  for (size_t i = 0; i < n; i++) {
    CF1_CUDA(cudaMemcpyAsync(c->stage_out.p + (i & 1) * half, static_cast<const char *>(dev) + i * step,
                             std::min(step, bytes - i * step), cudaMemcpyDeviceToHost, s));
    CF1_CUDA(cudaEventRecord(c->io_ev[2 + (i & 1)], s));
    if (i) drain(i - 1);
  }
  drain(n - 1);
}

}  // namespace cf1
