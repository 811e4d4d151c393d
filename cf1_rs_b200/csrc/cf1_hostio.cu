// Staged copies between the device and pageable host memory (cf1_hostio.cuh).
#include <algorithm>

#include "cf1_hostio.cuh"

namespace cf1 {

cudaMemoryType memory_type(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();  // not a pointer CUDA knows
    return cudaMemoryTypeUnregistered;
  }
  return a.type;
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
