// Copies between the device and the caller's ordinary (pageable) memory.
//
// A cudaMemcpy from or to pageable memory passes through the driver's own
// staging on one thread (6-8 GB/s here, page faults of a fresh destination
// included).  Large ones go through two page-locked chunks of the context
// instead: the DMA of one chunk runs while several host threads copy the
// other.  Page-locked, managed or device pointers are copied directly.
#pragma once
#include "cf1_context.cuh"
#include "cf1_hostcopier.h"

namespace cf1 {

constexpr size_t IO_CHUNK = 4u << 20;  // bytes of a staging chunk
// Smaller copies are left to the driver: the chunks' page-locked memory costs
// a context's first one ~10 ms, which 3 MB of state words never win back.
constexpr size_t IO_STAGE_MIN = 16u << 20;

// What CUDA knows about the pointer: unregistered is ordinary host memory.
cudaMemoryType memory_type(const void *p);
inline bool pageable(const void *p) { return memory_type(p) == cudaMemoryTypeUnregistered; }

// bytes from the device to dst, in order after what is queued on the
// context's stream; returns when they are there.
void copy_out(cf1gpu_ctx *c, void *dst, const void *dev, size_t bytes);

}  // namespace cf1
