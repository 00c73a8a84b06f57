// Device memory into ordinary (pageable) host memory through two pinned chunks.
//
// A pageable copy runs at 3-4 GB/s: the driver stages it through its own
// buffer with one thread.  Here the DMA fills one pinned chunk while up to
// eight threads move the other one's bytes into place (and take the page
// faults of a fresh destination).  Measured: 23 MB in two buffers 7 -> 2.7 ms,
// 188 MB in two 52 -> 19 ms.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace gtob {

constexpr size_t kPinChunk = size_t(4) << 20;
// pin: 2 * kPinChunk bytes of pinned memory, or null (a plain copy).  Ordered after the work already
// on stream s; returns once the copy is complete.
void copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t s, unsigned char* pin);

}  // namespace gtob
