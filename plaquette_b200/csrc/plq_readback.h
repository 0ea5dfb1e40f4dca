// plq_readback.h -- large device-to-host copies into pageable memory.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

// Copies `bytes` from the device after the work queued on `stream`.  Copies of
// kReadbackStaged and more into pageable memory go through pinned buffers on
// several host threads and are complete on return; any other is queued on the
// stream as cudaMemcpyAsync queues it.
constexpr size_t kReadbackStaged = size_t(32) << 20;
cudaError_t plq_readback(void *dst, const void *src, size_t bytes, int device, cudaStream_t stream);
// Gives back the pinned buffers that earlier copies from `device` left for later ones.
void plq_readback_release(int device);
