// Copies between ordinary (pageable) host memory and the device, and device
// scratch for one call, for the entry points that take host buffers.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

// Host -> device on `s`; on return the host buffer has been read.
cudaError_t staged_to_device(void *dst, const void *src, size_t bytes, cudaStream_t s);
// Device -> host after the work on `s`; on return the host buffer is written.
cudaError_t staged_to_host(void *dst, const void *src, size_t bytes, cudaStream_t s);

// Device memory for one call, ordered on its stream and taken from a pool of the
// library's own that keeps up to kScratchKept bytes per device between calls.
constexpr size_t kScratchKept = (size_t)256 << 20;
cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s);
