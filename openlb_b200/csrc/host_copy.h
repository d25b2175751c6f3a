// Device-to-host copies into ordinary (pageable) memory.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace olb_b200 {

// A handle that copies results out holds one of these for its lifetime.  All
// holders of a process share one set of staging buffers and copy threads, made
// once they have copied a good deal and given back with the last holder.
class HostCopyHold {
public:
  HostCopyHold();
  ~HostCopyHold();
  HostCopyHold(const HostCopyHold&) = delete;
  HostCopyHold& operator=(const HostCopyHold&) = delete;
};

// Copies `bytes` from device memory to `dst` after the work on `stream`.  `dst`
// is complete once the stream is synchronised; a copy into pageable memory is
// complete when the call returns.
cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, int device, cudaStream_t stream);

} // namespace olb_b200
