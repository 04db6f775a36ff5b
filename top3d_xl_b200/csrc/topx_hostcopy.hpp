// Copies between pageable host memory and the device for the host-buffer entry points of the C ABI.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace topx {

// Copies `bytes` between h (host) and d (device) on stream st.  On return the host memory is free to reuse (h2d:
// the copy is queued on st; d2h: the data is there).  A copy from or to page-locked memory goes directly, a short one
// through the runtime.  A long one from or to pageable memory is staged here: the runtime's own staging is
// one thread's memcpy (10 GB/s on a 16-core host, a fresh destination's page faults included), so
// kCopyThreads threads copy alternate chunks through page-locked slots while earlier chunks are on the bus.
void host_to_device(void* d, const void* h, size_t bytes, cudaStream_t st);
void device_to_host(void* h, const void* d, size_t bytes, cudaStream_t st);

// The page-locked slots (kCopyThreads x 2 x 1 MB) are shared by the process: made once long copies have moved 64 MB (those
// before go through the runtime), used by one copy at a time (another thread's copy meanwhile goes through the
// runtime), given back when the last holder is gone.
class HostCopyHold {
 public:
  HostCopyHold();
  ~HostCopyHold();
  HostCopyHold(const HostCopyHold&) = delete;
  HostCopyHold& operator=(const HostCopyHold&) = delete;
};

}  // namespace topx
