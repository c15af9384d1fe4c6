// Device memory of libaq.so: one pool per device, in stream order.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace aq {

// Memory of the current device: there for work on st, and for other streams
// once they wait for st.
cudaError_t pool_alloc(void** p, size_t bytes, cudaStream_t st);

// Given back in the order of st, a stream of the memory's own device (null:
// that device's legacy stream, whichever device is current).  pool_free(null)
// does nothing.  After an error the memory still counts as in use.
cudaError_t pool_free(void* p, cudaStream_t st);

// What the current device's pool keeps beyond what is in use goes back to the
// device.  Waits for the device.
cudaError_t pool_release();

// A device made current for a scope.
class OnDevice {
  int was = -1;

 public:
  explicit OnDevice(int dev) {
    int now = -1;
    if (cudaGetDevice(&now) == cudaSuccess && now != dev && cudaSetDevice(dev) == cudaSuccess) was = now;
  }
  ~OnDevice() {
    if (was >= 0) cudaSetDevice(was);
  }
  OnDevice(const OnDevice&) = delete;
};

}  // namespace aq
