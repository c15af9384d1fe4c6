// Shared host/device helpers of libaq.so.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/aq.h"
#include "aq_pool.h"

#define AQ_CUDA_TRY(expr)                        \
  do {                                           \
    cudaError_t aq_err_ = (expr);                \
    if (aq_err_ != cudaSuccess) {                \
      aq::set_last_cuda_error(aq_err_, #expr);   \
      return AQ_E_CUDA;                          \
    }                                            \
  } while (0)

namespace aq {

void set_last_cuda_error(cudaError_t e, const char* what);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

inline int num_sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// Launch a kernel that waits for the one before it in the stream by itself
// (kernel_begin, ahead of its first global access), so that its launch
// overlaps that one's end.
struct PdlConfig {
  cudaLaunchAttribute at;
  cudaLaunchConfig_t c;
  PdlConfig(unsigned grid, unsigned block, size_t smem, cudaStream_t st) : c() {
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
  }
  PdlConfig(const PdlConfig&) = delete;
};

template <class... P, class... A>
inline cudaError_t launch_pdl(void (*f)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
  const PdlConfig c(grid, block, smem, st);
  return cudaLaunchKernelEx(&c.c, f, P(args)...);
}

inline unsigned grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 0x7fffffffLL) b = 0x7fffffffLL;
  return (unsigned)b;
}

}  // namespace aq
