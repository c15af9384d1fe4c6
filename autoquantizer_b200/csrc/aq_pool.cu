// libaq.so: the device memory pool.
//
// Simulators, adjoints and the scratch of single calls take their memory
// from one pool per device.  The pool keeps up to POOL_KEEP bytes that were
// given back beyond what is in use (the release threshold counts both, so it
// follows: with 1.4 GB in use and a threshold of 1 GiB, each call's scratch was
// unmapped and mapped again; the driver's own default keeps none past the next
// synchronization, and mapping memory anew took 0.1 to 10 ms an allocation,
// more than the work of small calls), and gives back everything it can when
// an allocation fails or pool_release is called.  The driver's pool is safe for several threads and
// streams: memory freed on one stream goes to another only after the free.
#include "aq_pool.h"

#include <stdint.h>
#include <string.h>

#include <mutex>
#include <unordered_map>

namespace aq {

constexpr uint64_t POOL_KEEP = uint64_t(1) << 30;
constexpr int POOL_DEVICES = 64;

struct PoolBlock {
  cudaMemPool_t pool;
  size_t bytes;
  int device;
};

static std::mutex g_pool_mu;
static cudaMemPool_t g_pool[POOL_DEVICES];
static std::unordered_map<void*, PoolBlock> g_pool_live;
static std::unordered_map<cudaMemPool_t, uint64_t> g_pool_used;

// `by` more (or fewer) bytes in use in a pool; g_pool_mu held
static void pool_count(cudaMemPool_t pool, int64_t by) {
  uint64_t& used = g_pool_used[pool];
  used += by;
  uint64_t keep = used + POOL_KEEP;
  cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
}

static cudaError_t pool_of(int dev, cudaMemPool_t* out) {
  if (dev < 0 || dev >= POOL_DEVICES) return cudaDeviceGetDefaultMemPool(out, dev);
  std::lock_guard<std::mutex> g(g_pool_mu);
  if (!g_pool[dev]) {
    cudaMemPoolProps props;
    memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t p;
    const cudaError_t e = cudaMemPoolCreate(&p, &props);
    if (e != cudaSuccess) return e;
    g_pool[dev] = p;
  }
  *out = g_pool[dev];
  return cudaSuccess;
}

cudaError_t pool_alloc(void** p, size_t bytes, cudaStream_t st) {
  *p = nullptr;
  int dev = 0;
  cudaMemPool_t pool;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = pool_of(dev, &pool);
  if (e != cudaSuccess) return e;
  e = cudaMallocFromPoolAsync(p, bytes ? bytes : 1, pool, st);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    cudaDeviceSynchronize();
    cudaMemPoolTrimTo(pool, 0);
    e = cudaMallocFromPoolAsync(p, bytes ? bytes : 1, pool, st);
    if (e != cudaSuccess) cudaGetLastError();
  }
  if (e == cudaSuccess) {
    std::lock_guard<std::mutex> g(g_pool_mu);
    g_pool_live[*p] = PoolBlock{pool, bytes, dev};
    pool_count(pool, (int64_t)bytes);
  }
  return e;
}

cudaError_t pool_free(void* p, cudaStream_t st) {
  if (!p) return cudaSuccess;
  PoolBlock b;
  {
    std::lock_guard<std::mutex> g(g_pool_mu);
    const auto it = g_pool_live.find(p);
    if (it == g_pool_live.end()) return cudaErrorInvalidValue;
    b = it->second;
    // before the free, after which another thread may be given p
    pool_count(b.pool, -(int64_t)b.bytes);
    g_pool_live.erase(it);
  }
  const OnDevice on(b.device);
  const cudaError_t e = cudaFreeAsync(p, st);
  if (e != cudaSuccess) {  // still in use
    cudaGetLastError();
    std::lock_guard<std::mutex> g(g_pool_mu);
    g_pool_live[p] = b;
    pool_count(b.pool, (int64_t)b.bytes);
  }
  return e;
}

cudaError_t pool_release() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return e;
  cudaMemPool_t pool = nullptr;
  {
    std::lock_guard<std::mutex> g(g_pool_mu);
    if (dev >= 0 && dev < POOL_DEVICES) pool = g_pool[dev];
  }
  return pool ? cudaMemPoolTrimTo(pool, 0) : cudaSuccess;
}

}  // namespace aq
