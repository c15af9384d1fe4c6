"""The device memory pool (csrc/aq_pool.cu) against a stand-in for the CUDA
runtime, on the CPU: memory is freed on the device it came from, a free that
fails is not counted as given back, an allocation that fails is retried after
the pool is trimmed, and threads share the pool."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "autoquantizer_b200", "csrc")

FAKE = r"""
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>
#include <map>
#include <mutex>
typedef int cudaError_t;
typedef struct FakeStream* cudaStream_t;
typedef struct FakePool { int device; uint64_t threshold; uint64_t used; int trims; }* cudaMemPool_t;
enum { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
enum { cudaMemAllocationTypePinned = 1, cudaMemLocationTypeDevice = 1, cudaMemPoolAttrReleaseThreshold = 4 };
struct cudaMemPoolProps { int allocType; struct { int type, id; } location; };
struct Fake {
  std::mutex mu;
  int synchronized = 0, failing_allocs = 0, failing_frees = 0, wrong_device = 0, last_free_device = -1;
  std::map<void*, std::pair<cudaMemPool_t, size_t>> live;
  std::map<int, cudaMemPool_t> pools;
};
inline Fake& fake() { static Fake f; return f; }
inline int& current() { static thread_local int d = 0; return d; }
inline cudaError_t cudaGetDevice(int* d) { *d = current(); return 0; }
inline cudaError_t cudaSetDevice(int d) { current() = d; return 0; }
inline cudaError_t cudaGetLastError() { return 0; }
inline cudaError_t cudaDeviceSynchronize() { std::lock_guard<std::mutex> g(fake().mu); ++fake().synchronized; return 0; }
inline cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* q) {
  *p = new FakePool{q->location.id, 0, 0, 0};
  fake().pools[q->location.id] = *p;
  return 0;
}
inline cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t*, int) { return cudaErrorInvalidValue; }
inline cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, int, void* v) { p->threshold = *(uint64_t*)v; return 0; }
inline cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t) { std::lock_guard<std::mutex> g(fake().mu); ++p->trims; return 0; }
inline cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) {
  std::lock_guard<std::mutex> g(fake().mu);
  if (fake().failing_allocs > 0) { --fake().failing_allocs; return cudaErrorMemoryAllocation; }
  *p = malloc(n);
  fake().live[*p] = {pool, n};
  pool->used += n;
  return 0;
}
inline cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  std::lock_guard<std::mutex> g(fake().mu);
  if (fake().failing_frees > 0) { --fake().failing_frees; return cudaErrorInvalidValue; }
  auto it = fake().live.find(p);
  if (it == fake().live.end()) return cudaErrorInvalidValue;
  fake().last_free_device = current();
  if (it->second.first->device != current()) ++fake().wrong_device;
  it->second.first->used -= it->second.second;
  fake().live.erase(it);
  free(p);
  return 0;
}
"""

MAIN = r"""
#include "aq_pool.cu"
#include <stdio.h>
#include <thread>
#include <vector>
using namespace aq;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  const uint64_t keep = uint64_t(1) << 30;
  void *a = nullptr, *b = nullptr;
  // freed on its own device, whichever is current
  cudaSetDevice(1);
  CHECK(pool_alloc(&a, 1000, nullptr) == cudaSuccess);
  cudaSetDevice(0);
  CHECK(pool_alloc(&b, 500, nullptr) == cudaSuccess);
  CHECK(fake().pools[1]->threshold == 1000 + keep && fake().pools[0]->threshold == 500 + keep);
  CHECK(pool_free(a, nullptr) == cudaSuccess);
  CHECK(fake().last_free_device == 1 && fake().wrong_device == 0 && current() == 0);
  CHECK(fake().pools[1]->threshold == keep);
  // a free that fails: still in use, and can be freed later
  fake().failing_frees = 1;
  CHECK(pool_free(b, nullptr) != cudaSuccess);
  CHECK(fake().pools[0]->threshold == 500 + keep);
  CHECK(pool_free(b, nullptr) == cudaSuccess && fake().pools[0]->threshold == keep);
  CHECK(pool_free(nullptr, nullptr) == cudaSuccess && pool_free(&a, nullptr) != cudaSuccess);
  // an allocation that fails: the pool is trimmed, then once more
  fake().failing_allocs = 1;
  CHECK(pool_alloc(&a, 64, nullptr) == cudaSuccess && fake().synchronized == 1 && fake().pools[0]->trims == 1);
  CHECK(pool_free(a, nullptr) == cudaSuccess);
  fake().failing_allocs = 2;
  CHECK(pool_alloc(&a, 64, nullptr) == cudaErrorMemoryAllocation && a == nullptr);
  CHECK(fake().pools[0]->threshold == keep);
  // what is kept is given back on request, the current device's only
  cudaSetDevice(1);
  CHECK(pool_release() == cudaSuccess && fake().pools[1]->trims == 1 && fake().pools[0]->trims == 2);
  cudaSetDevice(7);
  CHECK(pool_release() == cudaSuccess);  // no pool there
  // threads
  std::vector<std::thread> ts;
  for (int t = 0; t < 4; ++t)
    ts.emplace_back([t] {
      cudaSetDevice(t & 1);
      void* p[8];
      for (int r = 0; r < 2000; ++r) {
        for (int k = 0; k < 8; ++k) pool_alloc(&p[k], 16 + 8 * k, nullptr);
        for (int k = 0; k < 8; ++k) pool_free(p[k], nullptr);
      }
    });
  for (auto& t : ts) t.join();
  CHECK(fake().live.empty() && fake().wrong_device == 0);
  CHECK(fake().pools[0]->threshold == keep && fake().pools[1]->threshold == keep);
  return 0;
}
"""


def test_pool_on_a_stand_in_runtime(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "pool")
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "main.cpp"),
                    "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stdout
