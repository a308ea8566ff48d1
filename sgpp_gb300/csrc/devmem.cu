#include "devmem.h"

#include <cstdint>
#include <mutex>
#include <vector>

namespace sgmev {

namespace {
std::mutex g_mu;
std::vector<cudaMemPool_t> g_pools;  // per device: the library's own pool (nullptr: not made yet)
std::vector<void*> g_pinned;         // recycled pinned blocks
constexpr size_t kPinnedBytes = 64;
constexpr size_t kKeptStreams = 32, kKeptBuffers = 16;
std::vector<double*> g_buffers;  // idle pinned buffers
std::vector<std::vector<cudaStream_t>> g_streams;  // per device: idle streams of past operators

// The library allocates from a pool of its own, not from the device's default pool: its release
// threshold is raised so that freed blocks stay for the next operator, and raising it on the
// default pool would stop every other cudaMallocAsync user of the process from returning memory.
cudaMemPool_t library_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(g_mu);
  if (static_cast<int>(g_pools.size()) <= dev) g_pools.resize(dev + 1, nullptr);
  if (g_pools[dev]) return g_pools[dev];
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  uint64_t keep = UINT64_MAX;  // keep freed blocks for the next operator
  if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess)
    (void)cudaGetLastError();
  g_pools[dev] = pool;
  return pool;
}
}  // namespace

cudaError_t dev_malloc(void** p, size_t bytes, cudaStream_t s) {
  *p = nullptr;
  cudaMemPool_t pool = library_pool();
  if (!pool) return cudaErrorMemoryAllocation;
  const size_t n = bytes == 0 ? 1 : bytes;
  cudaError_t e = cudaMallocFromPoolAsync(p, n, pool, s);
  if (e == cudaErrorMemoryAllocation) {
    // hand the pool's unused blocks back to the device and try once more
    (void)cudaGetLastError();
    cudaMemPoolTrimTo(pool, 0);
    e = cudaMallocFromPoolAsync(p, n, pool, s);
  }
  if (e != cudaSuccess) {
    *p = nullptr;
    (void)cudaGetLastError();
  }
  return e;
}

size_t dev_available() {
  size_t free_b = 0, total_b = 0;
  cudaMemPool_t pool = library_pool();
  uint64_t reserved = 0, used = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || !pool ||
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
    (void)cudaGetLastError();
  return free_b + static_cast<size_t>(reserved > used ? reserved - used : 0);
}

void dev_free(void* p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

cudaStream_t stream_acquire() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (dev < static_cast<int>(g_streams.size()) && !g_streams[dev].empty()) {
      cudaStream_t s = g_streams[dev].back();  // the one most recently in use
      g_streams[dev].pop_back();
      return s;
    }
  }
  cudaStream_t s = nullptr;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  return s;
}

void stream_release(cudaStream_t s) {
  if (!s) return;
  int dev = 0;
  if (cudaStreamGetDevice(s, &dev) == cudaSuccess) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (static_cast<int>(g_streams.size()) <= dev) g_streams.resize(dev + 1);
    if (g_streams[dev].size() < kKeptStreams) {
      g_streams[dev].push_back(s);
      return;
    }
  } else {
    (void)cudaGetLastError();
  }
  cudaStreamDestroy(s);
}

double* pinned_buffer() {
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_buffers.empty()) {
      double* p = g_buffers.back();
      g_buffers.pop_back();
      return p;
    }
  }
  double* p = nullptr;
  if (cudaMallocHost(&p, kPinnedBuffer) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  return p;
}

void pinned_buffer_release(double* p) {
  if (!p) return;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_buffers.size() < kKeptBuffers) {
      g_buffers.push_back(p);
      return;
    }
  }
  cudaFreeHost(p);
}

void* pinned_block() {
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_pinned.empty()) {
      void* p = g_pinned.back();
      g_pinned.pop_back();
      return p;
    }
  }
  void* p = nullptr;
  if (cudaMallocHost(&p, kPinnedBytes) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  return p;
}

void pinned_release(void* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_mu);
  g_pinned.push_back(p);
}

}  // namespace sgmev
