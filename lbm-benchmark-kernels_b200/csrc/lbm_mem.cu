// lbm_mem.cu -- the device memory pools and page-locked host memory of
// lbm_mem.cuh.
#include "lbm_mem.cuh"

#include <sys/mman.h>

#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <unordered_set>

#include "../../include/lbm_b200.h"

namespace {

constexpr int kMaxDevices = 64;
struct Pool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;  // orders the pool's allocations and frees
  bool none = false;              // the device has no pools
};
struct HostBlock {
  void* map;  // nullptr: cudaMallocHost
  size_t mapBytes;
};

std::mutex g_lock;
Pool g_pools[kMaxDevices];
std::unordered_set<void*> g_direct;  // device blocks from cudaMalloc
std::unordered_map<void*, HostBlock> g_host;

// The pool of device `dev`, made on first use; null where it has none.
Pool* pool_of(int dev) {
  if (dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> hold(g_lock);
  Pool& p = g_pools[dev];
  if (p.none) return nullptr;
  if (!p.pool) {
    int has = 0;
    cudaDeviceGetAttribute(&has, cudaDevAttrMemoryPoolsSupported, dev);
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long keep = lbm::kPoolKeep;
    if (!has || cudaMemPoolCreate(&p.pool, &props) != cudaSuccess) {
      p.none = true;
    } else if (cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
               cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) != cudaSuccess) {
      cudaMemPoolDestroy(p.pool);
      p.pool = nullptr;
      p.none = true;
    }
    if (p.none) {
      cudaGetLastError();
      return nullptr;
    }
  }
  return &p;
}

}  // namespace

namespace lbm {

cudaError_t dev_alloc(void** p, size_t bytes) {
  *p = nullptr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  Pool* pool = bytes > 0 && bytes <= kPoolBlock ? pool_of(dev) : nullptr;
  if (pool) {
    e = cudaMallocFromPoolAsync(p, bytes, pool->pool, pool->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(pool->stream);
    if (e == cudaSuccess) return e;
    // out of memory with freed blocks kept: give those back and try without
    *p = nullptr;
    cudaGetLastError();
    cudaMemPoolTrimTo(pool->pool, 0);
  }
  e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation && !pool && (pool = pool_of(dev))) {
    cudaGetLastError();
    cudaMemPoolTrimTo(pool->pool, 0);
    e = cudaMalloc(p, bytes);
  }
  if (e == cudaSuccess && *p) {
    std::lock_guard<std::mutex> hold(g_lock);
    g_direct.insert(*p);
  }
  return e;
}

void dev_free(void* p) {
  if (!p) return;
  bool direct;
  {
    std::lock_guard<std::mutex> hold(g_lock);
    direct = g_direct.erase(p) != 0;
  }
  if (direct) {
    cudaFree(p);
    return;
  }
  cudaPointerAttributes at;
  Pool* pool = cudaPointerGetAttributes(&at, p) == cudaSuccess ? pool_of(at.device) : nullptr;
  if (pool) cudaFreeAsync(p, pool->stream);
}

cudaError_t host_alloc(void** p, size_t bytes) {
  constexpr size_t kHuge = 2ull << 20;
  const size_t n = (bytes + kHuge - 1) / kHuge * kHuge + (bytes == 0 ? kHuge : 0);
  void* map = mmap(nullptr, n + kHuge, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (map != MAP_FAILED) {
    void* a = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(map) + kHuge - 1) / kHuge * kHuge);
    madvise(a, n, MADV_HUGEPAGE);  // a hint: plain pages work too
    if (cudaHostRegister(a, n, cudaHostRegisterPortable) == cudaSuccess) {
      std::lock_guard<std::mutex> hold(g_lock);
      g_host[a] = HostBlock{map, n + kHuge};
      *p = a;
      return cudaSuccess;
    }
    cudaGetLastError();
    munmap(map, n + kHuge);
  }
  const cudaError_t e = cudaMallocHost(p, bytes);
  if (e == cudaSuccess) {
    for (size_t k = 0; k < bytes; ++k) static_cast<char*>(*p)[k] = 0;
    std::lock_guard<std::mutex> hold(g_lock);
    g_host[*p] = HostBlock{nullptr, 0};
  }
  return e;
}

void host_free(void* p) {
  if (!p) return;
  HostBlock b{nullptr, 0};
  {
    std::lock_guard<std::mutex> hold(g_lock);
    auto it = g_host.find(p);
    if (it == g_host.end()) return;
    b = it->second;
    g_host.erase(it);
  }
  if (!b.map) {
    cudaFreeHost(p);
    return;
  }
  cudaHostUnregister(p);
  munmap(b.map, b.mapBytes);
}

}  // namespace lbm

extern "C" {

// Declared in include/lbm_b200.h.
int lbm_b200_release_memory(void) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  Pool* pool = pool_of(dev);
  if (!pool) return 0;
  e = cudaStreamSynchronize(pool->stream);
  if (e == cudaSuccess) e = cudaMemPoolTrimTo(pool->pool, 0);
  return (int)e;
}

}  // extern "C"
