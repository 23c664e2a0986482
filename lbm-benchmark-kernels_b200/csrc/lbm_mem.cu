// lbm_mem.cu -- the device memory pools and page-locked host memory of
// lbm_mem.cuh.
#include "lbm_mem.cuh"

#include <sys/mman.h>

#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <vector>

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
struct Block {
  size_t bytes;
  int dev;
  bool keep;  // worth keeping for the next one when it is freed
};
std::unordered_map<void*, Block> g_direct;  // device blocks from cudaMalloc
struct Kept {
  void* p;
  size_t bytes;
  int dev;
};
std::vector<Kept> g_kept;  // freed blocks, oldest first
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

// Frees kept blocks of device `dev`, oldest first, until `room` bytes fit beside
// the others; keeps block p of that size, if there is one.
void make_room(int dev, size_t room, void* p) {
  std::vector<void*> out;
  {
    std::lock_guard<std::mutex> hold(g_lock);
    size_t sum = room;
    for (const Kept& k : g_kept) sum += k.dev == dev ? k.bytes : 0;
    for (size_t i = 0; i < g_kept.size() && sum > lbm::kBlockKeep;) {
      if (g_kept[i].dev != dev) {
        ++i;
        continue;
      }
      sum -= g_kept[i].bytes;
      out.push_back(g_kept[i].p);
      g_kept.erase(g_kept.begin() + i);
    }
    if (p) g_kept.push_back(Kept{p, room, dev});
  }
  for (void* q : out) cudaFree(q);
}

// Gives back what is kept on device `dev`.
void release(int dev, Pool* pool) {
  make_room(dev, lbm::kBlockKeep, nullptr);
  if (pool) cudaMemPoolTrimTo(pool->pool, 0);
}

}  // namespace

namespace lbm {

// From cudaMalloc, once more without what is kept if there is no memory.
static cudaError_t dev_alloc_direct(void** p, size_t bytes, int dev, bool keep) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    release(dev, pool_of(dev));
    e = cudaMalloc(p, bytes);
  }
  if (e == cudaSuccess && *p) {
    std::lock_guard<std::mutex> hold(g_lock);
    g_direct[*p] = Block{bytes, dev, keep};
  }
  return e;
}

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
    // out of memory with freed blocks kept: try without the pool
    *p = nullptr;
    cudaGetLastError();
  }
  return dev_alloc_direct(p, bytes, dev, false);
}

cudaError_t dev_alloc_block(void** p, size_t bytes) {
  *p = nullptr;
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  {
    // the tightest of the kept blocks, at most a quarter larger
    std::lock_guard<std::mutex> hold(g_lock);
    size_t best = g_kept.size();
    for (size_t i = 0; i < g_kept.size(); ++i)
      if (g_kept[i].dev == dev && g_kept[i].bytes >= bytes && g_kept[i].bytes <= bytes + bytes / 4 &&
          (best == g_kept.size() || g_kept[i].bytes < g_kept[best].bytes))
        best = i;
    if (best < g_kept.size()) {
      *p = g_kept[best].p;
      g_direct[*p] = Block{g_kept[best].bytes, dev, true};
      g_kept.erase(g_kept.begin() + best);
      return cudaSuccess;
    }
  }
  return dev_alloc_direct(p, bytes, dev, bytes <= kBlockKeep);
}

void dev_free(void* p) {
  if (!p) return;
  Block b{0, 0, false};
  bool direct = false;
  {
    std::lock_guard<std::mutex> hold(g_lock);
    auto it = g_direct.find(p);
    if (it != g_direct.end()) {
      direct = true;
      b = it->second;
      g_direct.erase(it);
    }
  }
  if (b.keep) {
    make_room(b.dev, b.bytes, p);
    return;
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
  if (pool) e = cudaStreamSynchronize(pool->stream);
  if (e == cudaSuccess) release(dev, pool);
  return (int)e;
}

}  // extern "C"
