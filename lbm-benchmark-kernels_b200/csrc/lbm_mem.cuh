// lbm_mem.cuh -- memory of instances and batches.
//
// Device memory: cudaMalloc and cudaFree take 0.3-0.5 ms each and wait for the
// device, and an instance or a batched domain makes a dozen of them. Blocks up
// to kPoolBlock come from a stream-ordered pool per device instead, which keeps
// at most kPoolKeep bytes of freed memory. Arrays whose pointers the library
// gives out are blocks from cudaMalloc, as pool memory has no
// cudaIpcGetMemHandle and is not mapped to peers by cudaDeviceEnablePeerAccess;
// freed, they are kept whole, at most kBlockKeep bytes per device, for the next
// of about their size. lbm_b200_release_memory gives both back. A block is
// ready for any stream when dev_alloc returns; dev_free wants the work on it
// complete, as seen from the host. Safe from several threads.
//
// Host memory: page-locked, zeroed, in whole 2 MiB pages. These make locking about three times
// as fast as cudaMallocHost (40 MB: 5.8 ms against 17 and 2.7 for clearing it;
// freeing 1.0 against 4.2).
#pragma once
#include <cstddef>

#include <cuda_runtime.h>

namespace lbm {

constexpr size_t kPoolBlock = 64ull << 20;
constexpr size_t kPoolKeep = 192ull << 20;
constexpr size_t kBlockKeep = 64ull << 20;

cudaError_t dev_alloc(void** p, size_t bytes);
template <class T>
cudaError_t dev_alloc(T** p, size_t bytes) {
  return dev_alloc(reinterpret_cast<void**>(p), bytes);
}
// A block of its own, from cudaMalloc.
cudaError_t dev_alloc_block(void** p, size_t bytes);
template <class T>
cudaError_t dev_alloc_block(T** p, size_t bytes) {
  return dev_alloc_block(reinterpret_cast<void**>(p), bytes);
}
void dev_free(void* p);

cudaError_t host_alloc(void** p, size_t bytes);
template <class T>
cudaError_t host_alloc(T** p, size_t bytes) {
  return host_alloc(reinterpret_cast<void**>(p), bytes);
}
void host_free(void* p);

}  // namespace lbm
