// A model of the CUDA runtime in host memory, for the host layer
// (csrc/lbm_capi.cu, lbm_batch.cu, lbm_mem.cu compiled as plain C++): what the
// library enqueues on a stream runs only when something waits for that stream,
// so that work which nothing orders does not happen to be in order. Device
// memory is host memory filled with 0xCD; built with the address sanitizer, a
// use after a free or of an undersized block ends the program.
//
// The model is as loose as the CUDA documentation allows: an asynchronous copy
// arrives when the stream runs; cudaFreeAsync on an idle stream gives the block
// away at once; cudaFree waits for the block's device first; calls wait for the
// current device only.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <set>
#include <vector>

struct CUstream_st {
  int dev;
  std::deque<std::function<void()>> q;
  std::vector<std::function<void()>>* capture = nullptr;
};
struct CUevent_st {
  double at = 0.0;
};
struct CUgraph_st {
  std::vector<std::function<void()>> ops;
};
struct CUgraphExec_st {
  std::vector<std::function<void()>> ops;
};

namespace fake {

struct Block {
  int dev;
  size_t bytes;
  bool pool;
};
inline int device = 0;
inline std::set<cudaStream_t> streams;
inline std::map<void*, Block> blocks;
inline int failAfter = -1;  // device allocations that succeed before all fail; -1: all succeed
inline size_t capacity = SIZE_MAX;  // device memory there is
inline bool failed = false; // one has failed
inline cudaError_t last = cudaSuccess;
inline bool staged = true;  // copies from the host read their source at the call; false: when the stream runs
inline double now = 0.0;    // ms; moved on by what the cases' launches do
inline int calls = 0;       // copies, clears, waits and allocations so far

inline void run(cudaStream_t s) {
  while (!s->q.empty()) {
    std::function<void()> op = std::move(s->q.front());
    s->q.pop_front();
    op();
  }
}
inline void run_device(int dev) {
  for (cudaStream_t s : streams)
    if (s->dev == dev) run(s);
}
// What a kernel launch does, when its stream runs.
inline void launch(cudaStream_t s, std::function<void()> op) {
  if (s->capture)
    s->capture->push_back(std::move(op));
  else
    s->q.push_back(std::move(op));
}
inline void enqueue(cudaStream_t s, std::function<void()> op) {
  ++calls;
  if (s)
    launch(s, std::move(op));
  else
    op();
}
inline cudaError_t allocate(void** p, size_t bytes, bool pool) {
  *p = nullptr;
  ++calls;
  size_t used = 0;
  for (const auto& b : blocks) used += b.second.bytes;
  if (failAfter == 0 || (capacity != SIZE_MAX && used + bytes > capacity)) {
    failed = true;
    return last = cudaErrorMemoryAllocation;
  }
  if (failAfter > 0) --failAfter;
  if (bytes == 0) return cudaSuccess;
  *p = std::malloc(bytes);
  std::memset(*p, 0xCD, bytes);
  blocks[*p] = Block{device, bytes, pool};
  return cudaSuccess;
}

}  // namespace fake

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = fake::device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { fake::device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = fake::last;
  fake::last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrL2CacheSize ? 4 << 20 : a == cudaDevAttrMultiProcessorCount ? 148 : 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  ++fake::calls;
  fake::run_device(fake::device);
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = new CUstream_st{fake::device, {}};
  fake::streams.insert(*s);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }  // its work still completes
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  ++fake::calls;
  if (s) fake::run(s);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = new CUevent_st; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  for (cudaStream_t s : fake::streams) fake::run(s);
  delete e;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  fake::launch(s, [=] { e->at = fake::now; });
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) {
  for (cudaStream_t s : fake::streams) fake::run(s);
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(b->at - a->at);
  return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) { return fake::allocate(p, n, false); }
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  fake::run_device(fake::blocks.at(p).dev);
  fake::blocks.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps*) {
  *pool = reinterpret_cast<cudaMemPool_t>(1);
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  return fake::allocate(p, n, true);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  fake::blocks.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* at, const void* p) {
  at->device = fake::blocks.at(const_cast<void*>(p)).dev;
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostRegister(void*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }

cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  ++fake::calls;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
  if (fake::staged && kind == cudaMemcpyHostToDevice) {
    const std::vector<char> copy((const char*)s, (const char*)s + n);
    fake::enqueue(st, [=] { std::memcpy(d, copy.data(), n); });
    return cudaSuccess;
  }
  fake::enqueue(st, [=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t st) {
  fake::enqueue(st, [=] {
    for (size_t k = 0; k < h; ++k) std::memcpy((char*)d + k * dp, (const char*)s + k * sp, w);
  });
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  fake::enqueue(st, [=] { std::memset(d, v, n); });
  return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  s->capture = new std::vector<std::function<void()>>();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  *g = new CUgraph_st{*s->capture};
  delete s->capture;
  s->capture = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = new CUgraphExec_st{g->ops};
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) {
  for (auto& op : e->ops) s->q.push_back(op);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete e; return cudaSuccess; }
}
