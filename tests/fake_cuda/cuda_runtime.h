// Stand-in for the CUDA runtime, for checks of host code without a GPU: a
// stream is a queue whose operations run when it is synchronised and not
// before (the latest that CUDA allows), device memory is host memory, and
// operations on a block that has gone back to the pool are counted in
// fake().faults.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <set>
#include <vector>

enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1 };
enum cudaMemAllocationType { cudaMemAllocationTypePinned = 1 };
enum cudaMemLocationType { cudaMemLocationTypeDevice = 1 };
enum cudaMemPoolAttr { cudaMemPoolAttrReleaseThreshold = 4 };
enum cudaDeviceAttr { cudaDevAttrComputeCapabilityMajor = 75 };
constexpr unsigned cudaStreamNonBlocking = 1;

struct FakeStream {
  std::vector<std::function<void()>> queue;
  void run() {
    for (auto& op : queue) op();
    queue.clear();
  }
};
using cudaStream_t = FakeStream*;
using cudaMemPool_t = void*;
struct cudaMemPoolProps {
  cudaMemAllocationType allocType;
  struct {
    cudaMemLocationType type;
    int id;
  } location;
};
struct cudaDeviceProp {
  char name[256];
};

struct Fake {
  int faults = 0;
  std::set<void*> live;  // device blocks
  std::set<FakeStream*> streams;
};
inline Fake& fake() {
  static Fake f;
  return f;
}

inline const char* cudaGetErrorString(cudaError_t) { return "error"; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
inline cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 10, cudaSuccess; }
inline cudaError_t cudaGetDeviceProperties(cudaDeviceProp*, int) { return cudaSuccess; }
inline cudaError_t cudaMallocHost(void** p, size_t bytes) { return *p = std::malloc(bytes), cudaSuccess; }
inline cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
inline cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { return *p = p, cudaSuccess; }
inline cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }

inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  fake().streams.insert(*s = new FakeStream);
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) { return s->run(), cudaSuccess; }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) {
  // returns at once; what is pending still runs, later
  if (s->queue.empty()) {
    fake().streams.erase(s);
    delete s;
  }
  return cudaSuccess;
}
inline cudaError_t cudaMallocFromPoolAsync(void** p, size_t bytes, cudaMemPool_t, cudaStream_t) {
  fake().live.insert(*p = std::malloc(bytes));
  return cudaSuccess;
}
inline cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  s->queue.push_back([p] {
    if (!fake().live.erase(p)) ++fake().faults;
  });
  return cudaSuccess;
}
inline cudaError_t cudaMemsetAsync(void* p, int value, size_t bytes, cudaStream_t s) {
  s->queue.push_back([=] {
    if (fake().live.count(p))
      std::memset(p, value, bytes);
    else
      ++fake().faults;
  });
  return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t s) {
  s->queue.push_back([=] {
    if (fake().live.count(dst))
      std::memcpy(dst, src, bytes);
    else
      ++fake().faults;
  });
  return cudaSuccess;
}
