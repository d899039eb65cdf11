// The few CUDA runtime calls of hostcopy.cuh on host memory, with two devices, a
// record of what was called, and errors on demand.
#pragma once
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <set>
#include <stddef.h>

enum cudaError_t { cudaSuccess, cudaErrorInvalidValue, cudaErrorMemoryAllocation };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum { cudaMemoryTypeUnregistered, cudaMemoryTypeHost };
enum { cudaEventDisableTiming = 2, cudaHostAllocPortable = 1 };
struct cudaPointerAttributes {
  int type;
};
struct FakeStream {
  int device;
};
typedef FakeStream *cudaStream_t;
typedef int *cudaEvent_t;

struct Fake {
  static inline thread_local int device = 0;
  static inline std::atomic<int> copies{0}, wrong_device{0}, allocs{0}, events{0};
  static inline std::atomic<int> fail_copy{-1};  // this copy fails
  static inline std::atomic<bool> fail_alloc{false};
  static inline std::atomic<size_t> pinned_bytes{0};
  static inline std::mutex mu;
  static inline std::set<std::pair<const char *, const char *>> pinned;
};

inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int *d) {
  *d = Fake::device;
  return cudaSuccess;
}
inline cudaError_t cudaSetDevice(int d) {
  Fake::device = d;
  return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  if (Fake::fail_alloc) return cudaErrorMemoryAllocation;
  *p = malloc(n);
  std::lock_guard<std::mutex> lock(Fake::mu);
  Fake::pinned.insert({(char *)*p, (char *)*p + n});
  Fake::allocs++;
  Fake::pinned_bytes = n;
  return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void *p) {
  std::lock_guard<std::mutex> lock(Fake::mu);
  for (auto it = Fake::pinned.begin(); it != Fake::pinned.end(); ++it)
    if (it->first == p) {
      Fake::pinned.erase(it);
      free(p);
      return cudaSuccess;
    }
  return cudaErrorInvalidValue;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  std::lock_guard<std::mutex> lock(Fake::mu);
  a->type = cudaMemoryTypeUnregistered;
  for (auto &r : Fake::pinned)
    if (p >= r.first && p < r.second) a->type = cudaMemoryTypeHost;
  return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind,
                                   cudaStream_t st) {
  const int at = Fake::copies++;
  if (Fake::device != st->device) Fake::wrong_device++;
  if (at == Fake::fail_copy) return cudaErrorInvalidValue;
  memcpy(to, from, n);
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = new int;
  Fake::events++;
  return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete e;
  Fake::events--;
  return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
