// hostcopy.cuh -- copies between a field in pageable host memory and the device.
//
// One thread moves a pageable copy through the driver's staging buffer, and faults
// the pages of a fresh destination, at 4 to 11 GB/s; here COPY_THREADS threads each
// take a stretch of the field through a pinned buffer of their own (760 MB: up 68
// ms and now 21, down 190 and 50).  All copies go through the caller's stream, one
// stream does as well as eight.
//
// The buffers are one set per process, released with the last context.  Pinning
// costs 0.6 to 1 ms a megabyte, so the set is a thirty-second of the copy it is made
// for (2 to 16 MB), made anew when a copy would have it larger, and made only once
// COPY_PAYS bytes have been asked for since the last one: a program that opens one
// engine after another takes no longer for its first copies than the driver's way
// (up and down, fresh engine each: 97 MB 8 and 8 ms, the driver's way 9 and 21; 19 MB
// 2 and 5 the driver's way, 4 and 4 with a set of 2 MB).  A copy that finds the set
// in use, or no memory for it, goes the driver's way, as small ones and those in
// pinned memory do.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>

namespace nspt {

constexpr int COPY_THREADS = 8;
constexpr size_t COPY_LEAST = 16u << 20, COPY_PAYS = 48u << 20;
constexpr size_t COPY_CHUNK_MIN = 256u << 10, COPY_CHUNK_MAX = 2u << 20;

// a thread's buffer for a copy: a power of two
inline size_t copy_chunk(size_t bytes) {
  size_t c = COPY_CHUNK_MIN;
  while (c < COPY_CHUNK_MAX && c * COPY_THREADS * 32 < bytes) c *= 2;
  return c;
}

// A device made current in a scope, and the caller's given back
class OnDevice {
 public:
  explicit OnDevice(int device) {
    if (cudaGetDevice(&before_) != cudaSuccess || before_ == device ||
        cudaSetDevice(device) != cudaSuccess)
      before_ = -1;
  }
  ~OnDevice() {
    if (before_ >= 0) cudaSetDevice(before_);
  }
  OnDevice(const OnDevice &) = delete;
  OnDevice &operator=(const OnDevice &) = delete;

 private:
  int before_ = -1;
};

class HostStage {
 public:
  void user(int n) {
    std::lock_guard<std::mutex> lock(mu_);
    users_ += n;
    if (users_ == 0) release();
  }

  // Copy `bytes` between host and dev (of device `device`, whose stream st is).
  // The caller's current device is left as it was.
  cudaError_t copy(cudaStream_t st, int device, void *host, void *dev, size_t bytes,
                   bool to_host) {
    const cudaMemcpyKind kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
    const OnDevice current(device);
    std::unique_lock<std::mutex> lock(mu_, std::defer_lock);
    if (bytes < COPY_LEAST || pinned(host) || !lock.try_lock() || !ready(bytes)) {
      const cudaError_t e =
          cudaMemcpyAsync(to_host ? host : dev, to_host ? dev : host, bytes, kind, st);
      return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    const size_t chunk = std::min(chunk_, copy_chunk(bytes));
    const size_t chunks = (bytes + chunk - 1) / chunk;
    cudaError_t err[COPY_THREADS] = {};
    auto part = [&](int t) {
      char *pin = buf_ + t * chunk_;
      cudaEvent_t done;
      cudaError_t e = cudaEventCreateWithFlags(&done, cudaEventDisableTiming);
      if (e == cudaSuccess) {
        for (size_t c = t * chunks / COPY_THREADS;
             c < (t + 1) * chunks / COPY_THREADS && e == cudaSuccess; c++) {
          const size_t at = c * chunk, n = std::min(chunk, bytes - at);
          char *h = (char *)host + at, *d = (char *)dev + at;
          if (!to_host) memcpy(pin, h, n);
          e = cudaMemcpyAsync(to_host ? pin : d, to_host ? d : pin, n, kind, st);
          if (e == cudaSuccess) e = cudaEventRecord(done, st);
          if (e == cudaSuccess) e = cudaEventSynchronize(done);
          if (e == cudaSuccess && to_host) memcpy(h, pin, n);
        }
        cudaEventDestroy(done);
      }
      err[t] = e;
    };
    std::thread th[COPY_THREADS];
    int n = 1;
    try {
      for (; n < COPY_THREADS; n++)
        th[n] = std::thread([&part, device, n] {
          const OnDevice current(device);
          part(n);
        });
    } catch (...) {  // no more threads: this one does the rest
    }
    part(0);
    for (int t = n; t < COPY_THREADS; t++) part(t);
    for (int t = 1; t < n; t++) th[t].join();
    // after an error the stream may still use the buffers
    cudaError_t e = cudaStreamSynchronize(st);
    for (int t = 0; t < COPY_THREADS && e == cudaSuccess; t++) e = err[t];
    return e;
  }

 private:
  std::mutex mu_;
  int users_ = 0;
  char *buf_ = nullptr;
  size_t chunk_ = 0;  // bytes of a thread's buffer
  size_t asked_ = 0;  // bytes of large copies, up to COPY_PAYS

  static bool pinned(const void *host) {
    cudaPointerAttributes at;
    const bool p = cudaPointerGetAttributes(&at, host) == cudaSuccess &&
                   at.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return p;
  }
  void release() {  // with mu_ held
    if (buf_) cudaFreeHost(buf_);
    buf_ = nullptr;
    chunk_ = asked_ = 0;
  }
  bool ready(size_t bytes) {  // with mu_ held
    const size_t chunk = copy_chunk(bytes);
    if (buf_ && chunk_ >= chunk) return true;
    asked_ += std::min(bytes, COPY_PAYS);
    if (asked_ < COPY_PAYS) return false;
    char *p = nullptr;
    if (cudaHostAlloc((void **)&p, COPY_THREADS * chunk, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return buf_ != nullptr;  // the smaller set that is there
    }
    release();
    buf_ = p;
    chunk_ = chunk;
    asked_ = COPY_PAYS;
    return true;
  }
};

}  // namespace nspt
