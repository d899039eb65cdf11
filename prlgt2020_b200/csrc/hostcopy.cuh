// hostcopy.cuh -- copies between a field in pageable host memory and the device.
//
// One thread moves a pageable copy through the driver's staging buffer, and faults
// the pages of a fresh destination, at 4 to 11 GB/s; here COPY_THREADS threads each
// take a stretch of the field through a pinned buffer of their own (760 MB: up 68
// ms and now 21, down 190 and 50).  All copies go through the caller's stream, one
// stream does as well as eight.
//
// The buffers are one set per process (16 MB), released with the last context.  The
// driver takes 10 ms to make them, as long as it takes for 100 MB up or 45 MB down by
// itself, so they are made once COPY_PAYS bytes have been asked for since the last
// release: a program that opens one engine after another waits no longer for its
// copies than with the driver's.  (Huge pages of our own are pinned in 2 ms, but
// downloads through them are slower: 97 MB 4.4 ms and not 3.4, 155 MB 6.6 and 5.9.)
// A copy that finds the set in use, or no memory for it, goes the driver's way, as
// small ones and those in pinned memory do.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>

namespace nspt {

constexpr int COPY_THREADS = 8;
constexpr size_t COPY_LEAST = 16u << 20, COPY_PAYS = 128u << 20;
// a thread's buffer: 97 MB up in 2.7 ms with 2 MB, 3.9 with 512 KB, 4.6 with 256 KB
constexpr size_t COPY_CHUNK = 2u << 20;

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
    const size_t chunks = (bytes + COPY_CHUNK - 1) / COPY_CHUNK;
    cudaError_t err[COPY_THREADS] = {};
    auto part = [&](int t) {
      char *pin = buf_ + t * COPY_CHUNK;
      cudaEvent_t done;
      cudaError_t e = cudaEventCreateWithFlags(&done, cudaEventDisableTiming);
      if (e == cudaSuccess) {
        for (size_t c = t * chunks / COPY_THREADS;
             c < (t + 1) * chunks / COPY_THREADS && e == cudaSuccess; c++) {
          const size_t at = c * COPY_CHUNK, n = std::min(COPY_CHUNK, bytes - at);
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
    asked_ = 0;
  }
  bool ready(size_t bytes) {  // with mu_ held
    if (buf_) return true;
    asked_ += std::min(bytes, COPY_PAYS);
    if (asked_ < COPY_PAYS) return false;
    char *p = nullptr;
    if (cudaHostAlloc((void **)&p, COPY_THREADS * COPY_CHUNK, cudaHostAllocPortable) !=
        cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    buf_ = p;
    return true;
  }
};

}  // namespace nspt
