// Large copies between a caller's pageable memory and the device.
//
// The driver stages a pageable copy through its own pinned buffer with one
// thread: that thread's memcpy, and the page faults of a destination that was
// just allocated, set the time.  Here several threads take chunks in turn, each
// with two pinned chunks and a stream of its own, so that the transfers, the
// copies and the faults of the chunks overlap: 50 MB of packed bases to fresh
// memory 11.3 -> 2.5 ms, 17 MB of records in and 148 MB of entries and prefix
// table out (pga_build_kmer_adapter) 37-43 -> 8-10.  Below STAGE_MIN starting
// the threads costs what they save; those copies, and memory that is pinned or
// managed, go to the driver.  pga_gdb_load of warm memory, driver and staged: 4 MB
// 0.28 and 0.32 ms, 5 MB 0.33 and 0.36, 6 MB 0.39 and 0.38, 8 MB 0.49 and 0.46,
// 16 MB 0.92 and 0.73; pga_gdb_copy, 5 MB 0.34 and 0.37, 12 MB 0.78 and 0.57.
#pragma once
#include <atomic>
#include <cstdint>
#include <cstring>
#include <exception>
#include <thread>
#include <cuda_runtime.h>

namespace pga {

class HostCopier {
 public:
  static constexpr int WORKERS = 8;
  static constexpr size_t CHUNK = 1 << 20;
  static constexpr size_t STAGE_MIN = 6 << 20;

  // Copies `bytes` between `host` and `dev` in `st`'s order; a staged copy has
  // ended on return, any other is as cudaMemcpyAsync leaves it.
  cudaError_t copy(int device, void *dev, void *host, size_t bytes, bool to_host, cudaStream_t st) {
    const cudaMemcpyKind kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
    void *dst = to_host ? host : dev;
    const void *src = to_host ? dev : host;
    if (bytes < STAGE_MIN || !pageable(host) || !ready()) return cudaMemcpyAsync(dst, src, bytes, kind, st);
    cudaError_t e = cudaEventRecord(before_, st);
    if (e != cudaSuccess) return e;
    const size_t chunks = (bytes + CHUNK - 1) / CHUNK;
    std::atomic<size_t> next{0};
    std::atomic<int> err{(int)cudaSuccess};
    auto work = [&](int w) {
      cudaError_t r = cudaSetDevice(device);
      if (r == cudaSuccess) r = cudaStreamWaitEvent(st_[w], before_, 0);
      uint8_t *slot = pin_ + (size_t)w * 2 * CHUNK;
      size_t at = 0, had = chunks;  // the chunk in the other slot (chunks: none)
      for (int s = 0; r == cudaSuccess; s ^= 1) {
        const size_t c = err.load() == (int)cudaSuccess ? next.fetch_add(1) : chunks;
        if (!to_host) {
          // (the slot's copy before last has ended: each is waited for below)
          if (c >= chunks) break;
          memcpy(slot + s * CHUNK, (const uint8_t *)host + c * CHUNK, length(bytes, c));
          if (had < chunks) r = cudaStreamSynchronize(st_[w]);
          if (r == cudaSuccess)
            r = cudaMemcpyAsync((uint8_t *)dev + c * CHUNK, slot + s * CHUNK, length(bytes, c), kind, st_[w]);
          had = c;
          continue;
        }
        // the chunk before this one has arrived: write it out while this one comes
        if (had < chunks) r = cudaStreamSynchronize(st_[w]);
        if (r == cudaSuccess && c < chunks)
          r = cudaMemcpyAsync(slot + s * CHUNK, (const uint8_t *)dev + c * CHUNK, length(bytes, c), kind, st_[w]);
        if (r == cudaSuccess && had < chunks) memcpy((uint8_t *)host + had * CHUNK, slot + at, length(bytes, had));
        if (c >= chunks) break;
        had = c;
        at = s * CHUNK;
      }
      const cudaError_t end = cudaStreamSynchronize(st_[w]);
      if (r == cudaSuccess) r = end;
      if (r != cudaSuccess) err.store((int)r);
    };
    std::thread t[WORKERS];
    int n = (int)std::thread::hardware_concurrency();
    n = n < 1 ? 1 : n > WORKERS ? WORKERS : n;
    for (int w = 1; w < n; w++) {
      try {
        t[w] = std::thread(work, w);
      } catch (const std::exception &) {
        break;  // no thread or no memory for one: fewer threads, then
      }
    }
    work(0);
    for (int w = 1; w < n; w++)
      if (t[w].joinable()) t[w].join();
    return (cudaError_t)err.load();
  }

  // Gives back the pinned chunks and streams (on the context's device).
  void release() {
    for (cudaStream_t &s : st_) {
      if (s) cudaStreamDestroy(s);
      s = nullptr;
    }
    if (before_) cudaEventDestroy(before_);
    before_ = nullptr;
    if (pin_) cudaFreeHost(pin_);
    pin_ = nullptr;
  }

 private:
  static size_t length(size_t bytes, size_t c) { return bytes - c * CHUNK < CHUNK ? bytes - c * CHUNK : CHUNK; }
  static bool pageable(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return false;
  }
  bool ready() {
    if (pin_) return true;
    bool ok = cudaEventCreateWithFlags(&before_, cudaEventDisableTiming) == cudaSuccess;
    for (int w = 0; ok && w < WORKERS; w++) ok = cudaStreamCreateWithFlags(&st_[w], cudaStreamNonBlocking) == cudaSuccess;
    void *p = nullptr;
    ok = ok && cudaHostAlloc(&p, WORKERS * 2 * CHUNK, cudaHostAllocDefault) == cudaSuccess;
    if (ok) {
      pin_ = (uint8_t *)p;
      return true;
    }
    cudaGetLastError();
    release();
    return false;
  }

  uint8_t *pin_ = nullptr;
  cudaStream_t st_[WORKERS] = {};
  cudaEvent_t before_ = nullptr;
};

}  // namespace pga
