// Large copies between a caller's pageable memory and the device.
//
// The driver stages a pageable copy through its own pinned buffer with one
// thread: that thread's memcpy, and the page faults of a destination that was
// just allocated, set the time.  Here several threads take chunks in turn, each
// with two pinned chunks and a stream of its own, so that the transfers, the
// copies and the faults of the chunks overlap: 50 MB of packed bases to fresh
// memory 11.3 -> 2.5 ms, 17 MB of records in and 148 MB of entries and prefix
// table out (pga_build_kmer_adapter) 37-43 -> 8-10.  Below a size starting the
// threads costs what they save; those copies, and memory that is pinned or
// managed, go to the driver.  Where the line lies depends on the direction, and
// going out on whether the destination's pages are there.  Driver, and 8 and 4
// threads, us, each after 2 ms in which the threads' cores were idle:
//   in                6 MB 304, 358, 298    8 MB 391, 410, 340   16 MB 750, 604, 525   48 MB 2640, 1370, 1300
//   out, pages there  8 MB 512, 865, 864   16 MB 995, 1075, 970  20 MB 1230, 1073, 1050  48 MB 2890, 1875, 1800
//   out, fresh pages  4 MB 1840, 1110, 1060  8 MB 3660, 1260, 1250  16 MB 7310, 1510, 2200  48 MB 21800, 3620, 5710
#pragma once
#include <atomic>
#include <cstdint>
#include <cstring>
#include <exception>
#include <thread>
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

namespace pga {

class HostCopier {
 public:
  static constexpr int WORKERS = 8;
  static constexpr size_t CHUNK = 1 << 20;
  static constexpr size_t IN_MIN = 8 << 20, OUT_MIN = 20 << 20, FRESH_MIN = 4 << 20;  // least bytes staged

  // Copies `bytes` between `host` and `dev` in `st`'s order; a staged copy has
  // ended on return, any other is as cudaMemcpyAsync leaves it.
  cudaError_t copy(int device, void *dev, void *host, size_t bytes, bool to_host, cudaStream_t st) {
    const cudaMemcpyKind kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
    void *dst = to_host ? host : dev;
    const void *src = to_host ? dev : host;
    const bool faults = to_host && bytes >= FRESH_MIN && fresh(host, bytes);
    if (bytes < (faults ? FRESH_MIN : to_host ? OUT_MIN : IN_MIN) || !pageable(host) || !ready())
      return cudaMemcpyAsync(dst, src, bytes, kind, st);
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
    const int most = faults ? WORKERS : WORKERS / 2;
    n = n < 1 ? 1 : n > most ? most : n;
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
  // Whether of 16 pages across the destination half or more are not there yet.
  static bool fresh(const void *p, size_t bytes) {
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    int absent = 0;
    for (int i = 0; i < 16; i++) {
      unsigned char there = 1;
      const uintptr_t at = ((uintptr_t)p + bytes / 16 * i) & ~(page - 1);
      if (mincore((void *)at, 1, &there) == 0) absent += !(there & 1);
    }
    return absent >= 8;
  }
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
