// Test-only: csrc/hostcopy.h on fake device memory, with memory or threads
// running out while it starts its threads.  argv[1]: the allocation, from the
// copy's start on, that fails (0: none); argv[2]: the thread that cannot be
// started (0: none).  Copies in and out at sizes around whole chunks, and around
// the least that is worth starting threads for.
#include <cerrno>
#include <cstdio>
#include <dlfcn.h>
#include <new>
#include <pthread.h>
#include <vector>
#include "../../distributedpanga_b200/csrc/hostcopy.h"

static std::atomic<long> g_new{0}, g_thread{0};  // counts down to the one that fails
static std::atomic<long> g_started{0};

void *operator new(size_t n) {
  if (g_new.load() > 0 && --g_new == 0) throw std::bad_alloc();
  void *p = malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
  using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
  static Fn next = (Fn)dlsym(RTLD_NEXT, "pthread_create");
  if (g_thread.load() > 0 && --g_thread == 0) return EAGAIN;
  g_started++;
  return next(t, a, f, arg);
}

int main(int argc, char **argv) {
  const long bad_new = argc > 1 ? atol(argv[1]) : 0, bad_thread = argc > 2 ? atol(argv[2]) : 0;
  pga::HostCopier C;
  const size_t MB = 1 << 20;
  for (size_t bytes : {MB, 6 * MB - 1, 6 * MB, 16 * MB - 1, 16 * MB, 33 * MB + 7}) {
    std::vector<uint8_t> a(bytes), b(bytes), c(bytes);
    uint32_t x = 12345;
    for (auto &v : a) v = (uint8_t)((x = x * 1664525u + 1013904223u) >> 24);
    for (bool out : {false, true}) {
      g_new = bad_new;
      g_thread = bad_thread;
      const cudaError_t e = out ? C.copy(0, b.data(), c.data(), bytes, true, nullptr)
                                : C.copy(0, b.data(), a.data(), bytes, false, nullptr);
      g_new = g_thread = 0;
      if (bytes < 6 * MB && g_started) {
        printf("threads for a copy of %zu bytes\n", bytes);
        return 1;
      }
      if (e != cudaSuccess) {
        printf("copy of %zu bytes failed\n", bytes);
        return 1;
      }
    }
    if (a != c) {
      printf("copy of %zu bytes differs\n", bytes);
      return 1;
    }
  }
  C.release();
  printf("ok\n");
  return 0;
}
