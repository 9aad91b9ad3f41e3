// Test-only: which copies csrc/hostcopy.h starts threads for, on fake device
// memory.  argv: the bytes, the direction (in, out), whether the destination's
// pages are there (warm, fresh), where in a page it begins.  Prints the threads
// started and whether the copy is right.
#include <cstdio>
#include <dlfcn.h>
#include <pthread.h>
#include <string>
#include <sys/mman.h>
#include <vector>
#include "../../distributedpanga_b200/csrc/hostcopy.h"

static std::atomic<long> g_started{0};

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
  using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
  static Fn next = (Fn)dlsym(RTLD_NEXT, "pthread_create");
  g_started++;
  return next(t, a, f, arg);
}

int main(int argc, char **argv) {
  if (argc != 5) return 2;
  const size_t bytes = (size_t)atoll(argv[1]), at = (size_t)atoll(argv[4]);
  const bool out = argv[2] == std::string("out"), warm = argv[3] == std::string("warm");
  std::vector<uint8_t> src(bytes);
  uint32_t x = 1;
  for (auto &v : src) v = (uint8_t)((x = x * 1664525u + 1013904223u) >> 24);
  void *m = mmap(nullptr, bytes + at, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (m == MAP_FAILED) return 3;
  uint8_t *dst = (uint8_t *)m + at;
  if (warm) memset(m, 1, bytes + at);
  pga::HostCopier C;
  // (device memory is host memory: the destination of a copy in is the device's)
  const cudaError_t e = out ? C.copy(0, src.data(), dst, bytes, true, nullptr) : C.copy(0, dst, src.data(), bytes, false, nullptr);
  printf("%ld %d\n", g_started.load(), e == cudaSuccess && memcmp(dst, src.data(), bytes) == 0);
  C.release();
  return 0;
}
