// Host check of cf1_hostcopier.h: copies and shares come out whole with all
// the threads asked for, with some, and with none to be had -- pthread_create
// (given here) refuses from a given thread on, or operator new does.
#include <dlfcn.h>
#include <pthread.h>

#include <cerrno>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <new>

#include "cf1_hostcopier.h"

static std::atomic<int> threads_left{1 << 30}, started{0};
static std::atomic<long> news_left{1L << 60};

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
  using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
  static Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
  if (threads_left.fetch_sub(1) <= 0) return EAGAIN;
  started++;
  return real(t, a, f, arg);
}
void *operator new(size_t n) {
  if (news_left.fetch_sub(1) <= 0) throw std::bad_alloc();
  if (void *p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

static bool copies() {
  static unsigned char src[3 << 20], dst[3 << 20];
  cf1::HostCopier c(64u << 20);
  news_left = 1L << 60;
  for (size_t n : {(size_t)0, (size_t)1, (size_t)(64 << 10) - 1, (size_t)(64 << 10), (size_t)100'003, sizeof(src)}) {
    for (size_t i = 0; i < n; i++) src[i] = (unsigned char)(i * 31 + n), dst[i] = 0;
    // (at once, and after the threads have waited)
    for (int r = 0; r < 2; r++) {
      if (r) std::this_thread::sleep_for(std::chrono::milliseconds(2));
      c.copy(dst, src, n);
      if (std::memcmp(dst, src, n)) return false;
      std::memset(dst, 0, n);
    }
  }
  return true;
}

static bool shares(unsigned n) {
  std::atomic<int> done[16] = {};
  cf1::on_threads(n, [&](unsigned t) { done[t]++; });
  news_left = 1L << 60;
  for (unsigned t = 0; t < 16; t++)
    if (done[t] != (t < n)) return false;
  return true;
}

int main() {
  for (int left : {1 << 30, 0, 1, 3}) {
    threads_left = left;
    if (!copies()) return std::printf("copies, %d threads\n", left), 1;
    for (unsigned n : {0u, 1u, 2u, 5u, 16u}) {
      threads_left = left;
      if (!shares(n)) return std::printf("shares %u, %d threads\n", n, left), 1;
    }
  }
  threads_left = 1 << 30;
  if (started == 0) return std::puts("pthread_create was not intercepted"), 1;
  for (long left = 0; left < 12; left++) {
    news_left = left;
    if (!copies()) return std::printf("copies, %ld allocations\n", left), 1;
    news_left = left;
    if (!shares(5)) return std::printf("shares, %ld allocations\n", left), 1;
  }
  std::puts("ok");
  return 0;
}
