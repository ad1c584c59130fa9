// Preloaded into a test process: host calls that fail on demand, so that what the library does
// then can be tested without running the machine out of anything.
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <sys/mman.h>

#include <cstdlib>
#include <new>

extern "C" {
int threads_left = -1;               // pthread_create fails after this many (negative: never)
int fail_new = 0;                    // the next operator new of fail_new_min .. fail_new_max bytes
size_t fail_new_min = 0, fail_new_max = 0;
size_t fail_mmap = 0;                // every anonymous mmap of this many bytes, counted
int failed_mmaps = 0;

int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
  if (threads_left == 0) return EAGAIN;
  if (threads_left > 0) --threads_left;
  return real(t, a, f, arg);
}

void* mmap(void* addr, size_t n, int prot, int flags, int fd, off_t off) {
  using Fn = void* (*)(void*, size_t, int, int, int, off_t);
  static Fn real = (Fn)dlsym(RTLD_NEXT, "mmap");
  if (fail_mmap && n == fail_mmap && (flags & MAP_ANONYMOUS)) {
    ++failed_mmaps;
    errno = ENOMEM;
    return MAP_FAILED;
  }
  return real(addr, n, prot, flags, fd, off);
}
}

void* operator new(size_t n) {
  if (fail_new && n >= fail_new_min && n <= fail_new_max) {
    fail_new = 0;
    throw std::bad_alloc();
  }
  void* p = std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
