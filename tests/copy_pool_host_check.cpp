// Host build of the copy threads (csrc/copy_pool.h) for tests/test_copy_pool.py.
//
// usage: copy_pool_host_check threads rounds [of them the system gives]
// Two callers at once, one with chunks of 16 MB and one with chunks of 1 MB and
// less of ever other lengths; prints how many copies came out wrong, or wrote
// beyond their end.
#include <dlfcn.h>
#include <pthread.h>

#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <thread>
#include <vector>

#include "copy_pool.h"

static int g_threads_given = -1;  // pthread_create fails from then on; -1: never
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  using create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static const create real = (create)dlsym(RTLD_NEXT, "pthread_create");
  if (g_threads_given == 0) return EAGAIN;
  if (g_threads_given > 0) --g_threads_given;
  return real(t, a, f, arg);
}

namespace {
constexpr size_t kGuard = 4096;

int caller(lbx::CopyPool& pool, size_t len, int rounds, unsigned seed, bool waits) {
  int wrong = 0;
  std::vector<char> src(len), dst(len + kGuard);
  for (int r = 0; r < rounds; ++r) {
    const size_t n = len - (size_t)(r % 7) * (len / 9) - (size_t)(r % 3);
    for (size_t i = 0; i < n; i += 64) src[i] = (char)(seed + r + i / 64);
    std::fill(dst.begin(), dst.end(), (char)0x5a);
    if (waits || !pool.try_copy(dst.data(), src.data(), n)) pool.copy(dst.data(), src.data(), n);
    bool ok = std::memcmp(dst.data(), src.data(), n) == 0;
    for (size_t i = n; i < dst.size(); ++i) ok = ok && dst[i] == 0x5a;
    wrong += !ok;
  }
  return wrong;
}
}  // namespace

int main(int argc, char** argv) {
  if (argc != 3 && argc != 4) return 2;
  if (argc == 4) g_threads_given = std::atoi(argv[3]);
  lbx::CopyPool pool((unsigned)std::atoi(argv[1]));
  g_threads_given = -1;
  const int rounds = std::atoi(argv[2]);
  int wrong[2];
  std::thread a([&] { wrong[0] = caller(pool, (size_t)16 << 20, rounds, 1, true); });
  std::thread b([&] { wrong[1] = caller(pool, (size_t)1 << 20, 16 * rounds, 77, false); });
  a.join();
  b.join();
  std::printf("%d %d\n", wrong[0], wrong[1]);
  return 0;
}
