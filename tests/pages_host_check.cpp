// Host build of the look at a caller's pages (csrc/host_pages.h) for
// tests/test_host_pages.py: prints, in order, whether the pages are made of new
// memory, of the same with its first, its middle and its last page left out, of
// all of it written, of a part from the middle of a page on, and of memory that
// is not mapped.
#include <cstdio>

#include "host_pages.h"

int main() {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = 70;
  auto fresh = [&] {  // small pages: a huge one would be made at a single writing
    char* p = (char*)mmap(nullptr, n * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    madvise(p, n * page, MADV_NOHUGEPAGE);
    return p;
  };
  char* p = fresh();
  std::printf("%d", lbx::pages_made(p, n * page));
  for (size_t skip : {(size_t)0, n - 1, n}) {
    char* q = fresh();
    for (size_t i = 0; i < n; ++i)
      if (i != skip) q[i * page] = 1;
    std::printf(" %d", lbx::pages_made(q, n * page));
    if (skip == n) {
      std::printf(" %d", lbx::pages_made(q + page / 2, 3 * page));
      munmap(q, n * page);
      std::printf(" %d\n", lbx::pages_made(q, n * page));
    }
  }
  return 0;
}
