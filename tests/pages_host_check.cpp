// Host build of the look at a caller's pages (csrc/host_pages.h) for
// tests/test_host_pages.py: prints, in order, whether the pages are made of new
// memory, of the same with its first and last page written, as an allocator
// does, with its first and with its last third written, of all of it written,
// of a part from the middle of a page on, and of memory that is not mapped.
#include <cstdio>

#include "host_pages.h"

int main() {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = 70;
  auto fresh = [&] {  // small pages: a huge one would be made at a single writing
    char* p = (char*)mmap(nullptr, n * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    madvise(p, n * page, MADV_NOHUGEPAGE);
    return p;
  };
  const struct {
    size_t from, to;
  } written[] = {{n, 0}, {0, n / 3}, {n - n / 3, n}, {0, n}};
  for (const auto& w : written) {
    char* p = fresh();
    if (w.from > w.to) {
      std::printf("%d ", lbx::pages_made(p, n * page));
      p[0] = p[n * page - 1] = 1;
    }
    for (size_t i = w.from; i < w.to; ++i) p[i * page] = 1;
    std::printf("%d ", lbx::pages_made(p, n * page));
    if (w.to - w.from == n) std::printf("%d ", lbx::pages_made(p + page / 2, 3 * page));
    munmap(p, n * page);
    if (w.to - w.from == n) std::printf("%d\n", lbx::pages_made(p, n * page));
  }
  return 0;
}
