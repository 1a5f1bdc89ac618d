// host_pages.h -- what the host knows of a caller's memory (plain C++, so that
// the tests run it without the library).
#pragma once
#include <sys/mman.h>
#include <unistd.h>

#include <cstddef>
#include <cstdint>

namespace lbx {

// Whether the pages of [p, p + bytes) have been made, which a new array's are at
// its first writing: a look at the middle one (0.8 us; the first and the last page
// of new memory may hold the allocator's own words).
inline bool pages_made(const void* p, size_t bytes) {
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
  const uintptr_t at = ((uintptr_t)p + bytes / 2) & ~(page - 1);
  unsigned char in = 0;
  return mincore(reinterpret_cast<void*>(at), page, &in) == 0 && (in & 1);
}

}  // namespace lbx
