// host_pages.h -- what the host knows of a caller's memory (plain C++, so that
// the tests run it without the library).
#pragma once
#include <sys/mman.h>
#include <unistd.h>

#include <cstddef>
#include <cstdint>
#include <initializer_list>

namespace lbx {

// Whether the pages of [p, p + bytes) have been made, which a new array's are at
// its first writing: a look at a third and two thirds of it (0.8 us each; the
// first and the last page of new memory may hold the allocator's own words).
inline bool pages_made(const void* p, size_t bytes) {
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), third = bytes / 3;
  for (uintptr_t at : {(uintptr_t)p + third, (uintptr_t)p + 2 * third}) {
    unsigned char in = 0;
    if (mincore(reinterpret_cast<void*>(at & ~(page - 1)), page, &in) != 0 || !(in & 1)) return false;
  }
  return true;
}

}  // namespace lbx
