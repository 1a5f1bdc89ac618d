// Host build of the cell numbering of the box kernels (csrc/kernels.cuh) for
// tests/test_cells_host.py.
//
// usage: cells_host_check < lines of "nx ny nz c": the coordinates of the
// c-th thread's cell, or "beyond"; then the threads that the launch makes
#include <cstdio>

#include "kernels.cuh"

int main() {
  int n[3];
  unsigned long long c;
  while (std::scanf("%d %d %d %llu", &n[0], &n[1], &n[2], &c) == 4) {
    const lbx::Box3 b = lbx::make_box(n[0], n[1], n[2], 0);
    int x, y, z;
    const bool in = lbx::cells32(b) ? lbx::cell_coords<uint32_t>(b, (uint32_t)c, x, y, z)
                                    : lbx::cell_coords<uint64_t>(b, (uint64_t)c, x, y, z);
    const lbx::CellLaunch l = lbx::cell_launch(b, 128);
    const unsigned long long threads = (unsigned long long)l.grid.x * l.block.x;
    if (in)
      std::printf("%d %d %d %llu\n", x, y, z, threads);
    else
      std::printf("beyond %llu\n", threads);
  }
  return 0;
}
