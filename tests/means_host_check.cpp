// Host build of the restriction's means and of the interpolation in time
// (csrc/fx64.cuh) for tests/test_fx64_means.py.
//
// usage: means_host_check mean|weighted in.bin out.bin
//   mean:     8 doubles in, mean8 out
//   weighted: wp, a, wn, b in, weighted(wp, a, wn, b) out
#include <cstdio>
#include <cstring>

#include "fx64.cuh"

int main(int argc, char** argv) {
  if (argc != 4) return 2;
  std::FILE* in = std::fopen(argv[2], "rb");
  std::FILE* out = std::fopen(argv[3], "wb");
  if (!in || !out) return 3;
  const bool mean = std::strcmp(argv[1], "mean") == 0;
  const size_t n = mean ? 8 : 4;
  double v[8];
  while (std::fread(v, sizeof(double), n, in) == n) {
    const double r = mean ? lbx::mean8(v) : lbx::weighted(v[0], v[1], v[2], v[3]);
    std::fwrite(&r, sizeof(double), 1, out);
  }
  std::fclose(in);
  return std::fclose(out) == 0 ? 0 : 4;
}
