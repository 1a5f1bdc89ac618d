// Host build of the fixed-point FP64 collision (csrc/fx64.cuh) for
// tests/test_fx64.py: collides the cells of a file (15 FP64 populations each)
// and writes 16 doubles per cell: the populations after collide_f64 and 1 or 0
// for whether the fixed point took the cell.
//
// usage: fx_host_check in.bin out.bin omega_s omega_b
#include <cstdio>
#include <cstdlib>

#include "fx64.cuh"

int main(int argc, char** argv) {
  if (argc != 5) return 2;
  std::FILE* in = std::fopen(argv[1], "rb");
  std::FILE* out = std::fopen(argv[2], "wb");
  if (!in || !out) return 3;
  const double om_s = std::atof(argv[3]), om_b = std::atof(argv[4]);
  const lbx::FxRates r = lbx::fx_rates(om_s, om_b);
  double f[lbx::NV + 1];
  while (std::fread(f, sizeof(double), lbx::NV, in) == (size_t)lbx::NV) {
    double g[lbx::NV];
    for (int q = 0; q < lbx::NV; ++q) g[q] = f[q];
    f[lbx::NV] = lbx::collide_fx(g, r) ? 1.0 : 0.0;
    lbx::collide_f64(f, om_s, om_b, r);
    std::fwrite(f, sizeof(double), lbx::NV + 1, out);
  }
  std::fclose(in);
  return std::fclose(out) == 0 ? 0 : 4;
}
