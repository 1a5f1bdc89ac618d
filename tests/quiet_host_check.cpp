// Host build of what the levels of refined runs add to the fixed-point collision
// (csrc/fx64.cuh) for tests/test_fx64_quiet.py.
//
// usage: quiet_host_check in.bin out.bin omega_s omega_b
// 15 FP64 populations a cell in; 31 doubles out: the populations after
// collide_f64<true> at quiet rates, those after collide<double>, and 1 or 0 for
// whether the cell took the short form of the FP64 collision.
#include <cstdio>
#include <cstdlib>

#include "fx64.cuh"

int main(int argc, char** argv) {
  if (argc != 5) return 2;
  std::FILE* in = std::fopen(argv[1], "rb");
  std::FILE* out = std::fopen(argv[2], "wb");
  if (!in || !out) return 3;
  const double om_s = std::atof(argv[3]), om_b = std::atof(argv[4]);
  lbx::FxRates r = lbx::fx_rates(om_s, om_b);
  r.quiet = 1;
  double f[2 * lbx::NV + 1], g[lbx::NV];
  while (std::fread(f, sizeof(double), lbx::NV, in) == (size_t)lbx::NV) {
    for (int q = 0; q < lbx::NV; ++q) f[lbx::NV + q] = g[q] = f[q];
    f[2 * lbx::NV] = !lbx::collide_fx<true>(g, r) && lbx::is_rest(f) ? 1.0 : 0.0;
    lbx::collide_f64<true>(f, om_s, om_b, r);
    lbx::collide<double>(f + lbx::NV, om_s, om_b, 0.0);
    std::fwrite(f, sizeof(double), 2 * lbx::NV + 1, out);
  }
  std::fclose(in);
  return std::fclose(out) == 0 ? 0 : 4;
}
