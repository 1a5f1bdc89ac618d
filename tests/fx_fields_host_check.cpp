// Host build of the fixed-point equilibrium and hydrodynamic fields
// (csrc/fx64.cuh) for tests/test_fx64_fields.py.
//
// usage: fx_fields_host_check eq|hydro in.bin out.bin
//   eq:    4 doubles (rho, u) per cell in, 15 populations and the flag out
//   hydro: 15 populations per cell in, rho, u and the flag out
// The flag says whether the fixed point took the cell.
#include <cstdio>
#include <cstring>

#include "fx64.cuh"

int main(int argc, char** argv) {
  if (argc != 4) return 2;
  std::FILE* in = std::fopen(argv[2], "rb");
  std::FILE* out = std::fopen(argv[3], "wb");
  if (!in || !out) return 3;
  if (std::strcmp(argv[1], "eq") == 0) {
    double c[4], f[lbx::NV + 1];
    while (std::fread(c, sizeof(double), 4, in) == 4) {
      f[lbx::NV] = lbx::equilibrium_fx(c[0], c[1], c[2], c[3], f) ? 1.0 : 0.0;
      lbx::equilibrium_f64(c[0], c[1], c[2], c[3], f);
      std::fwrite(f, sizeof(double), lbx::NV + 1, out);
    }
  } else {
    double f[lbx::NV], c[5];
    while (std::fread(f, sizeof(double), lbx::NV, in) == (size_t)lbx::NV) {
      c[0] = c[1] = c[2] = c[3] = 0.0;
      c[4] = lbx::hydro_fx(f, c, c + 1) ? 1.0 : 0.0;
      std::fwrite(c, sizeof(double), 5, out);
    }
  }
  std::fclose(in);
  return std::fclose(out) == 0 ? 0 : 4;
}
