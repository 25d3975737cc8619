// The masked projection's pointwise kernels (sg_masked.cu, cut out by the test as masked_flux.inc) and the ordered solve's
// quotient (sg_masked_ordered.cu, as quotient.inc) run on the CPU: see block_emulator.h.
#include "block_emulator.h"

static struct { int x = 0; } blockIdx;
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
struct MpState { int done; };
struct Geo {
  const uint8_t* dropped;
  const double *A, *B, *rho4, *idz;
  int nx, ny, nz, layer, nc;
  size_t n, cells;
};
constexpr int TPB = 256, R_DSD = 0, R_BB = 1;
template <int OP> void finish_dot(double, double*, unsigned*, MpState*) {}
#include "masked_flux.inc"
#include "quotient.inc"

extern "C" {

// sg_masked_divergence's two kernels over a column's shares A and B (cells), rho0 / 4 and 1 / dzs by level
void tc_divergence(int nx, int ny, int nz, double dx, double dy, const float* u, const float* v, const float* w, const uint8_t* dropped, const double* A,
                   const double* B, const double* rho4, const double* idz, double* out) {
  Geo g{dropped, A, B, rho4, idz, nx, ny, nz, nx * ny, nz - 1, (size_t)nx * ny * nz, (size_t)nx * ny * (nz - 1)};
  std::vector<double> fu(g.cells), fv(g.cells), fw(g.cells);
  for (int pass = 0; pass < 2; pass++)
    for (blockIdx.x = 0; (size_t)blockIdx.x * TPB < g.cells; blockIdx.x++)
      emu::run(TPB, 0, [&] {
        if (pass == 0) k_mp_wind_flux(u, v, w, fu.data(), fv.data(), fw.data(), g);
        else k_mp_div<0>(fu.data(), fv.data(), fw.data(), out, nullptr, 1 / dx, 1 / dy, nullptr, nullptr, g, nullptr, 0);
      });
}

// how many of x[i] / d[i] the quotient from the reciprocal does not give to the last bit (the one for divisors below zero
// with `negative`)
int tc_quotients(const double* x, const double* d, int n, int negative) {
  int wrong = 0;
  for (int i = 0; i < n; i++) wrong += emu::bits((negative ? quotient_negative : quotient)(x[i], d[i], 1 / d[i])) != emu::bits(x[i] / d[i]);
  return wrong;
}

}  // extern "C"
