// The storm's electric potential on the device (src/core/electric.ts:15-60): Laplacian(phi) = -rho/eps0 at the nodes,
// phi = 0 on the ground and top levels, periodic in x and y. A 2-D DFT of each interior level's right-hand side, one
// stretched vertical tridiagonal per horizontal mode with fixed ends, the inverse DFT: the FP64 spectral solve of
// sg_spectral64.cuh over the interior levels. All in FP64: the reference's own tests hold the solution to 1e-9 of the
// discrete Poisson equation and the plate field to 5e-7. Used by the standalone solver (sg_electric.cu) and by the
// lightning of an electrified run (sg_lightning.cu), each on its own buffers.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <vector>
#include "sg_spectral64.cuh"

namespace sg {

constexpr int ELEC_MAXNI = 128;  // interior levels

// The host tables of a grid as the sweep takes them (S.shape() set): minus the eigenvalue of the 5-point horizontal
// Laplacian per mode (electric.ts:29), the rows' off-diagonals 1/(hz dzs) below and above each level (:45), and every
// mode's elimination in the reference's order (:46-48): piv = di - lo cp_{j-1}, c = up / piv, b = lo / piv, and a = 1 / piv
// with the right-hand side's -1/eps0 and the transforms' factor; the twiddles exp(2 pi i t / n).
inline void elec_host_tables(const Spectral64& S, double dx, double dy, const double* dzs, const double* hz, std::vector<double>& a,
                             std::vector<double>& b, std::vector<double>& c, std::vector<double2>& tx, std::vector<double2>& ty) {
  const double EPSILON0 = 8.8541878128e-12;  // src/core/electric.ts:6
  const double PI = 3.14159265358979323846;
  const int nx = S.nx, ny = S.ny, ni = S.levels;
  const size_t spec = (size_t)ni * S.modes;
  const double factor = -S.factor() / EPSILON0;
  a.assign(spec, 0.0); b.assign(spec, 0.0); c.assign(spec, 0.0);
  for (int m = 0; m <= S.mh; m++)
    for (int q = 0; q < ny; q++) {
      const double lam = 4 * std::pow(std::sin(PI * m / nx), 2) / (dx * dx) + 4 * std::pow(std::sin(PI * q / ny), 2) / (dy * dy);
      double cprev = 0;
      for (int j = 0; j < ni; j++) {
        const int k = j + 1;
        const double lo = 1 / (hz[k] * dzs[k - 1]), up = 1 / (hz[k] * dzs[k]), di = -lo - up - lam, low = j > 0 ? lo : 0;
        const double ip = 1 / (j == 0 ? di : di - low * cprev);
        cprev = j < ni - 1 ? up * ip : 0;
        const size_t at = (size_t)j * S.modes + (size_t)m * ny + q;
        a[at] = factor * ip; b[at] = low * ip; c[at] = cprev;
      }
    }
  tx.resize(nx); ty.resize(ny);
  for (int t = 0; t < nx; t++) tx[t] = make_double2(std::cos(2 * PI * t / nx), std::sin(2 * PI * t / nx));
  for (int t = 0; t < ny; t++) ty[t] = make_double2(std::cos(2 * PI * t / ny), std::sin(2 * PI * t / ny));
}

// phi (device, n) of rho (device, n); phi's ground and top levels are left as they are (zero: the caller clears them once).
inline void elec_solve_launch(const Spectral64& S, const double* rho, double* phi, cudaStream_t st) {
  const size_t layer = (size_t)S.nx * S.ny;
  S.solve(rho + layer, phi + layer, 0, st);
}

}  // namespace sg
