// The masked projection's conjugate gradients (src/core/terrain.ts:306-336) in one order of operations that stays as it is:
// the reference's where a value is formed (node by node gradients, quotients where it divides, direct Fourier sums from
// the first term on), with the products fused into their sums, and trees over blocks of 256 for the dot products, which
// the reference adds one by one. sg_masked.cu runs it where the solve's residuals lose their orthogonality, so that
// rounding decides the iterations and every other order gives another answer: see k_mp_xinv's watch.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

namespace sg {

struct OrderedState {
  double bb, tol2bb, rz, rr, alpha, beta, tolerance;
  int k, done, maxIt;
};

struct OrderedSolve {
  const uint8_t *solid, *wall, *dropped;
  // A, B, invMass, rho4, dzs, idz: as k_mp_flux takes them; lo, cp, piv, rpiv: the sweep's lower coefficient, upper /
  // pivot, pivot and its reciprocal of each mode and layer
  const double *A, *B, *invMass, *rho4, *dzs, *idz, *lo, *cp, *piv, *rpiv;
  const double2 *twx, *twy;
  int nx, ny, nz, layer, nc, mh, modes;
  size_t n, cells;
  double dx, dy, rdx, rdy;  // rdx, rdy: 1 / dx, 1 / dy
  // The caller's vectors, cells long but fu, fv and fw (n); S1, S2 nc * modes; part parts() long; arrived zero.
  double *b, *q, *r, *z, *d, *e, *sd, *fu, *fv, *fw, *part;
  double2 *S1, *S2;
  unsigned* arrived;
  OrderedState* st;

  size_t parts() const;
  // Masked u, v, w and the first guess p: to the projected winds and the pressure kept. `graph` holds eight iterations
  // after the first call (the buffers are the caller's object's own).
  cudaError_t solve(float* u, float* v, float* w, double* p, double dt, int maxIt, double tolerance, cudaGraphExec_t* graph, OrderedState* end,
                    cudaStream_t s) const;
};

}  // namespace sg
