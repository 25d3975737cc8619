// The storm's electric potential on the device: the reference's ElectricSolver (src/core/electric.ts:15-60), which
// the lightning re-solves for every flash (Lightning.discharge, src/core/lightning.ts:231). Laplacian(phi) = -rho/eps0
// at the nodes, phi = 0 on the ground and top levels, periodic in x and y: a 2-D DFT of each interior level's right-hand
// side, one stretched vertical tridiagonal per horizontal mode with fixed ends (Thomas, the reference's rows and
// pivots), the inverse DFT. All in FP64: the reference's own tests hold the solution to 1e-9 of the discrete Poisson
// equation and the plate field to 5e-7, and a solve is small (the standard grid's is 60 thousand nodes). Its five launches
// are sg_spectral64's: mixed-radix transforms along x (two real rows a complex one) and y, the sweeps, y and x back.
#include <cuda_runtime.h>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "sg_elec_solve.cuh"
#include "sg_kernels.h"
#include "stormgpu.h"

struct sg_electric {
  sg_context* ctx = nullptr;
  int nx = 0, ny = 0, nz = 0;
  char* mem = nullptr;
  double *rho = nullptr, *phi = nullptr;
  sg::Spectral64 sp;
};

extern "C" {

int sg_electric_create(sg_context* ctx, const sg_grid* g, sg_electric** out) {
  if (!ctx || !out) return SG_ERR_INVALID;
  *out = nullptr;
  if (!g || !g->dzs || !g->hz || g->nx < 1 || g->ny < 1 || !(g->dx > 0) || !(g->dy > 0))
    return sg_context_fail(ctx, SG_ERR_INVALID, "electric solver: a grid with nx, ny >= 1, dx, dy > 0 and its level arrays");
  if (g->nz < 3) return sg_context_fail(ctx, SG_ERR_INVALID, "the electric solver needs an interior level");
  if (g->nz - 2 > sg::ELEC_MAXNI) return sg_context_fail(ctx, SG_ERR_INVALID, "electric solver: at most 130 levels");
  // (the transforms' pairs of rows and columns in shared memory: at most 64 KB)
  if (g->nx > 2048 || g->ny > 2048) return sg_context_fail(ctx, SG_ERR_INVALID, "electric solver: nx and ny at most 2048");
  const int nx = g->nx, ny = g->ny, nz = g->nz;
  for (int k = 0; k < nz; k++)
    if (!(g->hz[k] > 0) || (k < nz - 1 && !(g->dzs[k] > 0))) return sg_context_fail(ctx, SG_ERR_INVALID, "electric solver: level spacings must be positive");
  if (cudaSetDevice(sg_context_device(ctx)) != cudaSuccess) return sg_context_fail(ctx, SG_ERR_DEVICE, "electric solver: cudaSetDevice");
  sg::Spectral64 sp;
  sp.shape(nx, ny, nz - 2);
  const size_t n = (size_t)nx * ny * nz, spec = (size_t)sp.levels * sp.modes;
  // one allocation: rho, phi [n]; the spectrum [ni][mh + 1][ny] complex; the sweep's coefficients [ni][modes]; twiddles
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t oRho = 0, oPhi = oRho + al(n * 8), oS = oPhi + al(n * 8), oA = oS + al(spec * 16), oB = oA + al(spec * 8), oC = oB + al(spec * 8),
               oTx = oC + al(spec * 8), oTy = oTx + al((size_t)nx * 16), total = oTy + al((size_t)ny * 16);
  auto* s = new sg_electric;
  s->ctx = ctx; s->nx = nx; s->ny = ny; s->nz = nz;
  cudaError_t e = sg::spectral64_limits();
  if (e != cudaSuccess) { delete s; return sg_context_fail(ctx, SG_ERR_DEVICE, "electric solver: shared memory"); }
  e = cudaMalloc(&s->mem, total);
  if (e != cudaSuccess) { delete s; cudaGetLastError(); return sg_context_fail(ctx, SG_ERR_BUDGET, "electric solver: device memory"); }
  s->rho = (double*)(s->mem + oRho); s->phi = (double*)(s->mem + oPhi);
  sp.S = (double2*)(s->mem + oS); sp.a = (double*)(s->mem + oA); sp.b = (double*)(s->mem + oB); sp.c = (double*)(s->mem + oC);
  sp.twx = (double2*)(s->mem + oTx); sp.twy = (double2*)(s->mem + oTy);
  s->sp = sp;
  std::vector<double> a, b, c;
  std::vector<double2> tx, ty;
  sg::elec_host_tables(sp, g->dx, g->dy, g->dzs, g->hz, a, b, c, tx, ty);
  cudaStream_t st = sg_context_stream(ctx);
  if ((e = cudaMemcpyAsync(sp.a, a.data(), spec * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(sp.b, b.data(), spec * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(sp.c, c.data(), spec * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(sp.twx, tx.data(), tx.size() * 16, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(sp.twy, ty.data(), ty.size() * 16, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemsetAsync(s->phi, 0, n * 8, st)) != cudaSuccess ||
      (e = cudaStreamSynchronize(st)) != cudaSuccess) {
    cudaFree(s->mem); delete s;
    return sg_context_fail(ctx, SG_ERR_DEVICE, (std::string("electric solver: ") + cudaGetErrorString(e)).c_str());
  }
  *out = s;
  return SG_OK;
}

int sg_electric_solve(sg_electric* s, const double* rho, double* phi) {
  if (!s) return SG_ERR_INVALID;
  if (!rho || !phi) return sg_context_fail(s->ctx, SG_ERR_INVALID, "electric solver: rho and phi buffers");
  cudaSetDevice(sg_context_device(s->ctx));
  const size_t n = (size_t)s->nx * s->ny * s->nz;
  cudaStream_t st = sg_context_stream(s->ctx);
  cudaError_t e;
  if ((e = cudaMemcpyAsync(s->rho, rho, n * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess)
    return sg_context_fail(s->ctx, SG_ERR_DEVICE, (std::string("electric solver: ") + cudaGetErrorString(e)).c_str());
  sg::elec_solve_launch(s->sp, s->rho, s->phi, st);  // (phi's ground and top levels are zero since the solver was made)
  if ((e = cudaMemcpyAsync(phi, s->phi, n * 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess || (e = cudaStreamSynchronize(st)) != cudaSuccess ||
      (e = cudaGetLastError()) != cudaSuccess)
    return sg_context_fail(s->ctx, SG_ERR_DEVICE, (std::string("electric solver: ") + cudaGetErrorString(e)).c_str());
  return SG_OK;
}

int sg_electric_destroy(sg_electric* s) {
  if (!s) return SG_ERR_INVALID;
  cudaSetDevice(sg_context_device(s->ctx));
  cudaStreamSynchronize(sg_context_stream(s->ctx));
  cudaFree(s->mem);
  delete s;
  return SG_OK;
}

}  // extern "C"
