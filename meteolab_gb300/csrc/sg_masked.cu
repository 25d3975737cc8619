// Terrain on GB300 (src/core/terrain.ts): the ground heights of a terrain form and the cut-cell geometry on the host
// (terrainHeights :37-63, solidMask :80-84, groundLevels :87-91, nodeHeights :101-105, faceApertures :119-134,
// slopeArea :141-150), and MaskedProjection (:168-363) on the device: the node mass flux rho0 u made divergence-free
// over the dual cells cut by the ground. The masked operator S = -D M (rho0 H)^-1 D^T is solved by preconditioned
// conjugate gradients with the flat operator's spectral inverse (PressureSolver.solve, src/core/pressure.ts:95-140) as
// the preconditioner, all in FP64 as the reference. The transport's faces with terrain (FluxTransport.setTerrain and
// setVelocityMasked, src/core/advection.ts:78-184) are solved the same way over node vectors, with the flat face solve
// as the preconditioner (sg_faces_*).
//
// Layout: velocities FP32 [n] (node x + nx (y + ny z)); the cells' vectors FP64 [nc * nx * ny], nc = nz - 1 (cell
// x + nx (y + ny k) between node levels k and k + 1); spectra FP64 complex [nc][nx/2 + 1][ny]. One CG iteration is seven
// launches (the faces' six): the new direction with the column fluxes of its gradient, their divergence with d.Sd (the
// faces: one kernel for both), the q/r update with r.r and the preconditioner's x-transform, its y-transform, vertical
// sweeps and y-inverse (sg_spectral64.cuh), and its x-inverse with r.z. Each dot product is finished, and acted on, by
// the block that ends last, from the partials in a fixed order (the result does not depend on scheduling); alpha, beta
// and the stopping test stay on the device. Eight iterations are one CUDA graph,
// replayed until the device's stop flag is set: the host reads one int per eight iterations (a projection whose rounding
// would decide its iterations starts again in a fixed order of operations: sg_masked_ordered.cu); every kernel of an
// iteration after the stop returns at once, so the iterations done, the residual and the result are those
// of the reference's loop (:313-329), which stops at the first top-of-loop test it passes. The FP64 pipe bounds the
// kernels (two operations a clock and SM), so their FP64 instructions are counted: see k_mp_flux and sg_spectral64.cuh.
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "sg_kernels.h"
#include "sg_masked_ordered.cuh"
#include "sg_spectral64.cuh"
#include "stormgpu.h"

using namespace sg;

namespace {

constexpr double PI_ = 3.141592653589793;  // Math.PI
constexpr double LEAST_SHARE = .2;         // terrain.ts:69

// ---------------------------------------------------------------- host geometry

struct HostGrid {
  int nx, ny, nz, layer;
  size_t n;
  double dx, dy, width, depth;
  const double *zs, *dzs, *hz;
  double volumeTop(int k) const { return k < nz - 1 ? zs[k] + dzs[k] / 2 : zs[k]; }  // terrain.ts:72
};

bool host_grid(const sg_grid* g, HostGrid& h) {
  if (!g || !g->zs || !g->dzs || !g->hz || g->nx < 1 || g->ny < 1 || g->nz < 3 || !(g->dx > 0) || !(g->dy > 0)) return false;
  h.nx = g->nx; h.ny = g->ny; h.nz = g->nz; h.layer = g->nx * g->ny; h.n = (size_t)h.layer * g->nz;
  h.dx = g->dx; h.dy = g->dy; h.width = g->dx * g->nx; h.depth = g->dy * g->ny;
  h.zs = g->zs; h.dzs = g->dzs; h.hz = g->hz;
  return true;
}

double js_round(double x) { const double f = std::floor(x); return x - f >= 0.5 ? f + 1 : f; }  // Math.round

// terrainHeights: the form's height per column (periodic distances), two 1-2-1 passes (x, then y), lowest column at 0.
void terrain_heights(const HostGrid& g, const sg_terrain& t, float* h) {
  const int nx = g.nx, ny = g.ny;
  const double cx = (std::isnan(t.x) ? g.width / 2000 : t.x) * 1000, cy = (std::isnan(t.y) ? g.depth / 2000 : t.y) * 1000;
  const double a = std::max(t.width * 1000, 2 * std::max(g.dx, g.dy)), top = t.height * 1000, a2 = a * a;
  const double axis = (std::isnan(t.heading) ? 0 : t.heading) * PI_ / 180, sx = std::sin(axis), sy = std::cos(axis);
  const double lambda = (std::isnan(t.wavelength) ? 4 : t.wavelength) * 1000;
  for (int j = 0; j < ny; j++) {
    double ey = (j + .5) * g.dy - cy;
    ey -= g.depth * js_round(ey / g.depth);
    for (int i = 0; i < nx; i++) {
      double ex = (i + .5) * g.dx - cx;
      ex -= g.width * js_round(ex / g.width);
      const double across = ex * sy - ey * sx;
      double v;
      switch (t.kind) {
        case SG_TERRAIN_HILL: v = top / std::pow(1 + (ex * ex + ey * ey) / a2, 1.5); break;
        case SG_TERRAIN_RIDGE: v = top / (1 + across * across / a2); break;
        case SG_TERRAIN_SCHAR: { const double c = std::cos(PI_ * across / lambda); v = top * std::exp(-across * across / a2) * (c * c); break; }
        default: v = top / (1 + std::exp((std::max(std::fabs(ex), std::fabs(ey)) - a) / (.25 * a)));
      }
      h[i + (size_t)nx * j] = (float)v;
    }
  }
  std::vector<float> tmp((size_t)nx * ny);
  for (int pass = 0; pass < 2; pass++) {
    for (int j = 0; j < ny; j++) {
      const float* row = h + (size_t)nx * j;
      for (int i = 0; i < nx; i++) tmp[i + (size_t)nx * j] = (float)(((double)row[(i + nx - 1) % nx] + 2 * (double)row[i] + (double)row[(i + 1) % nx]) / 4);
    }
    for (int j = 0; j < ny; j++) {
      const float *s = tmp.data() + (size_t)nx * ((j + ny - 1) % ny), *c = tmp.data() + (size_t)nx * j, *nn = tmp.data() + (size_t)nx * ((j + 1) % ny);
      for (int i = 0; i < nx; i++) h[i + (size_t)nx * j] = (float)(((double)s[i] + 2 * (double)c[i] + (double)nn[i]) / 4);
    }
  }
  double low = INFINITY;
  for (size_t c = 0; c < (size_t)nx * ny; c++) low = std::min(low, (double)h[c]);
  for (size_t c = 0; c < (size_t)nx * ny; c++) h[c] = (float)((double)h[c] - low);
}

// solidMask and groundLevels: a column is solid from level 0 up while the ground leaves less than LEAST_SHARE of the
// level's volume above it (never the top two levels); its ground node is the first level that is not.
void solid_levels(const HostGrid& g, const float* ground, uint8_t* solid, int32_t* levels) {
  std::fill(solid, solid + g.n, (uint8_t)0);
  for (int c = 0; c < g.layer; c++) {
    int z = 0;
    while (z < g.nz - 2 && g.volumeTop(z) - (double)ground[c] < LEAST_SHARE * g.hz[z]) { solid[c + (size_t)z * g.layer] = 1; z++; }
    levels[c] = z;
  }
}

// nodeHeights: the ground node's volume above the ground, nothing in the ground, the level's hz elsewhere.
void node_heights(const HostGrid& g, const uint8_t* solid, const int32_t* levels, const float* ground, double* h) {
  for (int z = 0; z < g.nz; z++)
    for (int c = 0; c < g.layer; c++) {
      const size_t i = c + (size_t)z * g.layer;
      h[i] = solid[i] ? 0 : z == levels[c] ? g.volumeTop(z) - (double)ground[c] : g.hz[z];
    }
}

// faceApertures: each face to x + 1 (ax) or y + 1 (ay) open above the mean ground of its two columns in each level's
// layer of volume; a layer's open part next to a solid node carried up to the first face with both nodes fluid.
void face_apertures(const HostGrid& g, const uint8_t* solid, const float* ground, double* ax, double* ay) {
  std::fill(ax, ax + g.n, 0.0);
  std::fill(ay, ay + g.n, 0.0);
  auto shave = [&](double* out, int c, int other) {
    const double face = ((double)ground[c] + (double)ground[other]) / 2;
    double carry = 0;
    for (int k = 0; k < g.nz; k++) {
      const double bottom = k > 0 ? g.volumeTop(k - 1) : 0, open = face <= bottom ? g.hz[k] : std::max(0.0, g.volumeTop(k) - face);
      const size_t i = c + (size_t)k * g.layer;
      if (solid[i] || solid[other + (size_t)k * g.layer]) carry += open;
      else { out[i] = open + carry; carry = 0; }
    }
  };
  for (int j = 0; j < g.ny; j++)
    for (int i = 0; i < g.nx; i++) {
      const int c = i + j * g.nx;
      shave(ax, c, (i + 1) % g.nx + j * g.nx);
      shave(ay, c, i + ((j + 1) % g.ny) * g.nx);
    }
}

void slope_area(const HostGrid& g, const float* h, float* area) {
  const int nx = g.nx, ny = g.ny;
  for (int j = 0; j < ny; j++)
    for (int i = 0; i < nx; i++) {
      const double hx = ((double)h[(i + 1) % nx + nx * j] - (double)h[(i + nx - 1) % nx + nx * j]) / (2 * g.dx);
      const double hy = ((double)h[i + nx * ((j + 1) % ny)] - (double)h[i + nx * ((j + ny - 1) % ny)]) / (2 * g.dy);
      area[i + (size_t)nx * j] = (float)std::sqrt(1 + hx * hx + hy * hy);
    }
}

// ---------------------------------------------------------------- device

// The solve's scalars on the device. done: 0 iterating, 1 stopped (converged, no descent, or out of iterations),
// 2 a zero right-hand side (nothing to project), 4 the residuals have lost their orthogonality (see k_mp_xinv).
struct MpState {
  double bb, tol2bb, rz, rr, rz0, alpha, beta, tolerance;
  double watch;  // the square of what r . z0 may grow to, of r.z r0.z0
  int k, done, maxIt, keepRR;
};
constexpr double WATCH_LIMIT = 1e-18;
enum { STOP = 1, ZERO = 2, DRIFT = 4, ANY = 7 };
enum { R_BB, R_RR0, R_RZ0, R_DSD, R_RR, R_RZN };

struct Geo {
  const uint8_t *solid, *wall, *dropped;
  // A, B: a column's shares of each cell layer's fluxes (see k_mp_flux); invMass 1 / (rho0 h), wMass rho0 / 4 of it, zero
  // where w is; rho4 rho0 / 4; idz 1 / dzs
  const double *A, *B, *invMass, *wMass, *rho, *rho4, *dzs, *idz, *hz;
  int nx, ny, nz, layer, nc;
  size_t n, cells;
  double dx, dy;
};

constexpr int TPB = 256;

// Sum over the block (valid in thread 0); every thread of the block calls it.
__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  v = 0;
  if (wid == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;
}

// mask (terrain.ts:229-234): the solid nodes at rest, w zero at the wall nodes and on the ground and top levels.
__global__ void k_mp_mask(float* __restrict__ u, float* __restrict__ v, float* __restrict__ w, Geo g) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  if (g.solid[i]) { u[i] = 0; v[i] = 0; w[i] = 0; }
  else if (g.wall[i] || i < (size_t)g.layer || i >= g.n - g.layer) w[i] = 0;
}

// Adds a dot product's block sums and acts on it in the block that finishes last (a counter; no block waits): the
// partials in a fixed order, so the result does not depend on which block that is (the scalars of :306-329).
// WATCH: with a second sum, r . z0.
template <int OP, bool WATCH = false>
__device__ __forceinline__ void finish_dot(double dot, double* __restrict__ part, unsigned* __restrict__ arrived, MpState* __restrict__ st,
                                           double dot0 = 0) {
  __shared__ double sh[32];
  __shared__ bool last;
  const int id = blockIdx.y * gridDim.x + blockIdx.x, nparts = gridDim.x * gridDim.y;
  const double mine = block_sum(dot, sh);
  double mine0 = 0;
  if (WATCH) {
    __syncthreads();  // (sh is read by the first sum's warp)
    mine0 = block_sum(dot0, sh);
  }
  if (threadIdx.x == 0) {
    part[id] = mine;
    if (WATCH) part[nparts + id] = mine0;
    __threadfence();
    last = atomicAdd(arrived, 1u) == (unsigned)nparts - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v = 0, v0 = 0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
    v += __ldcg(part + i);
    if (WATCH) v0 += __ldcg(part + nparts + i);
  }
  __syncthreads();  // (sh is read by the first sum's warp)
  const double s = block_sum(v, sh);
  double s0 = 0;
  if (WATCH) {
    __syncthreads();
    s0 = block_sum(v0, sh);
  }
  if (threadIdx.x != 0) return;
  *arrived = 0;
  if (OP == R_BB) {
    st->bb = s; st->tol2bb = st->tolerance * st->tolerance * s; st->rr = st->keepRR ? s : 0; st->k = 0;
    if (!(s > 0)) st->done = ZERO;
  } else if (OP == R_RR0) {  // the first guess's residual: the first top-of-loop test
    if (st->maxIt > 0) { st->rr = s; if (s <= st->tol2bb) st->done = STOP; }
  } else if (OP == R_RZ0) {
    st->rz = st->rz0 = s;
    if (st->maxIt <= 0 || (st->keepRR && !(st->rr > st->tol2bb))) st->done |= STOP;
  } else if (OP == R_DSD) {
    if (!(s > 0)) st->done = STOP;
    else st->alpha = st->rz / s;
  } else if (OP == R_RR) {
    // The update's residual and the next iteration's top-of-loop test: what follows the update in this iteration changes
    // no result, so a solve that passes stops here and counts it. The faces keep the last update's residual (:137), the
    // projection the last one tested (:314).
    if (st->keepRR) {
      st->rr = s;
      if (!(s > st->tol2bb)) { st->k++; st->done = STOP; }
    } else if (st->k + 1 < st->maxIt) {
      st->rr = s;
      if (s <= st->tol2bb) { st->k++; st->done = STOP; }
    }
  } else {
    st->beta = s / st->rz; st->rz = s; st->k++;
    if (st->k >= st->maxIt) st->done = STOP;
    if (WATCH && s0 * s0 > st->watch * st->rz0 * fmax(s, 1e-10 * st->rz0)) st->done = DRIFT;
  }
}

// The operator works on column fluxes: for every column and cell layer k, with the shares A = rho0 low / 4 of the node
// below (0 when solid) and B = rho0 (high + low of a solid node) / 4 of the one above, fu = A u_k + B u_(k+1), fv alike,
// fw = rho0 w / 4 at k + 1 less that at k; a cell's divergence is the difference of its four columns' fluxes. The
// gradient of a cell vector, over the node masses, is formed a column at a time from the same shares (the operator's
// adjoint), so one march up the column makes S d's fluxes without a pass over node velocities: 26 FP64 instructions a
// layer here and 13 a cell in k_mp_div, against 59 with the nodes between and some 340 with the divides they replace.
// Each thread marches `seg` layers of one column. DIR: of the new direction z + beta d, which it also writes.
template <bool DIR>
__global__ void __launch_bounds__(TPB) k_mp_flux(const double* __restrict__ d, const double* __restrict__ z, double* __restrict__ dn,
                                                 double* __restrict__ fu, double* __restrict__ fv, double* __restrict__ fw, Geo g, int seg,
                                                 const MpState* __restrict__ st, int skip) {
  if (st->done & skip) return;
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= g.layer) return;
  const int j = col / g.nx, x = col - j * g.nx, j0 = j * g.nx, jm = (j == 0 ? g.ny - 1 : j - 1) * g.nx, xm = x == 0 ? g.nx - 1 : x - 1;
  const int k0 = blockIdx.y * seg, k1 = min(g.nc, k0 + seg);
  const double beta = DIR ? st->beta : 0;
  struct Layer { double u, v, w; };  // of one cell layer: the x and y differences and the sum over h of the node's four cells
  auto layer_of = [&](int k) {
    Layer L{0, 0, 0};
    if (k < 0 || k >= g.nc) return L;
    const size_t l = (size_t)k * g.layer;
    double a = d[xm + jm + l], b = d[x + jm + l], c = d[xm + j0 + l], e = d[col + l];
    if (DIR) {
      a = fma(beta, a, z[xm + jm + l]); b = fma(beta, b, z[x + jm + l]); c = fma(beta, c, z[xm + j0 + l]); e = fma(beta, e, z[col + l]);
      if (k >= k0 && k < k1) dn[col + l] = e;
    }
    const double ab = a + b, ce = c + e;
    L.u = (a + c) - (b + e); L.v = ab - ce; L.w = (ab + ce) * g.idz[k];
    return L;
  };
  auto share_a = [&](int k) { return k >= 0 && k < g.nc ? g.A[col + (size_t)k * g.layer] : 0.0; };
  auto share_b = [&](int k) { return k >= 0 && k < g.nc ? g.B[col + (size_t)k * g.layer] : 0.0; };
  struct Vel { double u, v, w; };
  auto node = [&](int k, const Layer& below, const Layer& here, double b, double a) {
    const size_t i = col + (size_t)k * g.layer;
    const double m = g.invMass[i];
    return Vel{fma(a, here.u, b * below.u) * m, fma(a, here.v, b * below.v) * m, (below.w - here.w) * g.wMass[i]};
  };
  Layer L0 = layer_of(k0 - 1), L1 = layer_of(k0);
  double a = share_a(k0);
  Vel lo = node(k0, L0, L1, share_b(k0 - 1), a);
  for (int k = k0; k < k1; k++) {
    const Layer L2 = layer_of(k + 1);
    const double b = share_b(k), an = share_a(k + 1);
    const Vel hi = node(k + 1, L1, L2, b, an);
    const size_t c = col + (size_t)k * g.layer;
    fu[c] = fma(a, lo.u, b * hi.u);
    fv[c] = fma(a, lo.v, b * hi.v);
    fw[c] = fma(g.rho4[k + 1], hi.w, -(g.rho4[k] * lo.w));
    lo = hi; a = an; L1 = L2;
  }
}

// The column fluxes of the node winds (divergencePart, :240-264). Where a column has no open share of the layer the winds
// are not read: what the arrays hold under the ground stays out, numbers or not.
__global__ void __launch_bounds__(TPB) k_mp_wind_flux(const float* __restrict__ u, const float* __restrict__ v, const float* __restrict__ w,
                                                      double* __restrict__ fu, double* __restrict__ fv, double* __restrict__ fw, Geo g) {
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.cells) return;
  const int k = (int)(c / g.layer);
  const size_t up = c + g.layer;
  const double a = g.A[c], b = g.B[c];
  const bool open = b > 0;
  fu[c] = open ? a * (double)u[c] + b * (double)u[up] : 0;
  fv[c] = open ? a * (double)v[c] + b * (double)v[up] : 0;
  fw[c] = g.rho4[k + 1] * (double)w[up] - g.rho4[k] * (double)w[c];
}

// Every cell's divergence from its four columns' fluxes, with sx and sy for 1 / dx and 1 / dy (their squares for S d: the
// gradient's own is applied here). DOT 1: with the sum of out . with; 2: of out . out.
template <int DOT>
__global__ void __launch_bounds__(TPB) k_mp_div(const double* __restrict__ fu, const double* __restrict__ fv, const double* __restrict__ fw,
                                                double* __restrict__ out, const double* __restrict__ with, double sx, double sy,
                                                double* __restrict__ part, unsigned* __restrict__ arrived, Geo g, MpState* __restrict__ st, int skip) {
  if (st && (st->done & skip)) return;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double dot = 0;
  if (c < g.cells) {
    double val = 0;
    if (!g.dropped[c]) {
      const int k = (int)(c / g.layer), rem = (int)(c - (size_t)k * g.layer), j = rem / g.nx, i = rem - j * g.nx;
      const int i1 = i + 1 == g.nx ? 0 : i + 1, j0 = j * g.nx, j1 = (j + 1 == g.ny ? 0 : j + 1) * g.nx;
      const size_t l = (size_t)k * g.layer, p = i + j0 + l, q = i1 + j0 + l, r = i + j1 + l, s = i1 + j1 + l;
      const double ddx = (fu[q] + fu[s]) - (fu[p] + fu[r]), ddy = (fv[r] + fv[s]) - (fv[p] + fv[q]), ddz = (fw[p] + fw[q]) + (fw[r] + fw[s]);
      val = fma(ddx, sx, fma(ddy, sy, ddz * g.idz[k]));
    }
    out[c] = val;
    if (DOT == 1) dot = val * with[c];
    if (DOT == 2) dot = val * val;
  }
  if (DOT == 1) finish_dot<R_DSD>(dot, part, arrived, st);
  if (DOT == 2) finish_dot<R_BB>(dot, part, arrived, st);
}

// What the iterations here take from the reference's tables, once a plan: the sweep's 1 / pivot (with the transforms'
// factor) and lower / pivot, zero for the modes with an infinite pivot (which are left with a pivot of 1 and its
// reciprocal of 0: OrderedSolve), the columns' shares of the fluxes, zero where a layer's upper half is shut, and the nodes' weights of w.
__global__ void k_mp_tables(double* __restrict__ piv, double* __restrict__ rpiv, const double* __restrict__ lo, double* __restrict__ a,
                            double* __restrict__ b, double factor, size_t spec, const double* __restrict__ low, const double* __restrict__ high,
                            double* __restrict__ A, double* __restrict__ B, double* __restrict__ wMass, Geo g) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < spec) {
    const double p = piv[i], ip = isinf(p) ? 0 : 1 / p;
    if (ip == 0) piv[i] = 1;
    rpiv[i] = ip; a[i] = factor * ip; b[i] = lo[i] * ip;
  }
  if (i < g.cells) {
    const int k = (int)(i / g.layer);
    const double lw = low[i], hi = high[i];
    const bool solid = g.solid[i] != 0;
    A[i] = hi > 0 && !solid ? g.rho4[k] * lw : 0;
    B[i] = hi > 0 ? g.rho4[k + 1] * (hi + (solid ? lw : 0)) : 0;
  }
  if (i < g.n) wMass[i] = g.wall[i] || i < (size_t)g.layer || i >= g.n - g.layer ? 0 : g.rho4[i / g.layer] * g.invMass[i];
}

// The first guess q = V phi from the last pressure (:311).
__global__ void k_mp_start(const double* __restrict__ p, double* __restrict__ q, double dt, Geo g, const MpState* __restrict__ st) {
  if (st->done & ZERO) return;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < g.cells) q[c] = g.dropped[c] ? 0 : p[c] * dt * g.dzs[c / g.layer];
}

// r = -b - S q with its square (:313).
__global__ void __launch_bounds__(TPB) k_mp_resid(const double* __restrict__ b, const double* __restrict__ sq, double* __restrict__ r,
                                                  double* __restrict__ part, unsigned* __restrict__ arrived, Geo g, MpState* __restrict__ st) {
  if (st->done & ZERO) return;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0;
  if (c < g.cells) { v = -b[c] - sq[c]; r[c] = v; }
  finish_dot<R_RR0>(v * v, part, arrived, st);
}

// q += alpha d, r -= alpha S d and the new residual's square (:324), with the preconditioner's x-transform of the new r:
// the rows of a block's group are updated on their way into shared memory.
__global__ void k_mp_update_xfwd(double* __restrict__ q, double* __restrict__ r, const double* __restrict__ d, const double* __restrict__ sd,
                                 double2* __restrict__ S, int nx, int ny, int pairs, Fft64 P, const double2* __restrict__ tw,
                                 double* __restrict__ part, unsigned* __restrict__ arrived, MpState* __restrict__ st) {
  extern __shared__ double2 z64[];
  if (st->done) return;
  const double alpha = st->alpha;
  const int k = blockIdx.y, y0 = blockIdx.x * 2 * pairs, rows = min(2 * pairs, ny - y0);
  const size_t base = (size_t)k * nx * ny + (size_t)y0 * nx;
  double rr = 0;
  for (int e = threadIdx.x; e < (rows + (rows & 1)) * nx; e += blockDim.x) {
    const int row = e / nx, x = e - row * nx;
    double v = 0;
    if (row < rows) {
      q[base + e] = fma(alpha, d[base + e], q[base + e]);
      v = fma(-alpha, sd[base + e], r[base + e]);
      r[base + e] = v;
      rr = fma(v, v, rr);
    }
    reinterpret_cast<double*>(&z64[(row >> 1) * nx + x])[row & 1] = v;
  }
  __syncthreads();
  const double2* Z = fft64_rows(z64, z64 + pairs * nx, (rows + 1) / 2, P, tw);
  fft64_unpack(Z, S, nx, ny, y0, rows, k);
  finish_dot<R_RR>(rr, part, arrived, st);
}

// The preconditioner's x inverse: z = the plain solution (the face solve's), or with dzs V phi, zero in the dropped cells
// (:355), and the sum r . z (OP: what it is for).
//
// WATCH: with r . z0, z0 the first z, which conjugate gradients keep at zero. Rounding makes it grow (over ground that
// leaves a column a small open share of a layer, by a factor of ten in some iterations), and what it has grown to says how
// far rounding has come to decide the iterations (Paige 1976). Over 220 solves on drawn grounds and grids, again with a
// first guess of 1e-16 of the pressure: the 120 with |r . z0| below 1e-9 of sqrt(r.z r0.z0) throughout agreed to 3e-10, half
// of them to 1e-14, and as well with the ordered solve; of the 100 others nine in ten agreed to no better than 9e-10, half to
// no better than 1e-7, the worst to 5e-3 (profiles/masked_projection_routes.md). A solve that passes 1e-9 (or 1e-14 r0.z0, which
// r.z alone would be compared with at tighter tolerances) stops, and starts again in one fixed order of operations
// (OrderedSolve). An iteration there takes 0.39 ms on 80 x 64 x 50 nodes, 0.13 here.
template <int OP, bool WATCH = false>
__global__ void k_mp_xinv(const double2* __restrict__ S, double* __restrict__ out, const double* __restrict__ r, int nx, int ny, int pairs, Fft64 P,
                          const double2* __restrict__ tw, const double* __restrict__ dzs, const uint8_t* __restrict__ dropped,
                          double* __restrict__ part, unsigned* __restrict__ arrived, MpState* __restrict__ st, int skip,
                          const double* __restrict__ z0 = nullptr) {
  extern __shared__ double2 z64[];
  if (st->done & skip) return;
  const int k = blockIdx.y, y0 = blockIdx.x * 2 * pairs, rows = min(2 * pairs, ny - y0);
  fft64_pack(S, z64, nx, ny, y0, rows, k);
  __syncthreads();
  const double2* Z = fft64_rows(z64, z64 + pairs * nx, (rows + 1) / 2, P, tw);
  const size_t base = (size_t)k * nx * ny + (size_t)y0 * nx;
  const double h = dzs ? dzs[k] : 1;
  double dot = 0, dot0 = 0;
  for (int e = threadIdx.x; e < rows * nx; e += blockDim.x) {
    const int row = e / nx, x = e - row * nx;
    const double2 v = Z[(row >> 1) * nx + x];
    double val = row & 1 ? -v.y : v.x;
    if (dzs) val = dropped[base + e] ? 0 : val * h;
    const double re = r[base + e];
    dot = fma(re, val, dot);
    if (WATCH) dot0 = fma(re, z0[base + e], dot0);
    out[base + e] = val;
  }
  finish_dot<OP, WATCH>(dot, part, arrived, st, dot0);
}

// The potential phi = q / V and the pressure kept, phi / dt (:332).
__global__ void k_mp_finish(const double* __restrict__ q, double* __restrict__ p, double dt, Geo g, const MpState* __restrict__ st) {
  if (st->done & ZERO) return;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < g.cells) p[c] = q[c] / g.dzs[c / g.layer] / dt;
}

// u = M (u* - G phi) (gradientPart :270-300 of q = V phi at each node): the correction added in FP32 stores, then masked
// (:334-336).
__global__ void __launch_bounds__(TPB) k_mp_correct(float* __restrict__ u, float* __restrict__ v, float* __restrict__ w, const double* __restrict__ q,
                                                    Geo g, const MpState* __restrict__ st) {
  if (st->done & ZERO) return;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  if (g.solid[i]) { u[i] = 0; v[i] = 0; w[i] = 0; return; }
  const int k = (int)(i / g.layer), col = (int)(i - (size_t)k * g.layer), j = col / g.nx, x = col - j * g.nx;
  const int xm = x == 0 ? g.nx - 1 : x - 1, jm = (j == 0 ? g.ny - 1 : j - 1) * g.nx, j0 = j * g.nx;
  double gu = 0, gv = 0, gw = 0;
  for (int side = 0; side < 2; side++) {  // the layer above the node, then the one below
    const int kc = k - side;
    if (kc < 0 || kc >= g.nc) continue;
    const size_t l = (size_t)kc * g.layer;
    const double a = q[xm + jm + l], b = q[x + jm + l], c = q[xm + j0 + l], d = q[x + j0 + l];
    const double f = side ? g.B[col + l] : g.A[col + l], ab = a + b, cd = c + d, s = (ab + cd) * g.idz[kc];
    gu = fma(f, (a + c) - (b + d), gu); gv = fma(f, ab - cd, gv); gw += side ? s : -s;
  }
  const double m = g.invMass[i];
  u[i] = (float)((double)u[i] + gu * m / g.dx);
  v[i] = (float)((double)v[i] + gv * m / g.dy);
  const float wn = (float)((double)w[i] + gw * g.wMass[i]);
  w[i] = g.wall[i] || i < (size_t)g.layer || i >= g.n - g.layer ? 0.0f : wn;
}

// Flat ground (:336-339): PressureSolver.divergence (pressure.ts:50-66), per unit time dt.
__global__ void k_mp_flat_div(const float* __restrict__ u, const float* __restrict__ v, const float* __restrict__ w, double* __restrict__ out,
                              double dt, Geo g) {
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.cells) return;
  const int k = (int)(c / g.layer), rem = (int)(c - (size_t)k * g.layer), j = rem / g.nx, i = rem - j * g.nx;
  const int i1 = i + 1 == g.nx ? 0 : i + 1, y0 = j * g.nx, y1 = (j + 1 == g.ny ? 0 : j + 1) * g.nx;
  const size_t l0 = (size_t)k * g.layer, l1 = l0 + g.layer;
  const size_t a = i + y0 + l0, b = i1 + y0 + l0, e = i + y1 + l0, f = i1 + y1 + l0, gg = i + y0 + l1, h = i1 + y0 + l1, s = i + y1 + l1,
               t = i1 + y1 + l1;
  const double r0 = g.rho[k] / 4, r1 = g.rho[k + 1] / 4;
  const double ddx = (r0 * ((double)u[b] + (double)u[f] - (double)u[a] - (double)u[e]) + r1 * ((double)u[h] + (double)u[t] - (double)u[gg] - (double)u[s])) / g.dx;
  const double ddy = (r0 * ((double)v[e] + (double)v[f] - (double)v[a] - (double)v[b]) + r1 * ((double)v[s] + (double)v[t] - (double)v[gg] - (double)v[h])) / g.dy;
  const double ddz = (r1 * ((double)w[gg] + (double)w[h] + (double)w[s] + (double)w[t]) - r0 * ((double)w[a] + (double)w[b] + (double)w[e] + (double)w[f])) / g.dzs[k];
  out[c] = (ddx + ddy + ddz) / dt;
}

// PressureSolver.correct (pressure.ts:69-92): u -= dt G p; w only at the interior levels.
__global__ void k_mp_flat_correct(const double* __restrict__ p, float* __restrict__ u, float* __restrict__ v, float* __restrict__ w, double dt, Geo g) {
  const size_t node = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= g.n) return;
  const int k = (int)(node / g.layer), rem = (int)(node - (size_t)k * g.layer), j = rem / g.nx, i = rem - j * g.nx, nz = g.nz;
  const int im = i == 0 ? g.nx - 1 : i - 1, jm = (j == 0 ? g.ny - 1 : j - 1) * g.nx, j0 = j * g.nx;
  const size_t lo = (size_t)(k > 0 ? k - 1 : 0) * g.layer, hi = (size_t)(k < nz - 2 ? k : nz - 2) * g.layer;
  const double wLo = k > 0 ? g.dzs[k - 1] / g.hz[k] : 0, wHi = k < nz - 1 ? g.dzs[k] / g.hz[k] : 0;
  auto P = [&](int ii, int jj, size_t base) { return p[base + ii + jj]; };
  const double gx = (wLo * (P(i, jm, lo) + P(i, j0, lo) - P(im, jm, lo) - P(im, j0, lo)) + wHi * (P(i, jm, hi) + P(i, j0, hi) - P(im, jm, hi) - P(im, j0, hi))) / (4 * g.dx);
  const double gy = (wLo * (P(im, j0, lo) + P(i, j0, lo) - P(im, jm, lo) - P(i, jm, lo)) + wHi * (P(im, j0, hi) + P(i, j0, hi) - P(im, jm, hi) - P(i, jm, hi))) / (4 * g.dy);
  u[node] = (float)((double)u[node] - dt * gx);
  v[node] = (float)((double)v[node] - dt * gy);
  if (k > 0 && k < nz - 1) {
    const size_t below = (size_t)(k - 1) * g.layer, above = (size_t)k * g.layer;
    const double gz = (P(im, jm, above) + P(i, jm, above) + P(im, j0, above) + P(i, j0, above) - P(im, jm, below) - P(i, jm, below) - P(im, j0, below) -
                       P(i, j0, below)) / (4 * g.hz[k]);
    w[node] = (float)((double)w[node] - dt * gz);
  }
}

// ---------------------------------------------------------------- the transport's faces with terrain
// (FluxTransport.setTerrain and setVelocityMasked, src/core/advection.ts:78-184): node vectors [n].

struct FaceGeo {
  const uint8_t* open;  // bit 1 the face to x + 1, 2 to y + 1, 4 to z + 1: both nodes fluid
  const double *ax, *ay, *hn, *rho, *dzs, *cx, *cy, *cz;
  int nx, ny, nz, layer;
  size_t n;
  double dx, dy;
};

struct Node {
  int x, y, z;
  size_t l, e, w, no, so;
};
__device__ __forceinline__ Node node_of(size_t i, const FaceGeo& g) {
  Node a;
  a.z = (int)(i / g.layer);
  const int rem = (int)(i - (size_t)a.z * g.layer);
  a.y = rem / g.nx; a.x = rem - a.y * g.nx;
  a.l = (size_t)a.z * g.layer;
  a.e = (size_t)(a.x + 1 == g.nx ? 0 : a.x + 1) + (size_t)a.y * g.nx + a.l;
  a.w = (size_t)(a.x == 0 ? g.nx - 1 : a.x - 1) + (size_t)a.y * g.nx + a.l;
  a.no = (size_t)a.x + (size_t)(a.y + 1 == g.ny ? 0 : a.y + 1) * g.nx + a.l;
  a.so = (size_t)a.x + (size_t)(a.y == 0 ? g.ny - 1 : a.y - 1) * g.nx + a.l;
  return a;
}

// faces (advection.ts:190-200) of the node velocity, shut where a face is not open (:120).
__global__ void k_tm_faces(const float* __restrict__ u, const float* __restrict__ v, const float* __restrict__ w, double* __restrict__ mx,
                           double* __restrict__ my, double* __restrict__ mz, FaceGeo g) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  const Node a = node_of(i, g);
  const uint8_t o = g.open[i];
  const double r = g.rho[a.z];
  mx[i] = o & 1 ? r * ((double)u[i] + (double)u[a.e]) / 2 : 0;
  my[i] = o & 2 ? r * ((double)v[i] + (double)v[a.no]) / 2 : 0;
  mz[i] = o & 4 ? (g.rho[a.z] + g.rho[a.z + 1]) / 2 * ((double)w[i] + (double)w[i + g.layer]) / 2 : 0;
}

// The apertures' divergence of the face fluxes (:96-105): MODE 0 b = -(h div) with its square, 1 div = h div / hn.
template <int MODE>
__global__ void __launch_bounds__(TPB) k_tm_tdiv(const double* __restrict__ mx, const double* __restrict__ my, const double* __restrict__ mz,
                                                 double* __restrict__ out, double* __restrict__ part, unsigned* __restrict__ arrived, FaceGeo g,
                                                 MpState* __restrict__ st) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double dot = 0;
  if (i < g.n) {
    const Node a = node_of(i, g);
    double v = (g.ax[i] * mx[i] - g.ax[a.w] * mx[a.w]) / g.dx + (g.ay[i] * my[i] - g.ay[a.so] * my[a.so]) / g.dy +
               (mz[i] - (a.z > 0 ? mz[i - g.layer] : 0));
    if (MODE == 0) { v = -v; dot = v * v; }
    else v = v / g.hn[i];
    out[i] = v;
  }
  if (MODE == 0) finish_dot<R_BB>(dot, part, arrived, st);
}

// S d = -h div(M rho0 grad d) (:170-176) at each node, d the new direction z + beta d formed at the node and its six
// neighbours, with the sum d . S d: six differences times the faces' coefficients (cx = rho0 ax / dx^2 of an open face to
// x + 1, cy alike, cz = rho0 / dzs to z + 1, zero when shut).
__global__ void __launch_bounds__(TPB) k_tm_apply(const double* __restrict__ d, const double* __restrict__ z, double* __restrict__ dn, double* __restrict__ out,
                                                  double* __restrict__ part, unsigned* __restrict__ arrived, FaceGeo g, MpState* __restrict__ st) {
  if (st->done) return;
  const double beta = st->beta;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double dot = 0;
  if (i < g.n) {
    const Node a = node_of(i, g);
    auto dir = [&](size_t at) { return fma(beta, d[at], z[at]); };
    const double di = dir(i);
    dn[i] = di;
    double v = g.cx[i] * (di - dir(a.e));
    v = fma(g.cx[a.w], di - dir(a.w), v);
    v = fma(g.cy[i], di - dir(a.no), v);
    v = fma(g.cy[a.so], di - dir(a.so), v);
    if (a.z + 1 < g.nz) v = fma(g.cz[i], di - dir(i + g.layer), v);
    if (a.z > 0) v = fma(g.cz[i - g.layer], di - dir(i - g.layer), v);
    out[i] = v;
    dot = di * v;
  }
  finish_dot<R_DSD>(dot, part, arrived, st);
}

// The fluxes lose M rho0 grad(q) (:150).
__global__ void k_tm_correct(const double* __restrict__ q, double* __restrict__ mx, double* __restrict__ my, double* __restrict__ mz, FaceGeo g,
                             const MpState* __restrict__ st) {
  if (st->done & ZERO) return;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  const Node a = node_of(i, g);
  const uint8_t o = g.open[i];
  const double r = g.rho[a.z], qi = q[i];
  mx[i] += o & 1 ? -r * (q[a.e] - qi) / g.dx : 0;
  my[i] += o & 2 ? -r * (q[a.no] - qi) / g.dy : 0;
  mz[i] += o & 4 ? -((g.rho[a.z] + g.rho[a.z + 1]) / 2) * (q[i + g.layer] - qi) / g.dzs[a.z] : 0;
}

int blocks(size_t count) { return (int)((count + TPB - 1) / TPB); }
// Shared memory beyond 48 KB for rows of more than 1536 points.
cudaError_t solve_limits() {
  cudaError_t e = spectral64_limits();
  for (const void* k : {(const void*)k_mp_update_xfwd, (const void*)k_mp_xinv<R_RZ0>, (const void*)k_mp_xinv<R_RZN>, (const void*)k_mp_xinv<R_RZN, true>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SPECTRAL64_SMEM);
  return e;
}
// Layers a thread of k_mp_flux marches: two layers' work is its start, so as many as leave the chip's 152 SMs four blocks
// of 64 columns each, within 4..16.
int flux_seg(int layer, int nc) { return std::min(16, std::max(4, (int)((size_t)layer * nc / (152 * (size_t)TPB)))); }

}  // namespace

struct sg_masked {
  sg_context* ctx = nullptr;
  HostGrid hg{};
  Geo geo{};
  int maxIt = 200;
  double tolerance = 1e-6;
  bool any = false;
  char* mem = nullptr;
  float *u = nullptr, *v = nullptr, *w = nullptr;
  double *p = nullptr, *b = nullptr, *q = nullptr, *r = nullptr, *z = nullptr, *d[2] = {}, *sd = nullptr, *fu = nullptr, *fv = nullptr,
         *fw = nullptr, *z0 = nullptr, *part = nullptr;
  unsigned* arrived = nullptr;
  Spectral64 sp;
  OrderedSolve ordered{};
  MpState* st = nullptr;
  std::vector<uint8_t> dropped;
  cudaGraphExec_t chunk = nullptr, orderedChunk = nullptr;
  int force = 0, route = 0;  // sg_debug_masked_route
  int iterations = 0;
  double residual = 0;
};

struct sg_faces {
  sg_context* ctx = nullptr;
  FaceGeo fg{};
  int maxIt = 400;
  double tolerance = 1e-10;
  char* mem = nullptr;
  float *u = nullptr, *v = nullptr, *w = nullptr;
  double *mx = nullptr, *my = nullptr, *mz = nullptr, *div = nullptr, *q = nullptr, *r = nullptr, *z = nullptr, *d[2] = {},
         *sd = nullptr, *part = nullptr;
  unsigned* arrived = nullptr;
  Spectral64 sp;
  MpState* st = nullptr;
  cudaGraphExec_t chunk = nullptr;
  int iterations = 0;
  double residual = 0;
};

namespace {

constexpr int REPLAY = 8;

// The preconditioner's x-inverse into z with r . z, on the shape of a solve.
template <int OP, bool WATCH = false>
void enqueue_xinv(const Spectral64& S, double* z, const double* r, const double* dzs, const uint8_t* dropped, double* part, unsigned* arrived,
                  MpState* st, int skip, cudaStream_t s, const double* z0 = nullptr) {
  k_mp_xinv<OP, WATCH><<<dim3(S.x.groups, S.levels), S.x.threads, S.x.smem, s>>>(S.S, z, r, S.nx, S.ny, S.x.pairs, S.px, S.twx, dzs, dropped, part, arrived, st, skip, z0);
}
// The preconditioner after the x-transform of r: the flat solve of -r (:351-356; the face solve's flatSolve,
// advection.ts:179-184, whose right-hand side over and back times each level's height is -r too).
template <int OP, bool WATCH = false>
void enqueue_precondition(const Spectral64& S, double* z, const double* r, const double* dzs, const uint8_t* dropped, double* part, unsigned* arrived,
                          MpState* st, int skip, cudaStream_t s, const double* z0 = nullptr) {
  S.forward_y(s, &st->done, skip);
  S.sweep(s, 1, &st->done, skip);
  S.inverse_y(s, &st->done, skip);
  enqueue_xinv<OP, WATCH>(S, z, r, dzs, dropped, part, arrived, st, skip, s, z0);
}
// The start's: the x-transform of r as it stands, then the same.
void enqueue_first_precondition(const Spectral64& S, double* z, const double* r, const double* dzs, const uint8_t* dropped, double* part,
                                unsigned* arrived, MpState* st, cudaStream_t s) {
  S.forward_x(r, s, &st->done, ANY);
  enqueue_precondition<R_RZ0>(S, z, r, dzs, dropped, part, arrived, st, ANY, s);
}
// The end of an iteration from S d on: the update with its x-transform, the preconditioner (WATCH: with its watch on z0).
template <bool WATCH>
void enqueue_descent(const Spectral64& S, double* q, double* r, double* z, const double* d, const double* sd, const double* dzs, const uint8_t* dropped,
                     double* part, unsigned* arrived, MpState* st, cudaStream_t s, const double* z0 = nullptr) {
  k_mp_update_xfwd<<<dim3(S.x.groups, S.levels), S.x.threads, S.x.smem, s>>>(q, r, d, sd, S.S, S.nx, S.ny, S.x.pairs, S.px, S.twx, part, arrived, st);
  enqueue_precondition<R_RZN, WATCH>(S, z, r, dzs, dropped, part, arrived, st, ANY, s, z0);
}

// One iteration of setVelocityMasked's loop (:127-145); `odd`: which of the two direction buffers is the last one's.
void enqueue_face_iteration(sg_faces* f, int odd, cudaStream_t s) {
  double *last = f->d[odd], *next = f->d[odd ^ 1];
  k_tm_apply<<<blocks(f->fg.n), TPB, 0, s>>>(last, f->z, next, f->sd, f->part, f->arrived, f->fg, f->st);
  enqueue_descent<false>(f->sp, f->q, f->r, f->z, next, f->sd, nullptr, nullptr, f->part, f->arrived, f->st, s);
}

// The fluxes of a cell vector's gradient (of z + beta d where dn is given).
void enqueue_flux(sg_masked* m, const double* d, const double* z, double* dn, int skip, cudaStream_t s) {
  const Geo& g = m->geo;
  const int seg = flux_seg(g.layer, g.nc), tpb = 64;
  const dim3 grid((g.layer + tpb - 1) / tpb, (g.nc + seg - 1) / seg);
  if (dn) k_mp_flux<true><<<grid, tpb, 0, s>>>(d, z, dn, m->fu, m->fv, m->fw, g, seg, m->st, skip);
  else k_mp_flux<false><<<grid, tpb, 0, s>>>(d, nullptr, nullptr, m->fu, m->fv, m->fw, g, seg, m->st, skip);
}

// One iteration of the loop (:314-329).
void enqueue_iteration(sg_masked* m, int odd, cudaStream_t s) {
  const Geo& g = m->geo;
  double *last = m->d[odd], *next = m->d[odd ^ 1];
  enqueue_flux(m, last, m->z, next, ANY, s);
  k_mp_div<1><<<blocks(g.cells), TPB, 0, s>>>(m->fu, m->fv, m->fw, m->sd, next, 1 / (g.dx * g.dx), 1 / (g.dy * g.dy), m->part, m->arrived, g, m->st, ANY);
  enqueue_descent<true>(m->sp, m->q, m->r, m->z, next, m->sd, g.dzs, g.dropped, m->part, m->arrived, m->st, s, m->z0);
}

int fail(sg_masked* m, const char* what, cudaError_t e) {
  return sg_context_fail(m->ctx, SG_ERR_DEVICE, (std::string("masked projection: ") + what + ": " + cudaGetErrorString(e)).c_str());
}

}  // namespace

extern "C" {

int sg_terrain_heights(const sg_grid* grid, const sg_terrain* form, float* out) {
  HostGrid g;
  if (!host_grid(grid, g) || !form || !out) return SG_ERR_INVALID;
  if (form->kind < SG_TERRAIN_HILL || form->kind > SG_TERRAIN_SCHAR || !std::isfinite(form->height) || !std::isfinite(form->width)) return SG_ERR_INVALID;
  terrain_heights(g, *form, out);
  return SG_OK;
}

int sg_terrain_geometry(const sg_grid* grid, const float* ground, uint8_t* solid, int32_t* levels, double* heights, double* ax, double* ay,
                        float* slope) {
  HostGrid g;
  if (!host_grid(grid, g) || !ground) return SG_ERR_INVALID;
  std::vector<uint8_t> s(g.n);
  std::vector<int32_t> lv(g.layer);
  solid_levels(g, ground, s.data(), lv.data());
  if (solid) std::memcpy(solid, s.data(), g.n);
  if (levels) std::memcpy(levels, lv.data(), (size_t)g.layer * 4);
  if (heights) node_heights(g, s.data(), lv.data(), ground, heights);
  if (ax && ay) face_apertures(g, s.data(), ground, ax, ay);
  else if (ax || ay) {
    std::vector<double> tx(g.n), ty(g.n);
    face_apertures(g, s.data(), ground, tx.data(), ty.data());
    if (ax) std::memcpy(ax, tx.data(), g.n * 8);
    if (ay) std::memcpy(ay, ty.data(), g.n * 8);
  }
  if (slope) slope_area(g, ground, slope);
  return SG_OK;
}

int sg_masked_create(sg_context* ctx, const sg_grid* grid, const double* rho, const float* ground, double tolerance, int max_iterations,
                     sg_masked** out) {
  if (!ctx || !out) return SG_ERR_INVALID;
  *out = nullptr;
  HostGrid g;
  if (!host_grid(grid, g) || !rho || !ground)
    return sg_context_fail(ctx, SG_ERR_INVALID, "masked projection: a grid with nx, ny >= 1, nz >= 3, dx, dy > 0, its level arrays, rho and the ground");
  if (g.nx > 2048 || g.ny > 2048) return sg_context_fail(ctx, SG_ERR_INVALID, "masked projection: nx and ny at most 2048");
  if (g.n > (size_t)1 << 30) return sg_context_fail(ctx, SG_ERR_INVALID, "masked projection: at most 2^30 nodes");
  if (!(tolerance >= 0) || max_iterations < 0) return sg_context_fail(ctx, SG_ERR_INVALID, "masked projection: tolerance >= 0, max_iterations >= 0");
  for (int k = 0; k < g.nz; k++)
    if (!(g.hz[k] > 0) || (k < g.nz - 1 && !(g.dzs[k] > 0)) || !(rho[k] > 0))
      return sg_context_fail(ctx, SG_ERR_INVALID, "masked projection: level spacings and densities must be positive");
  for (int c = 0; c < g.layer; c++)
    if (!std::isfinite(ground[c])) return sg_context_fail(ctx, SG_ERR_INVALID, "masked projection: finite ground heights");
  if (cudaSetDevice(sg_context_device(ctx)) != cudaSuccess) return sg_context_fail(ctx, SG_ERR_DEVICE, "masked projection: cudaSetDevice");
  const int nx = g.nx, ny = g.ny, nz = g.nz, nc = nz - 1, layer = g.layer, mh = nx / 2, modes = (mh + 1) * ny;
  const size_t n = g.n, cells = (size_t)layer * nc, spec = (size_t)nc * modes;
  Spectral64 sp;
  sp.shape(nx, ny, nc);

  // The constructor (:190-218): solid and wall nodes, 1 / (rho0 hn), the columns' shares of each
  // cell layer (of its half below the middle and above it that are above the ground), dropped cells.
  std::vector<uint8_t> solid(n), wall(n, 0), dropped(cells);
  std::vector<int32_t> levels(layer);
  std::vector<double> heights(n), inv(n, 0.0), low(cells), high(cells), rho4(nz), idz(nz, 0.0);
  solid_levels(g, ground, solid.data(), levels.data());
  node_heights(g, solid.data(), levels.data(), ground, heights.data());
  bool any = false;
  for (size_t i = 0; i < n; i++) any = any || solid[i];
  for (int c = 0; c < layer; c++) any = any || ground[c] > 0;
  for (int k = 0; k < nz; k++) rho4[k] = rho[k] / 4;
  for (int k = 0; k < nc; k++) idz[k] = 1 / g.dzs[k];
  for (int k = 0; k < nz; k++) {
    const double r = rho[k];
    for (int c = 0; c < layer; c++) {
      const size_t i = c + (size_t)k * layer;
      if (solid[i]) continue;
      inv[i] = 1 / (r * heights[i]);
      if (g.zs[k] <= (double)ground[c]) wall[i] = 1;
    }
  }
  for (int k = 0; k < nc; k++) {
    const double half = g.dzs[k] / 2, middle = g.zs[k] + half;
    for (int c = 0; c < layer; c++) {
      const size_t at = c + (size_t)k * layer;
      const double h = (double)ground[c];
      low[at] = std::min(1.0, std::max(0.0, (middle - std::max(h, g.zs[k])) / half));
      high[at] = std::min(1.0, std::max(0.0, (g.zs[k + 1] - std::max(h, middle)) / half));
    }
  }
  for (int k = 0; k < nc; k++)
    for (int j = 0; j < ny; j++) {
      const double *b0 = high.data() + (size_t)k * layer + (size_t)j * nx, *b1 = high.data() + (size_t)k * layer + (size_t)((j + 1) % ny) * nx;
      uint8_t* out = dropped.data() + (size_t)k * layer + (size_t)j * nx;
      for (int i = 0; i < nx; i++) {
        const int i1 = i + 1 == nx ? 0 : i + 1;
        out[i] = b0[i] == 0 && b0[i1] == 0 && b1[i] == 0 && b1[i1] == 0;
      }
    }

  // The flat solve's rows per mode (pressure.ts:36-44, :118-140): lower coefficient, pivot and cp = up / pivot of each
  // cell layer in the reference's elimination order. Modes it zeroes and the uniform mode's pinned lowest cell get an
  // infinite pivot (their values come out zero).
  std::vector<double> tlo(spec, 0.0), tcp(spec, 0.0), tpiv(spec, 0.0);
  std::vector<double> own(nc);
  for (int k = 0; k < nc; k++) own[k] = rho[k] * g.dzs[k] / (2 * g.hz[k]) + rho[k + 1] * g.dzs[k] / (2 * g.hz[k + 1]);
  auto exact = [](double x) { return x < 1e-12 ? 0 : x > 1 - 1e-12 ? 1 : x; };
  for (int m = 0; m <= mh; m++)
    for (int q = 0; q < ny; q++) {
      const double sx = exact(std::pow(std::sin(PI_ * m / nx), 2)), cx = exact(std::pow(std::cos(PI_ * m / nx), 2));
      const double sy = exact(std::pow(std::sin(PI_ * q / ny), 2)), cy = exact(std::pow(std::cos(PI_ * q / ny), 2));
      const double a = 4 * (sx * cy / (g.dx * g.dx) + cx * sy / (g.dy * g.dy)), b = cx * cy;
      const size_t mode = (size_t)m * ny + q;
      if ((a == 0 && b == 0) || (nc == 1 && a == 0)) {
        for (int k = 0; k < nc; k++) tpiv[(size_t)k * modes + mode] = INFINITY;
        continue;
      }
      const bool pinned = a == 0;
      double cprev = 0;
      for (int k = 0; k < nc; k++) {
        double di = -a / 2 * own[k], lo = 0, up = 0;
        if (k > 0) { lo = -a / 2 * rho[k] * g.dzs[k - 1] / (2 * g.hz[k]); const double v = b * rho[k] / (g.hz[k] * g.dzs[k]); lo += v; di -= v; }
        if (k < nc - 1) { up = -a / 2 * rho[k + 1] * g.dzs[k + 1] / (2 * g.hz[k + 1]); const double v = b * rho[k + 1] / (g.hz[k + 1] * g.dzs[k]); up += v; di -= v; }
        bool zero = false;
        if (pinned && k == 0) { lo = 0; di = 1; up = 0; zero = true; }
        if (pinned && k == 1) lo = 0;
        const double piv = k == 0 ? di : di - lo * cprev;
        cprev = up / piv;
        const size_t at = (size_t)k * modes + mode;
        tlo[at] = lo; tcp[at] = cprev; tpiv[at] = zero ? INFINITY : piv;
      }
    }
  std::vector<double2> tx(nx), ty(ny);
  for (int t = 0; t < nx; t++) tx[t] = make_double2(std::cos(2 * PI_ * t / nx), std::sin(2 * PI_ * t / nx));
  for (int t = 0; t < ny; t++) ty[t] = make_double2(std::cos(2 * PI_ * t / ny), std::sin(2 * PI_ * t / ny));

  // One allocation, 256-byte aligned parts.
  auto al = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
  const size_t nparts = std::max({(size_t)blocks(cells), 2 * (size_t)sp.x.groups * nc, (size_t)ny * nc});  // (two sums a group: the watch)
  size_t off = 0;
  auto take = [&](size_t bytes) { const size_t o = off; off += al(bytes); return o; };
  // Some 175 bytes a node, 20 of them the ordered solve's own: its sweep's coefficients and its first spectrum (where the fast
  // one keeps z0); the two share the rest.
  const size_t oU = take(n * 4), oV = take(n * 4), oW = take(n * 4), oP = take(cells * 8), oB = take(cells * 8), oQ = take(cells * 8), oR = take(cells * 8),
               oZ = take(cells * 8), oD = take(cells * 8), oD2 = take(cells * 8), oSd = take(cells * 8), oFu = take(n * 8), oFv = take(n * 8),
               oFw = take(n * 8), oPart = take(nparts * 8), oLo = take(spec * 8), oPv = take(spec * 8),
               oRpv = take(spec * 8), oS1 = take(spec * 16), oLow = oQ, oHigh = oR, oOst = take(sizeof(OrderedState)), oA = take(spec * 8), oBb = take(spec * 8), oC = take(spec * 8), oS = take(spec * 16),
               oTx = take((size_t)nx * 16), oTy = take((size_t)ny * 16), oSt = take(sizeof(MpState)), oArr = take(sizeof(unsigned)), oSol = take(n),
               oWal = take(n), oDr = take(cells), oInv = take(n * 8), oWm = take(n * 8), oSa = take(cells * 8), oSb = take(cells * 8),
               oRho = take((size_t)nz * 8), oR4 = take((size_t)nz * 8), oDz = take((size_t)nz * 8), oIdz = take((size_t)nz * 8), oHz = take((size_t)nz * 8),
               total = off;
  auto* s = new sg_masked;
  s->ctx = ctx; s->hg = g; s->maxIt = max_iterations; s->tolerance = tolerance; s->any = any;
  s->dropped = dropped;
  cudaError_t e = solve_limits();
  if (e != cudaSuccess) { delete s; return sg_context_fail(ctx, SG_ERR_DEVICE, "masked projection: shared memory"); }
  e = cudaMalloc(&s->mem, total);
  if (e != cudaSuccess) { delete s; cudaGetLastError(); return sg_context_fail(ctx, SG_ERR_BUDGET, "masked projection: device memory"); }
  char* M = s->mem;
  s->u = (float*)(M + oU); s->v = (float*)(M + oV); s->w = (float*)(M + oW);
  s->p = (double*)(M + oP); s->b = (double*)(M + oB); s->q = (double*)(M + oQ); s->r = (double*)(M + oR); s->z = (double*)(M + oZ);
  s->d[0] = (double*)(M + oD); s->d[1] = (double*)(M + oD2); s->sd = (double*)(M + oSd); s->fu = (double*)(M + oFu); s->fv = (double*)(M + oFv);
  s->fw = (double*)(M + oFw); s->z0 = (double*)(M + oS1);  // (each of the two routes' own)
  s->part = (double*)(M + oPart); s->arrived = (unsigned*)(M + oArr); s->st = (MpState*)(M + oSt);
  sp.a = (double*)(M + oA); sp.b = (double*)(M + oBb); sp.c = (double*)(M + oC); sp.S = (double2*)(M + oS);
  sp.twx = (double2*)(M + oTx); sp.twy = (double2*)(M + oTy);
  s->sp = sp;
  Geo& G = s->geo;
  G.solid = (const uint8_t*)(M + oSol); G.wall = (const uint8_t*)(M + oWal); G.dropped = (const uint8_t*)(M + oDr);
  G.A = (const double*)(M + oSa); G.B = (const double*)(M + oSb); G.invMass = (const double*)(M + oInv); G.wMass = (const double*)(M + oWm);
  G.rho = (const double*)(M + oRho); G.rho4 = (const double*)(M + oR4); G.dzs = (const double*)(M + oDz); G.idz = (const double*)(M + oIdz);
  G.hz = (const double*)(M + oHz);
  G.nx = nx; G.ny = ny; G.nz = nz; G.layer = layer; G.nc = nc; G.n = n; G.cells = cells; G.dx = g.dx; G.dy = g.dy;
  OrderedSolve& O = s->ordered;
  O.solid = G.solid; O.wall = G.wall; O.dropped = G.dropped; O.A = G.A; O.B = G.B; O.invMass = G.invMass; O.rho4 = G.rho4;
  O.dzs = G.dzs; O.idz = G.idz; O.lo = (const double*)(M + oLo); O.cp = sp.c; O.piv = (const double*)(M + oPv); O.rpiv = (const double*)(M + oRpv);
  O.twx = sp.twx; O.twy = sp.twy;
  O.nx = nx; O.ny = ny; O.nz = nz; O.layer = layer; O.nc = nc; O.mh = mh; O.modes = modes; O.n = n; O.cells = cells;
  O.dx = g.dx; O.dy = g.dy; O.rdx = 1 / g.dx; O.rdy = 1 / g.dy;
  O.b = s->b; O.q = s->q; O.r = s->r; O.z = s->z; O.d = s->d[0]; O.e = s->d[1]; O.sd = s->sd; O.fu = s->fu; O.fv = s->fv; O.fw = s->fw;
  O.part = s->part; O.S1 = (double2*)(M + oS1); O.S2 = sp.S; O.arrived = s->arrived; O.st = (OrderedState*)(M + oOst);
  cudaStream_t st = sg_context_stream(ctx);
  std::vector<double> dz(nz, 0.0);
  std::copy(g.dzs, g.dzs + nz - 1, dz.begin());
  struct Up { size_t off; const void* src; size_t bytes; };
  const Up ups[] = {{oLo, tlo.data(), spec * 8}, {oPv, tpiv.data(), spec * 8}, {oC, tcp.data(), spec * 8}, {oTx, tx.data(), (size_t)nx * 16},
                    {oTy, ty.data(), (size_t)ny * 16}, {oSol, solid.data(), n}, {oWal, wall.data(), n}, {oDr, dropped.data(), cells},
                    {oInv, inv.data(), n * 8}, {oLow, low.data(), cells * 8}, {oHigh, high.data(), cells * 8},
                    {oRho, rho, (size_t)nz * 8}, {oR4, rho4.data(), (size_t)nz * 8}, {oDz, dz.data(), (size_t)nz * 8},
                    {oIdz, idz.data(), (size_t)nz * 8}, {oHz, g.hz, (size_t)nz * 8}};
  for (const Up& up : ups)
    if ((e = cudaMemcpyAsync(M + up.off, up.src, up.bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess) break;
  if (e == cudaSuccess) e = cudaMemsetAsync(s->arrived, 0, sizeof(unsigned), st);
  if (e == cudaSuccess) {
    k_mp_tables<<<blocks(std::max(spec, n)), TPB, 0, st>>>((double*)(M + oPv), (double*)(M + oRpv), O.lo, (double*)(M + oA), (double*)(M + oBb),
                                                               sp.factor(), spec, (const double*)(M + oLow), (const double*)(M + oHigh), (double*)(M + oSa), (double*)(M + oSb), (double*)(M + oWm), G);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaFree(s->mem); delete s;
    return sg_context_fail(ctx, SG_ERR_DEVICE, (std::string("masked projection: ") + cudaGetErrorString(e)).c_str());
  }
  *out = s;
  return SG_OK;
}

int sg_masked_mask(sg_masked* m, float* u, float* v, float* w) {
  if (!m) return SG_ERR_INVALID;
  if (!u || !v || !w) return sg_context_fail(m->ctx, SG_ERR_INVALID, "masked projection: u, v and w buffers");
  cudaSetDevice(sg_context_device(m->ctx));
  cudaStream_t s = sg_context_stream(m->ctx);
  const size_t n = m->geo.n;
  cudaError_t e;
  float* host[3] = {u, v, w};
  float* dev[3] = {m->u, m->v, m->w};
  for (int f = 0; f < 3; f++)
    if ((e = cudaMemcpyAsync(dev[f], host[f], n * 4, cudaMemcpyHostToDevice, s)) != cudaSuccess) return fail(m, "copy in", e);
  k_mp_mask<<<blocks(n), TPB, 0, s>>>(m->u, m->v, m->w, m->geo);
  for (int f = 0; f < 3; f++)
    if ((e = cudaMemcpyAsync(host[f], dev[f], n * 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return fail(m, "copy out", e);
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess) return fail(m, "mask", e);
  return SG_OK;
}

int sg_masked_divergence(sg_masked* m, const float* u, const float* v, const float* w, double* out) {
  if (!m) return SG_ERR_INVALID;
  if (!u || !v || !w || !out) return sg_context_fail(m->ctx, SG_ERR_INVALID, "masked projection: u, v, w and out buffers");
  cudaSetDevice(sg_context_device(m->ctx));
  cudaStream_t s = sg_context_stream(m->ctx);
  const size_t n = m->geo.n, cells = m->geo.cells;
  cudaError_t e;
  const float* host[3] = {u, v, w};
  float* dev[3] = {m->u, m->v, m->w};
  for (int f = 0; f < 3; f++)
    if ((e = cudaMemcpyAsync(dev[f], host[f], n * 4, cudaMemcpyHostToDevice, s)) != cudaSuccess) return fail(m, "copy in", e);
  k_mp_wind_flux<<<blocks(cells), TPB, 0, s>>>(m->u, m->v, m->w, m->fu, m->fv, m->fw, m->geo);
  k_mp_div<0><<<blocks(cells), TPB, 0, s>>>(m->fu, m->fv, m->fw, m->b, nullptr, 1 / m->geo.dx, 1 / m->geo.dy, nullptr, nullptr, m->geo, nullptr, 0);
  if ((e = cudaMemcpyAsync(out, m->b, cells * 8, cudaMemcpyDeviceToHost, s)) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess ||
      (e = cudaGetLastError()) != cudaSuccess)
    return fail(m, "divergence", e);
  return SG_OK;
}

int sg_masked_project(sg_masked* m, float* u, float* v, float* w, double dt, double* pressure) {
  if (!m) return SG_ERR_INVALID;
  if (!u || !v || !w || !pressure) return sg_context_fail(m->ctx, SG_ERR_INVALID, "masked projection: u, v, w and pressure buffers");
  if (!(dt > 0) || !std::isfinite(dt)) return sg_context_fail(m->ctx, SG_ERR_INVALID, "masked projection: dt > 0");
  cudaSetDevice(sg_context_device(m->ctx));
  cudaStream_t s = sg_context_stream(m->ctx);
  const Geo& g = m->geo;
  const size_t n = g.n, cells = g.cells;
  const int nb = blocks(n), cb = blocks(cells);
  cudaError_t e;
  float* host[3] = {u, v, w};
  float* dev[3] = {m->u, m->v, m->w};
  for (int f = 0; f < 3; f++)
    if ((e = cudaMemcpyAsync(dev[f], host[f], n * 4, cudaMemcpyHostToDevice, s)) != cudaSuccess) return fail(m, "copy in", e);
  if ((e = cudaMemcpyAsync(m->p, pressure, cells * 8, cudaMemcpyHostToDevice, s)) != cudaSuccess) return fail(m, "copy in", e);
  k_mp_mask<<<nb, TPB, 0, s>>>(m->u, m->v, m->w, g);
  m->iterations = 0; m->residual = 0; m->route = 0;
  if (!m->any) {
    // No terrain at all: the flat projection exactly (:336-339); the pressure is the flat solve's, not a first guess.
    k_mp_flat_div<<<cb, TPB, 0, s>>>(m->u, m->v, m->w, m->b, dt, g);
    m->sp.solve(m->b, m->p, 0, s);
    k_mp_flat_correct<<<nb, TPB, 0, s>>>(m->p, m->u, m->v, m->w, dt, g);
  } else {
    MpState init{};
    init.tolerance = m->tolerance; init.maxIt = m->maxIt; init.watch = m->force == 1 ? INFINITY : WATCH_LIMIT;
    if ((e = cudaMemcpyAsync(m->st, &init, sizeof(MpState), cudaMemcpyHostToDevice, s)) != cudaSuccess) return fail(m, "state", e);
    if ((e = cudaMemsetAsync(m->d[0], 0, cells * 8, s)) != cudaSuccess) return fail(m, "direction", e);  // (the first direction: z + 0 d)
    // b = D R M u*, bb; q from the first guess, r = -b - S q and its first test, z = P S0^-1 P r, rz (:306-312).
    k_mp_wind_flux<<<cb, TPB, 0, s>>>(m->u, m->v, m->w, m->fu, m->fv, m->fw, g);
    k_mp_div<2><<<cb, TPB, 0, s>>>(m->fu, m->fv, m->fw, m->b, nullptr, 1 / g.dx, 1 / g.dy, m->part, m->arrived, g, m->st, 0);
    k_mp_start<<<cb, TPB, 0, s>>>(m->p, m->q, dt, g, m->st);
    enqueue_flux(m, m->q, nullptr, nullptr, ZERO, s);
    k_mp_div<0><<<cb, TPB, 0, s>>>(m->fu, m->fv, m->fw, m->sd, nullptr, 1 / (g.dx * g.dx), 1 / (g.dy * g.dy), nullptr, nullptr, g, m->st, ZERO);
    k_mp_resid<<<cb, TPB, 0, s>>>(m->b, m->sd, m->r, m->part, m->arrived, g, m->st);
    enqueue_first_precondition(m->sp, m->z, m->r, g.dzs, g.dropped, m->part, m->arrived, m->st, s);
    if ((e = cudaMemcpyAsync(m->z0, m->z, cells * 8, cudaMemcpyDeviceToDevice, s)) != cudaSuccess) return fail(m, "first direction", e);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail(m, "launch", e);
    if (!m->chunk) {
      // Eight iterations as one graph (the buffers are the object's own, so one capture serves every call).
      cudaGraph_t graph = nullptr;
      if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) return fail(m, "capture", e);
      for (int it = 0; it < REPLAY; it++) enqueue_iteration(m, it & 1, s);
      e = cudaStreamEndCapture(s, &graph);
      if (e == cudaSuccess) e = cudaGraphInstantiate(&m->chunk, graph, 0);
      if (graph) cudaGraphDestroy(graph);
      if (e != cudaSuccess) { m->chunk = nullptr; return fail(m, "graph", e); }
    }
    // Every iteration either counts or stops, so maxIt / REPLAY + 1 replays always reach the stop.
    int done = m->force == 2 ? DRIFT : 0;
    for (int c = 0; !done; c++) {
      if ((e = cudaMemcpyAsync(&done, &m->st->done, 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return fail(m, "solve", e);
      if (done || c > m->maxIt / REPLAY + 1) break;
      if ((e = cudaGraphLaunch(m->chunk, s)) != cudaSuccess) return fail(m, "graph launch", e);
    }
    if (!done) return sg_context_fail(m->ctx, SG_ERR_DEVICE, "masked projection: the iterations did not stop");
    m->route = done == DRIFT ? 2 : done == ZERO ? 0 : 1;
    if (done == DRIFT) {
      // The winds and the first guess are still as they were.
      OrderedState fin{};
      if ((e = m->ordered.solve(m->u, m->v, m->w, m->p, dt, m->maxIt, m->tolerance, &m->orderedChunk, &fin, s)) != cudaSuccess) return fail(m, "solve", e);
      if (fin.done != ZERO) { m->iterations = fin.k; m->residual = std::sqrt(fin.rr / fin.bb); }
    } else {
      // u = M (u* - G phi); the pressure kept is phi / dt (:332-336).
      k_mp_finish<<<cb, TPB, 0, s>>>(m->q, m->p, dt, g, m->st);
      k_mp_correct<<<nb, TPB, 0, s>>>(m->u, m->v, m->w, m->q, g, m->st);
      MpState fin{};
      if ((e = cudaMemcpyAsync(&fin, m->st, sizeof(MpState), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return fail(m, "state", e);
      if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail(m, "solve", e);
      if (fin.done != ZERO) { m->iterations = fin.k; m->residual = std::sqrt(fin.rr / fin.bb); }
    }
  }
  for (int f = 0; f < 3; f++)
    if ((e = cudaMemcpyAsync(host[f], dev[f], n * 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return fail(m, "copy out", e);
  if ((e = cudaMemcpyAsync(pressure, m->p, cells * 8, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return fail(m, "copy out", e);
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess) return fail(m, "project", e);
  return SG_OK;
}

int sg_masked_stats(sg_masked* m, int32_t* iterations, double* residual) {
  if (!m) return SG_ERR_INVALID;
  if (iterations) *iterations = m->iterations;
  if (residual) *residual = m->residual;
  return SG_OK;
}

int sg_debug_masked_route(sg_masked* m, int force, int32_t* route) {
  if (!m || force < -1 || force > 2) return SG_ERR_INVALID;
  if (route) *route = m->route;
  if (force >= 0) m->force = force;
  return SG_OK;
}

int sg_masked_dropped(sg_masked* m, uint8_t* dropped) {
  if (!m || !dropped) return SG_ERR_INVALID;
  std::memcpy(dropped, m->dropped.data(), m->dropped.size());
  return SG_OK;
}

int sg_faces_create(sg_context* ctx, const sg_grid* grid, const double* rho, const float* ground, double tolerance, int max_iterations,
                    sg_faces** out) {
  if (!ctx || !out) return SG_ERR_INVALID;
  *out = nullptr;
  HostGrid g;
  if (!host_grid(grid, g) || !rho || !ground)
    return sg_context_fail(ctx, SG_ERR_INVALID, "masked faces: a grid with nx, ny >= 1, nz >= 3, dx, dy > 0, its level arrays, rho and the ground");
  if (g.nx > 2048 || g.ny > 2048) return sg_context_fail(ctx, SG_ERR_INVALID, "masked faces: nx and ny at most 2048");
  if (g.n > (size_t)1 << 30) return sg_context_fail(ctx, SG_ERR_INVALID, "masked faces: at most 2^30 nodes");
  if (!(tolerance >= 0) || max_iterations < 0) return sg_context_fail(ctx, SG_ERR_INVALID, "masked faces: tolerance >= 0, max_iterations >= 0");
  for (int k = 0; k < g.nz; k++)
    if (!(g.hz[k] > 0) || (k < g.nz - 1 && !(g.dzs[k] > 0)) || !(rho[k] > 0))
      return sg_context_fail(ctx, SG_ERR_INVALID, "masked faces: level spacings and densities must be positive");
  for (int c = 0; c < g.layer; c++)
    if (!std::isfinite(ground[c])) return sg_context_fail(ctx, SG_ERR_INVALID, "masked faces: finite ground heights");
  if (cudaSetDevice(sg_context_device(ctx)) != cudaSuccess) return sg_context_fail(ctx, SG_ERR_DEVICE, "masked faces: cudaSetDevice");
  const int nx = g.nx, ny = g.ny, nz = g.nz, layer = g.layer, mh = nx / 2, modes = (mh + 1) * ny;
  const size_t n = g.n, spec = (size_t)nz * modes;
  Spectral64 sp;
  sp.shape(nx, ny, nz);

  // setTerrain (advection.ts:78-90) with the model's geometry (model.ts:366-377): open faces, node heights (1 in the
  // ground), the faces' open heights.
  std::vector<uint8_t> solid(n), open(n, 0);
  std::vector<int32_t> levels(layer);
  std::vector<double> heights(n), hn(n), ax(n), ay(n);
  solid_levels(g, ground, solid.data(), levels.data());
  node_heights(g, solid.data(), levels.data(), ground, heights.data());
  face_apertures(g, solid.data(), ground, ax.data(), ay.data());
  for (size_t i = 0; i < n; i++) hn[i] = solid[i] ? 1 : heights[i];
  for (int z = 0; z < nz; z++)
    for (int y = 0; y < ny; y++)
      for (int x = 0; x < nx; x++) {
        const size_t i = x + (size_t)nx * y + (size_t)layer * z, l = (size_t)layer * z;
        if (solid[i]) continue;
        if (!solid[(x + 1) % nx + (size_t)nx * y + l]) open[i] |= 1;
        if (!solid[x + (size_t)nx * ((y + 1) % ny) + l]) open[i] |= 2;
        if (z < nz - 1 && !solid[i + layer]) open[i] |= 4;
      }

  // The faces' coefficients of S (k_tm_apply).
  std::vector<double> cx(n, 0.0), cy(n, 0.0), cz(n, 0.0);
  for (int z = 0; z < nz; z++) {
    const double rx = rho[z] / (g.dx * g.dx), ry = rho[z] / (g.dy * g.dy), rz = z < nz - 1 ? (rho[z] + rho[z + 1]) / 2 / g.dzs[z] : 0;
    for (size_t i = (size_t)z * layer; i < (size_t)(z + 1) * layer; i++) {
      if (open[i] & 1) cx[i] = rx * ax[i];
      if (open[i] & 2) cy[i] = ry * ay[i];
      if (open[i] & 4) cz[i] = rz;
    }
  }

  // The flat face solve's rows per mode (advection.ts:222-241) as the sweep takes them, each level's in the reference's
  // order (see the projection's above); the uniform mode's lowest level is pinned to zero.
  const double factor = sp.factor();
  std::vector<double> ta(spec, 0.0), tb(spec, 0.0), tcp(spec, 0.0);
  auto face = [&](int k) { return k < 0 || k >= nz - 1 ? 0.0 : (rho[k] + rho[k + 1]) / 2; };
  for (int m = 0; m <= mh; m++)
    for (int q = 0; q < ny; q++) {
      const double lam = m == 0 && q == 0 ? 0
                                          : 4 * std::pow(std::sin(PI_ * m / nx), 2) / (g.dx * g.dx) + 4 * std::pow(std::sin(PI_ * q / ny), 2) / (g.dy * g.dy);
      const bool pinned = lam == 0;
      const size_t mode = (size_t)m * ny + q;
      double cprev = 0;
      for (int k = 0; k < nz; k++) {
        double lo = k > 0 ? face(k - 1) / g.dzs[k - 1] : 0, up = k < nz - 1 ? face(k) / g.dzs[k] : 0, di = -rho[k] * g.hz[k] * lam - lo - up;
        bool zero = false;
        if (pinned && k == 0) { lo = 0; di = 1; up = 0; zero = true; }
        if (pinned && k == 1) lo = 0;
        const double ip = 1 / (k == 0 ? di : di - lo * cprev);
        cprev = up * ip;
        const size_t at = (size_t)k * modes + mode;
        ta[at] = zero ? 0 : factor * ip; tb[at] = zero ? 0 : lo * ip; tcp[at] = cprev;
      }
    }
  std::vector<double2> tx(nx), ty(ny);
  for (int t = 0; t < nx; t++) tx[t] = make_double2(std::cos(2 * PI_ * t / nx), std::sin(2 * PI_ * t / nx));
  for (int t = 0; t < ny; t++) ty[t] = make_double2(std::cos(2 * PI_ * t / ny), std::sin(2 * PI_ * t / ny));

  auto al = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
  const size_t nparts = std::max((size_t)blocks(n), (size_t)sp.x.groups * nz);
  size_t off = 0;
  auto take = [&](size_t bytes) { const size_t o = off; off += al(bytes); return o; };
  const size_t oU = take(n * 4), oV = take(n * 4), oW = take(n * 4), oMx = take(n * 8), oMy = take(n * 8), oMz = take(n * 8), oDiv = take(n * 8),
               oQ = take(n * 8), oR = take(n * 8), oZ = take(n * 8), oD = take(n * 8), oD2 = take(n * 8), oSd = take(n * 8), oPart = take(nparts * 8),
               oA = take(spec * 8), oBb = take(spec * 8), oC = take(spec * 8), oS = take(spec * 16), oTx = take((size_t)nx * 16),
               oTy = take((size_t)ny * 16), oSt = take(sizeof(MpState)), oArr = take(sizeof(unsigned)), oOpen = take(n), oAx = take(n * 8),
               oAy = take(n * 8), oHn = take(n * 8), oCx = take(n * 8), oCy = take(n * 8), oCz = take(n * 8), oRho = take((size_t)nz * 8),
               oDz = take((size_t)nz * 8), total = off;
  auto* f = new sg_faces;
  f->ctx = ctx; f->maxIt = max_iterations; f->tolerance = tolerance;
  cudaError_t e = solve_limits();
  if (e != cudaSuccess) { delete f; return sg_context_fail(ctx, SG_ERR_DEVICE, "masked faces: shared memory"); }
  e = cudaMalloc(&f->mem, total);
  if (e != cudaSuccess) { delete f; cudaGetLastError(); return sg_context_fail(ctx, SG_ERR_BUDGET, "masked faces: device memory"); }
  char* M = f->mem;
  f->u = (float*)(M + oU); f->v = (float*)(M + oV); f->w = (float*)(M + oW);
  f->mx = (double*)(M + oMx); f->my = (double*)(M + oMy); f->mz = (double*)(M + oMz); f->div = (double*)(M + oDiv);
  f->q = (double*)(M + oQ); f->r = (double*)(M + oR); f->z = (double*)(M + oZ); f->d[0] = (double*)(M + oD); f->d[1] = (double*)(M + oD2);
  f->sd = (double*)(M + oSd); f->part = (double*)(M + oPart); f->arrived = (unsigned*)(M + oArr); f->st = (MpState*)(M + oSt);
  sp.a = (double*)(M + oA); sp.b = (double*)(M + oBb); sp.c = (double*)(M + oC); sp.S = (double2*)(M + oS);
  sp.twx = (double2*)(M + oTx); sp.twy = (double2*)(M + oTy);
  f->sp = sp;
  FaceGeo& F = f->fg;
  F.open = (const uint8_t*)(M + oOpen); F.ax = (const double*)(M + oAx); F.ay = (const double*)(M + oAy); F.hn = (const double*)(M + oHn);
  F.cx = (const double*)(M + oCx); F.cy = (const double*)(M + oCy); F.cz = (const double*)(M + oCz);
  F.rho = (const double*)(M + oRho); F.dzs = (const double*)(M + oDz);
  F.nx = nx; F.ny = ny; F.nz = nz; F.layer = layer; F.n = n; F.dx = g.dx; F.dy = g.dy;
  cudaStream_t st = sg_context_stream(ctx);
  std::vector<double> dz(nz, 0.0);
  std::copy(g.dzs, g.dzs + nz - 1, dz.begin());
  struct Up { size_t off; const void* src; size_t bytes; };
  const Up ups[] = {{oA, ta.data(), spec * 8}, {oBb, tb.data(), spec * 8}, {oC, tcp.data(), spec * 8}, {oTx, tx.data(), (size_t)nx * 16},
                    {oTy, ty.data(), (size_t)ny * 16}, {oOpen, open.data(), n}, {oAx, ax.data(), n * 8}, {oAy, ay.data(), n * 8},
                    {oHn, hn.data(), n * 8}, {oCx, cx.data(), n * 8}, {oCy, cy.data(), n * 8}, {oCz, cz.data(), n * 8},
                    {oRho, rho, (size_t)nz * 8}, {oDz, dz.data(), (size_t)nz * 8}};
  for (const Up& up : ups)
    if ((e = cudaMemcpyAsync(M + up.off, up.src, up.bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess) break;
  if (e == cudaSuccess) e = cudaMemsetAsync(f->arrived, 0, sizeof(unsigned), st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaFree(f->mem); delete f;
    return sg_context_fail(ctx, SG_ERR_DEVICE, (std::string("masked faces: ") + cudaGetErrorString(e)).c_str());
  }
  *out = f;
  return SG_OK;
}

int sg_faces_set_velocity(sg_faces* f, const float* u, const float* v, const float* w, double* mx, double* my, double* mz, double* div) {
  if (!f) return SG_ERR_INVALID;
  if (!u || !v || !w) return sg_context_fail(f->ctx, SG_ERR_INVALID, "masked faces: u, v and w buffers");
  cudaSetDevice(sg_context_device(f->ctx));
  cudaStream_t s = sg_context_stream(f->ctx);
  const size_t n = f->fg.n;
  const int nb = blocks(n);
  auto fail_f = [&](const char* what, cudaError_t e) {
    return sg_context_fail(f->ctx, SG_ERR_DEVICE, (std::string("masked faces: ") + what + ": " + cudaGetErrorString(e)).c_str());
  };
  cudaError_t e;
  const float* host[3] = {u, v, w};
  float* dev[3] = {f->u, f->v, f->w};
  for (int k = 0; k < 3; k++)
    if ((e = cudaMemcpyAsync(dev[k], host[k], n * 4, cudaMemcpyHostToDevice, s)) != cudaSuccess) return fail_f("copy in", e);
  MpState init{};
  init.tolerance = f->tolerance; init.maxIt = f->maxIt; init.keepRR = 1;
  if ((e = cudaMemcpyAsync(f->st, &init, sizeof(MpState), cudaMemcpyHostToDevice, s)) != cudaSuccess ||
      (e = cudaMemsetAsync(f->q, 0, n * 8, s)) != cudaSuccess || (e = cudaMemsetAsync(f->d[0], 0, n * 8, s)) != cudaSuccess)
    return fail_f("state", e);
  // faces, shut next to the ground; r = b = -h div, bb (= the first rr); z = S0^-1 r, rz (:117-126).
  k_tm_faces<<<nb, TPB, 0, s>>>(f->u, f->v, f->w, f->mx, f->my, f->mz, f->fg);
  k_tm_tdiv<0><<<nb, TPB, 0, s>>>(f->mx, f->my, f->mz, f->r, f->part, f->arrived, f->fg, f->st);
  enqueue_first_precondition(f->sp, f->z, f->r, nullptr, nullptr, f->part, f->arrived, f->st, s);
  if ((e = cudaGetLastError()) != cudaSuccess) return fail_f("launch", e);
  if (!f->chunk) {
    cudaGraph_t graph = nullptr;
    if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) return fail_f("capture", e);
    for (int it = 0; it < REPLAY; it++) enqueue_face_iteration(f, it & 1, s);
    e = cudaStreamEndCapture(s, &graph);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&f->chunk, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (e != cudaSuccess) { f->chunk = nullptr; return fail_f("graph", e); }
  }
  int done = 0;
  for (int c = 0;; c++) {
    if ((e = cudaMemcpyAsync(&done, &f->st->done, 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess)
      return fail_f("solve", e);
    if (done || c > f->maxIt / REPLAY + 1) break;
    if ((e = cudaGraphLaunch(f->chunk, s)) != cudaSuccess) return fail_f("graph launch", e);
  }
  if (!done) return sg_context_fail(f->ctx, SG_ERR_DEVICE, "masked faces: the iterations did not stop");
  // The fluxes lose M rho0 grad(q); div the apertures' divergence over the node heights (:150-152).
  k_tm_correct<<<nb, TPB, 0, s>>>(f->q, f->mx, f->my, f->mz, f->fg, f->st);
  k_tm_tdiv<1><<<nb, TPB, 0, s>>>(f->mx, f->my, f->mz, f->div, nullptr, nullptr, f->fg, f->st);
  MpState fin{};
  if ((e = cudaMemcpyAsync(&fin, f->st, sizeof(MpState), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return fail_f("state", e);
  double* outs[4] = {mx, my, mz, div};
  const double* devs[4] = {f->mx, f->my, f->mz, f->div};
  for (int k = 0; k < 4; k++)
    if (outs[k] && (e = cudaMemcpyAsync(outs[k], devs[k], n * 8, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return fail_f("copy out", e);
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess) return fail_f("faces", e);
  if (fin.done == ZERO) { f->iterations = 0; f->residual = 0; }
  else { f->iterations = fin.k; f->residual = std::sqrt(fin.rr / fin.bb); }
  return SG_OK;
}

int sg_faces_stats(sg_faces* f, int32_t* iterations, double* residual) {
  if (!f) return SG_ERR_INVALID;
  if (iterations) *iterations = f->iterations;
  if (residual) *residual = f->residual;
  return SG_OK;
}

int sg_faces_destroy(sg_faces* f) {
  if (!f) return SG_ERR_INVALID;
  cudaSetDevice(sg_context_device(f->ctx));
  cudaStreamSynchronize(sg_context_stream(f->ctx));
  if (f->chunk) cudaGraphExecDestroy(f->chunk);
  cudaFree(f->mem);
  delete f;
  return SG_OK;
}

int sg_masked_destroy(sg_masked* m) {
  if (!m) return SG_ERR_INVALID;
  cudaSetDevice(sg_context_device(m->ctx));
  cudaStreamSynchronize(sg_context_stream(m->ctx));
  if (m->chunk) cudaGraphExecDestroy(m->chunk);
  if (m->orderedChunk) cudaGraphExecDestroy(m->orderedChunk);
  cudaFree(m->mem);
  delete m;
  return SG_OK;
}

}  // extern "C"
