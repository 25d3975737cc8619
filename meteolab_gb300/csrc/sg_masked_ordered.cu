// See sg_masked_ordered.cuh. One iteration is nine launches: the gradient over the node masses and its column fluxes, their
// divergence with d.Sd, the q/r update with r.r, five of the preconditioner (x and y sums, sweeps, y and x sums with r.z),
// the new direction. The FP64 pipe bounds it (two operations a clock and SM, a divide costs seven): the direct sums
// are 770 operations a cell at 127 x 113, 460 at 80 x 64, and are left as they are; what touches no rounding is taken out.
// A cell's V phi, a node's gradient and a column's fluxes are formed once instead of by every neighbour, divides by dx, dy,
// the spacings and the pivots are quotients from their reciprocals, and the sums fill their warps over several rows or
// columns. The stencils take 92 operations a cell so (234 before), an iteration on 80 x 64 x 50 nodes 0.39 ms (0.55 before), on
// 40 x 32 x 50 0.11 (0.20).
// Every operation below that could be contracted is written out, so that its rounding does not depend on its neighbours.
#include <algorithm>
#include "sg_masked_ordered.cuh"

namespace sg {
namespace {

enum { STOP = 1, ZERO = 2, ANY = 3 };
enum { R_BB, R_RZ0, R_RR0, R_RR, R_DSD, R_RZN };
constexpr int TPB = 256, REPLAY_ORDERED = 8;
using Geo = OrderedSolve;

// x / d to the last bit, from r = 1 / d correctly rounded: x r is within 1.5 units, the first remainder brings it within
// one, the second gives the rounded quotient (Markstein, IBM J. Res. Dev. 34, 1990). Five FP64 operations where a divide
// costs seven; finite operands away from underflow. The remainders are taken with the sign that leaves a zero its own: d > 0
// (spacings) here, d < 0 (pivots) below.
__device__ __forceinline__ double quotient(double x, double d, double r) {
  double q = __dmul_rn(x, r);
  q = __fma_rn(__fma_rn(q, d, -x), -r, q);
  return __fma_rn(__fma_rn(q, d, -x), -r, q);
}
__device__ __forceinline__ double quotient_negative(double x, double d, double r) {
  double q = __dmul_rn(x, r);
  q = __fma_rn(__fma_rn(-q, d, x), r, q);
  return __fma_rn(__fma_rn(-q, d, x), r, q);
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// Sum over the block (valid in thread 0); every thread of the block calls it.
__device__ __forceinline__ double block_sum(double v, double* sh) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  return wid == 0 ? warp_sum(lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0) : 0;
}

// In the block that ends last (a counter; no block waits): the sum of the partials in a fixed order, acted on (the scalars
// of :306-329). The block's own partials are written by thread 0, or by any before a barrier. Blocks of TPB threads.
template <int OP>
__device__ __forceinline__ void finish(const double* __restrict__ part, int nparts, double* sh, const Geo& g) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(g.arrived, 1u) == gridDim.x * gridDim.y - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v = 0;
  for (int i = threadIdx.x; i < nparts; i += TPB) v = __dadd_rn(v, __ldcg(part + i));
  const double s = block_sum(v, sh);
  if (threadIdx.x != 0) return;
  OrderedState* st = g.st;
  *g.arrived = 0;
  if (OP == R_BB) {
    st->bb = s; st->tol2bb = st->tolerance * st->tolerance * s; st->rr = 0; st->k = 0;
    if (!(s > 0)) st->done = ZERO;
  } else if (OP == R_RR0) {  // the first top-of-loop test
    if (st->maxIt > 0) { st->rr = s; if (s <= st->tol2bb) st->done = STOP; }
  } else if (OP == R_RZ0) {
    st->rz = s;
    if (st->maxIt <= 0) st->done = STOP;
  } else if (OP == R_DSD) {
    if (!(s > 0)) st->done = STOP;
    else st->alpha = st->rz / s;
  } else if (OP == R_RR) {  // the next iteration's test: what follows the update in this one changes no result
    if (st->k + 1 < st->maxIt) {
      st->rr = s;
      if (s <= st->tol2bb) { st->k++; st->done = STOP; }
    }
  } else {
    st->beta = s / st->rz; st->rz = s; st->k++;
    if (st->k >= st->maxIt) st->done = STOP;
  }
}

// V phi of a cell of layer k of q = V phi's vector, as the gradient weighs it: dzs (q / dzs), zero in the dropped cells.
__device__ __forceinline__ double v_phi(double q, size_t c, int k, const Geo& g) {
  const double h = g.dzs[k];
  return g.dropped[c] ? 0 : __dmul_rn(h, quotient(q, h, g.idz[k]));
}

// The first guess q = V phi from the last pressure (:311).
__global__ void k_or_start(const double* __restrict__ p, double dt, Geo g) {
  if (g.st->done & ZERO) return;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.cells) return;
  const int k = (int)(c / g.layer);
  const double q = g.dropped[c] ? 0 : __dmul_rn(__dmul_rn(p[c], dt), g.dzs[k]);
  g.q[c] = q; g.e[c] = v_phi(q, c, k, g);
}

// d = z (FIRST) or d = z + beta d (:331, :328); q as it stands (LAST); with V phi.
enum { FIRST, NEXT, LAST };
template <int MODE>
__global__ void k_or_dir(Geo g) {
  if (g.st->done & (MODE == NEXT ? ANY : ZERO)) return;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.cells) return;
  double v;
  if (MODE == LAST) v = g.q[c];
  else g.d[c] = v = MODE == FIRST ? g.z[c] : __fma_rn(g.st->beta, g.d[c], g.z[c]);
  g.e[c] = v_phi(v, c, (int)(c / g.layer), g);
}

// A thread marches `seg` cell layers of one column of e = V phi: each node's gradientPart (:270-300), the operator's
// adjoint over its mass, and from it the cells' column fluxes (k_mp_flux's). NODES: the gradients themselves, seg nodes.
template <bool NODES>
__global__ void __launch_bounds__(64) k_or_march(Geo g, int seg, int skip) {
  if (g.st->done & skip) return;
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= g.layer) return;
  const int j = col / g.nx, x = col - j * g.nx, j0 = j * g.nx, jm = (j == 0 ? g.ny - 1 : j - 1) * g.nx, xm = x == 0 ? g.nx - 1 : x - 1;
  const int k0 = blockIdx.y * seg, k1 = min(NODES ? g.nz : g.nc, k0 + seg);
  struct Layer { double u, v, w; };
  auto layer_of = [&](int k) {
    if (k < 0 || k >= g.nc) return Layer{0, 0, 0};
    const double* e = g.e + (size_t)k * g.layer;
    const double a = e[xm + jm], b = e[x + jm], c = e[xm + j0], d = e[col], ab = __dadd_rn(a, b);
    return Layer{__dsub_rn(__dadd_rn(__dsub_rn(a, b), c), d), __dsub_rn(__dsub_rn(ab, c), d), __dadd_rn(__dadd_rn(ab, c), d)};
  };
  auto node = [&](int k, const Layer& below, const Layer& above) {
    const size_t i = col + (size_t)k * g.layer;
    if (g.solid[i]) return Layer{0, 0, 0};
    const double r = g.rho4[k], m = g.invMass[i];
    double gu = 0, gv = 0, gw = 0;
    if (k < g.nc) {
      const double f = g.A[i];
      gu = quotient(__dmul_rn(f, above.u), g.dx, g.rdx); gv = quotient(__dmul_rn(f, above.v), g.dy, g.rdy);
      gw = -quotient(__dmul_rn(r, above.w), g.dzs[k], g.idz[k]);
    }
    if (k > 0) {
      const double f = g.B[i - g.layer];
      gu = __dadd_rn(gu, quotient(__dmul_rn(f, below.u), g.dx, g.rdx));
      gv = __dadd_rn(gv, quotient(__dmul_rn(f, below.v), g.dy, g.rdy));
      gw = __dadd_rn(gw, quotient(__dmul_rn(r, below.w), g.dzs[k - 1], g.idz[k - 1]));
    }
    return Layer{__dmul_rn(gu, m), __dmul_rn(gv, m), g.wall[i] || k == 0 || k == g.nc ? 0 : __dmul_rn(gw, m)};
  };
  Layer below = layer_of(k0 - 1), above = layer_of(k0);
  if (NODES) {
    for (int k = k0; k < k1; k++) {
      const Layer t = node(k, below, above);
      const size_t i = col + (size_t)k * g.layer;
      g.fu[i] = t.u; g.fv[i] = t.v; g.fw[i] = t.w;
      below = above; above = layer_of(k + 1);
    }
    return;
  }
  Layer lo = node(k0, below, above);
  for (int k = k0; k < k1; k++) {
    below = above; above = layer_of(k + 1);
    const Layer hi = node(k + 1, below, above);
    const size_t c = col + (size_t)k * g.layer;
    const double a = g.A[c], b = g.B[c];
    g.fu[c] = __fma_rn(a, lo.u, __dmul_rn(b, hi.u));
    g.fv[c] = __fma_rn(a, lo.v, __dmul_rn(b, hi.v));
    g.fw[c] = __fma_rn(g.rho4[k + 1], hi.w, -__dmul_rn(g.rho4[k], lo.w));
    lo = hi;
  }
}

// The column fluxes of the node winds; no wind is read where a column has no open share of the layer.
__global__ void __launch_bounds__(TPB) k_or_wind(const float* __restrict__ u, const float* __restrict__ v, const float* __restrict__ w, Geo g) {
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.cells) return;
  const int k = (int)(c / g.layer);
  const size_t up = c + g.layer;
  const double a = g.A[c], b = g.B[c];
  const bool open = b > 0;
  g.fu[c] = open ? __fma_rn(a, (double)u[c], __dmul_rn(b, (double)u[up])) : 0;
  g.fv[c] = open ? __fma_rn(a, (double)v[c], __dmul_rn(b, (double)v[up])) : 0;
  g.fw[c] = __fma_rn(g.rho4[k + 1], (double)w[up], -__dmul_rn(g.rho4[k], (double)w[c]));
}

// divergencePart (:240-264) of every cell from its four columns' fluxes, and OP's sum: R_BB out . out, R_DSD out . d; R_RR0
// r = -b - out (:313) and r . r.
template <int OP>
__global__ void __launch_bounds__(TPB) k_or_div(double* __restrict__ out, Geo g, int skip) {
  __shared__ double sh[32];
  if (g.st->done & skip) return;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double dot = 0;
  if (c < g.cells) {
    double val = 0;
    const int k = (int)(c / g.layer);
    if (!g.dropped[c]) {
      const int rem = (int)(c - (size_t)k * g.layer), j = rem / g.nx, i = rem - j * g.nx;
      const int i1 = i + 1 == g.nx ? 0 : i + 1, j0 = j * g.nx, j1 = (j + 1 == g.ny ? 0 : j + 1) * g.nx;
      const size_t l = (size_t)k * g.layer, p = i + j0 + l, q = i1 + j0 + l, r = i + j1 + l, s = i1 + j1 + l;
      const double ddx = __dadd_rn(__dsub_rn(__dsub_rn(g.fu[q], g.fu[p]), g.fu[r]), g.fu[s]);
      const double ddy = __dadd_rn(__dadd_rn(__dsub_rn(-g.fv[p], g.fv[q]), g.fv[r]), g.fv[s]);
      const double ddz = __dadd_rn(__dadd_rn(__dadd_rn(g.fw[p], g.fw[q]), g.fw[r]), g.fw[s]);
      val = __dadd_rn(__dadd_rn(quotient(ddx, g.dx, g.rdx), quotient(ddy, g.dy, g.rdy)), quotient(ddz, g.dzs[k], g.idz[k]));
    }
    if (OP == R_RR0) val = __dsub_rn(-g.b[c], val);
    out[c] = val;
    dot = __dmul_rn(val, OP == R_DSD ? g.d[c] : val);
  }
  const double s = block_sum(dot, sh);
  if (threadIdx.x == 0) g.part[blockIdx.x] = s;
  __syncthreads();
  finish<OP>(g.part, gridDim.x, sh, g);
}

// q += alpha d, r -= alpha S d, with r.r (:324).
__global__ void __launch_bounds__(TPB) k_or_update(Geo g) {
  __shared__ double sh[32];
  if (g.st->done) return;
  const double alpha = g.st->alpha;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0;
  if (c < g.cells) {
    g.q[c] = __fma_rn(alpha, g.d[c], g.q[c]);
    v = __fma_rn(-alpha, g.sd[c], g.r[c]);
    g.r[c] = v;
  }
  const double s = block_sum(__dmul_rn(v, v), sh);
  if (threadIdx.x == 0) g.part[blockIdx.x] = s;
  __syncthreads();
  finish<R_RR>(g.part, gridDim.x, sh, g);
}

// Forward x-sums of each cell row of -r: S1[k][m][y], m <= nx / 2. A block takes `rows` rows of a layer, so that their
// nx / 2 + 1 modes fill its warps.
__global__ void __launch_bounds__(TPB) k_or_xsum(Geo g, int rows, int skip) {
  extern __shared__ double row[];
  if (g.st->done & skip) return;
  const int y0 = blockIdx.x * rows, k = blockIdx.y, nx = g.nx, nm = g.mh + 1, nr = min(rows, g.ny - y0);
  const double* s = g.r + (size_t)k * g.layer + (size_t)y0 * nx;
  for (int i = threadIdx.x; i < nr * nx; i += TPB) row[i] = -s[i];
  __syncthreads();
  for (int u = threadIdx.x; u < nr * nm; u += TPB) {
    const int ry = u / nm, m = u - ry * nm;
    const double* v = row + ry * nx;
    double re = 0, im = 0;
    int t = 0;
    for (int x = 0; x < nx; x++) {
      const double2 tw = g.twx[t];
      re = __fma_rn(v[x], tw.x, re);
      im = __fma_rn(-v[x], tw.y, im);
      t += m;
      if (t >= nx) t -= nx;
    }
    g.S1[((size_t)k * nm + m) * g.ny + y0 + ry] = make_double2(re, im);
  }
}

// y-sums of the (cell layer, x-mode) columns, forward S1 to S2 or inverse S2 to S1 (unnormalised); a block takes `cols`.
template <bool FORWARD>
__global__ void __launch_bounds__(TPB) k_or_ysum(Geo g, int cols, int skip) {
  extern __shared__ double2 colv[];
  if (g.st->done & skip) return;
  const int ny = g.ny, all = g.nc * (g.mh + 1), c0 = blockIdx.x * cols, count = min(cols, all - c0) * ny;
  const double2* in = (FORWARD ? g.S1 : g.S2) + (size_t)c0 * ny;
  double2* out = (FORWARD ? g.S2 : g.S1) + (size_t)c0 * ny;
  for (int i = threadIdx.x; i < count; i += TPB) colv[i] = in[i];
  __syncthreads();
  for (int u = threadIdx.x; u < count; u += TPB) {
    const int c = u / ny, nn = u - c * ny;
    const double2* v = colv + c * ny;
    double re = 0, im = 0;
    int t = 0;
    for (int y = 0; y < ny; y++) {
      const double2 tw = g.twy[t], a = v[y];
      const double s = FORWARD ? -tw.y : tw.y;
      re = __fma_rn(a.x, tw.x, __fma_rn(-a.y, s, re));
      im = __fma_rn(a.y, tw.x, __fma_rn(a.x, s, im));
      t += nn;
      if (t >= ny) t -= ny;
    }
    out[u] = make_double2(re, im);
  }
}

// One mode a thread, the reference's sweep over the cell layers (pressure.ts:118-140); the forward values are kept in
// place for the back substitution. A mode the reference zeroes, and the pinned lowest cell of the uniform mode, have a
// pivot of 1 with the reciprocal 0 (their values come out zero). The recurrence is a dependent chain: each eight layers'
// coefficients and right-hand sides are loaded before their eight steps, so a step waits on the arithmetic, not on memory.
constexpr int AHEAD = 8;
__global__ void k_or_sweep(Geo g, int skip) {
  if (g.st->done & skip) return;
  const int mode = blockIdx.x * blockDim.x + threadIdx.x, modes = g.modes, nc = g.nc;
  if (mode >= modes) return;
  double2 d = make_double2(0, 0);
  for (int k0 = 0; k0 < nc; k0 += AHEAD) {
    double2 r[AHEAD];
    double a[AHEAD], m[AHEAD], w[AHEAD];
#pragma unroll
    for (int q = 0; q < AHEAD; q++) {
      const size_t at = (size_t)min(k0 + q, nc - 1) * modes + mode;
      r[q] = g.S2[at]; a[q] = g.lo[at]; m[q] = g.piv[at]; w[q] = g.rpiv[at];
    }
#pragma unroll
    for (int q = 0; q < AHEAD; q++)
      if (k0 + q < nc) {
        d = make_double2(quotient_negative(__fma_rn(-a[q], d.x, r[q].x), m[q], w[q]), quotient_negative(__fma_rn(-a[q], d.y, r[q].y), m[q], w[q]));
        g.S2[(size_t)(k0 + q) * modes + mode] = d;
      }
  }
  for (int k1 = nc - 2; k1 >= 0; k1 -= AHEAD) {
    double2 v[AHEAD];
    double c[AHEAD];
#pragma unroll
    for (int q = 0; q < AHEAD; q++) {
      const size_t at = (size_t)max(k1 - q, 0) * modes + mode;
      v[q] = g.S2[at]; c[q] = g.cp[at];
    }
#pragma unroll
    for (int q = 0; q < AHEAD; q++)
      if (k1 - q >= 0) {
        d = make_double2(__fma_rn(-c[q], d.x, v[q].x), __fma_rn(-c[q], d.y, v[q].y));
        g.S2[(size_t)(k1 - q) * modes + mode] = d;
      }
  }
}

// Inverse x-sums of the cell rows from their half spectra, / (nx ny): the preconditioner's z = V phi, zero in the dropped
// cells (:355), and OP's r . z. A block takes `rows` rows; each row's part of the sum is a warp's, over warps of 32 values
// (each thread of at most 256 its own, then a tree, then a tree over the warps).
template <int OP>
__global__ void __launch_bounds__(TPB) k_or_xinv(Geo g, int rows, int skip) {
  extern __shared__ double2 zs[];
  __shared__ double sh[32];
  if (g.st->done & skip) return;
  const int y0 = blockIdx.x * rows, k = blockIdx.y, nx = g.nx, nm = g.mh + 1, nr = min(rows, g.ny - y0);
  double* prod = reinterpret_cast<double*>(zs + rows * nm);
  for (int i = threadIdx.x; i < nr * nm; i += TPB) {
    const int m = i / nr, ry = i - m * nr;
    zs[ry * nm + m] = g.S1[((size_t)k * nm + m) * g.ny + y0 + ry];
  }
  __syncthreads();
  const double scale = 1.0 / ((double)nx * g.ny), h = g.dzs[k];
  const size_t base = (size_t)k * g.layer + (size_t)y0 * nx;
  for (int u = threadIdx.x; u < nr * nx; u += TPB) {
    const int ry = u / nx, x = u - ry * nx;
    const double2* z = zs + ry * nm;
    double v = z[0].x;
    int t = 0;
    for (int m = 1; m < nm; m++) {
      t += x;
      if (t >= nx) t -= nx;
      const double2 tw = g.twx[t];
      v = 2 * m == nx ? __fma_rn(z[m].x, tw.x, v) : __fma_rn(2.0, __fma_rn(z[m].x, tw.x, __dmul_rn(-z[m].y, tw.y)), v);
    }
    const double val = g.dropped[base + u] ? 0 : __dmul_rn(__dmul_rn(v, scale), h);
    g.z[base + u] = val;
    prod[u] = val;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, across = min(256, (nx + 31) / 32 * 32);
  for (int ry = threadIdx.x >> 5; ry < nr; ry += TPB / 32) {
    double mine = 0;
    for (int w = 0; w < across / 32; w++) {
      double dot = 0;
      for (int x = w * 32 + lane; x < nx; x += across) dot = __fma_rn(g.r[base + ry * nx + x], prod[ry * nx + x], dot);
      dot = __shfl_sync(0xffffffffu, warp_sum(dot), 0);
      if (lane == w) mine = dot;
    }
    mine = warp_sum(mine);
    if (lane == 0) {
      g.part[(size_t)k * g.ny + y0 + ry] = mine;
      __threadfence();
    }
  }
  __syncthreads();
  finish<OP>(g.part, g.ny * g.nc, sh, g);
}

// The pressure kept, q / V / dt (:332).
__global__ void k_or_finish(double* __restrict__ p, double dt, Geo g) {
  if (g.st->done & ZERO) return;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < g.cells) p[c] = g.q[c] / g.dzs[c / g.layer] / dt;
}

// u = M (u* - G phi): the correction added in FP32 stores, then masked (:334-336).
__global__ void k_or_correct(float* __restrict__ u, float* __restrict__ v, float* __restrict__ w, Geo g) {
  if (g.st->done & ZERO) return;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  if (g.solid[i]) { u[i] = 0; v[i] = 0; w[i] = 0; return; }
  u[i] = (float)((double)u[i] + g.fu[i]);
  v[i] = (float)((double)v[i] + g.fv[i]);
  const float wn = (float)((double)w[i] + g.fw[i]);
  w[i] = g.wall[i] || i < (size_t)g.layer || i >= g.n - g.layer ? 0.0f : wn;
}

int blocks(size_t count) { return (int)((count + TPB - 1) / TPB); }

template <bool NODES>
void enqueue_march(const Geo& g, int skip, cudaStream_t s) {
  // (two layers' work is a thread's start: as many layers as leave 152 SMs four blocks of 64 columns, within 4..16)
  const int levels = NODES ? g.nz : g.nc, seg = std::min(16, std::max(4, (int)((size_t)g.layer * levels / (152 * 256))));
  k_or_march<NODES><<<dim3((g.layer + 63) / 64, (levels + seg - 1) / seg), 64, 0, s>>>(g, seg, skip);
}

// The preconditioner z = P S0^-1 P r (:351-356): the flat solve of -r, z = V phi, with r.z.
template <int OP>
void enqueue_precondition(const Geo& g, int skip, cudaStream_t s) {
  const int nx = g.nx, ny = g.ny, nc = g.nc, nm = g.mh + 1, cols = std::max(1, TPB / ny);
  int rows = std::max(1, TPB / nm);
  k_or_xsum<<<dim3((ny + rows - 1) / rows, nc), TPB, (size_t)rows * nx * 8, s>>>(g, rows, skip);
  k_or_ysum<true><<<(nc * nm + cols - 1) / cols, TPB, (size_t)cols * ny * 16, s>>>(g, cols, skip);
  k_or_sweep<<<(g.modes + 63) / 64, 64, 0, s>>>(g, skip);
  k_or_ysum<false><<<(nc * nm + cols - 1) / cols, TPB, (size_t)cols * ny * 16, s>>>(g, cols, skip);
  rows = std::max(1, TPB / nx);
  k_or_xinv<OP><<<dim3((ny + rows - 1) / rows, nc), TPB, (size_t)rows * (nm * 16 + nx * 8), s>>>(g, rows, skip);
}

// One iteration of the loop (:314-329).
void enqueue_iteration(const Geo& g, cudaStream_t s) {
  const int cb = blocks(g.cells);
  enqueue_march<false>(g, ANY, s);
  k_or_div<R_DSD><<<cb, TPB, 0, s>>>(g.sd, g, ANY);
  k_or_update<<<cb, TPB, 0, s>>>(g);
  enqueue_precondition<R_RZN>(g, ANY, s);
  k_or_dir<NEXT><<<cb, TPB, 0, s>>>(g);
}

}  // namespace

size_t OrderedSolve::parts() const { return std::max((size_t)blocks(cells), (size_t)ny * nc); }

cudaError_t OrderedSolve::solve(float* u, float* v, float* w, double* p, double dt, int maxIt, double tolerance, cudaGraphExec_t* graph,
                                OrderedState* end, cudaStream_t s) const {
  const Geo& g = *this;
  const int cb = blocks(cells);
  OrderedState init{};
  init.tolerance = tolerance; init.maxIt = maxIt;
  cudaError_t e = cudaMemcpyAsync(st, &init, sizeof(init), cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return e;
  // b = D R M u*, bb; q from the first guess, r = -b - S q and its first test, z = P S0^-1 P r, rz, d = z (:306-314).
  k_or_wind<<<cb, TPB, 0, s>>>(u, v, w, g);
  k_or_div<R_BB><<<cb, TPB, 0, s>>>(b, g, 0);
  k_or_start<<<cb, TPB, 0, s>>>(p, dt, g);
  enqueue_march<false>(g, ZERO, s);
  k_or_div<R_RR0><<<cb, TPB, 0, s>>>(r, g, ZERO);
  enqueue_precondition<R_RZ0>(g, ANY, s);
  k_or_dir<FIRST><<<cb, TPB, 0, s>>>(g);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (!*graph) {
    cudaGraph_t captured = nullptr;
    if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) return e;
    for (int it = 0; it < REPLAY_ORDERED; it++) enqueue_iteration(g, s);
    e = cudaStreamEndCapture(s, &captured);
    if (e == cudaSuccess) e = cudaGraphInstantiate(graph, captured, 0);
    if (captured) cudaGraphDestroy(captured);
    if (e != cudaSuccess) { *graph = nullptr; return e; }
  }
  // Every iteration either counts or stops, so maxIt / 8 + 1 replays always reach the stop.
  int done = 0;
  for (int c = 0; !done; c++) {
    if (c > 0 && (e = cudaGraphLaunch(*graph, s)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(&done, &st->done, 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    if (!done && c > maxIt / REPLAY_ORDERED + 1) return cudaErrorLaunchFailure;
  }
  // u = M (u* - G phi); the pressure kept is phi / dt (:332-336).
  k_or_finish<<<cb, TPB, 0, s>>>(p, dt, g);
  k_or_dir<LAST><<<cb, TPB, 0, s>>>(g);
  enqueue_march<true>(g, ZERO, s);
  k_or_correct<<<blocks(n), TPB, 0, s>>>(u, v, w, g);
  if ((e = cudaMemcpyAsync(end, st, sizeof(*end), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
  return cudaGetLastError();
}

}  // namespace sg
