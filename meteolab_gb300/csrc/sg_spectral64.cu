// The FP64 spectral solves' kernels and launches (see sg_spectral64.cuh).
#include "sg_spectral64.cuh"

namespace sg {

Fft64 fft64_plan(int n) {
  Fft64 P;
  P.n = n;
  int rest = n;
  auto take = [&](int p) { while (rest % p == 0) { P.rad[P.nf++] = p; rest /= p; } };
  take(4); take(2); take(3); take(5);
  for (int p = 7; rest > 1; p += 2) take(p);
  return P;
}

namespace {

// Row pairs an x-transform block takes, and its threads: about a thousand points, so that a level of 64 rows of 80 is
// four blocks; fewer rows when the whole solve has few blocks.
X64 x64_shape(int nx, int ny, int levels) {
  const int all = (ny + 1) / 2;
  int pairs = std::max(1, std::min(std::min(8, all), 1024 / nx));
  while (pairs > 1 && (size_t)((all + pairs - 1) / pairs) * levels < 300) pairs = (pairs + 1) / 2;
  const int threads = std::min(256, std::max(64, (pairs * nx / 4 + 31) / 32 * 32));
  return {pairs, threads, (all + pairs - 1) / pairs, (size_t)2 * pairs * nx * sizeof(double2)};
}
Y64 y64_shape(int ny, int columns) {
  int cols = std::max(1, std::min(columns, 512 / ny));
  while (cols > 1 && (columns + cols - 1) / cols < 300) cols = (cols + 1) / 2;
  return {cols, std::min(256, std::max(32, (cols * ny / 4 + 31) / 32 * 32)), (columns + cols - 1) / cols, (size_t)2 * cols * ny * sizeof(double2)};
}

// x forward of `levels` levels of src (a block: the row pairs of its group, blockIdx.x, at level blockIdx.y).
__global__ void k64_xfwd(const double* __restrict__ src, double2* __restrict__ S, int nx, int ny, int pairs, Fft64 P, const double2* __restrict__ tw,
                         const int* __restrict__ done, int skip) {
  extern __shared__ double2 z64[];
  if (done && (*done & skip)) return;
  const int k = blockIdx.y, y0 = blockIdx.x * 2 * pairs, rows = min(2 * pairs, ny - y0);
  const double* s = src + (size_t)k * nx * ny + (size_t)y0 * nx;
  for (int e = threadIdx.x; e < (rows + (rows & 1)) * nx; e += blockDim.x) {
    const int r = e / nx, x = e - r * nx;
    reinterpret_cast<double*>(&z64[(r >> 1) * nx + x])[r & 1] = r < rows ? s[e] : 0.0;
  }
  __syncthreads();
  const double2* Z = fft64_rows(z64, z64 + pairs * nx, (rows + 1) / 2, P, tw);
  fft64_unpack(Z, S, nx, ny, y0, rows, k);
}

// y transforms of the columns (level, x-mode) in place, forward, or unnormalised inverse (the conjugate of the forward
// transform of the conjugate).
__global__ void k64_ycols(double2* __restrict__ S, int ny, int columns, int cols, Fft64 P, const double2* __restrict__ tw, int inverse,
                          const int* __restrict__ done, int skip) {
  extern __shared__ double2 z64[];
  if (done && (*done & skip)) return;
  const int c0 = blockIdx.x * cols, count = min(cols, columns - c0), total = count * ny;
  double2* g = S + (size_t)c0 * ny;
  for (int e = threadIdx.x; e < total; e += blockDim.x) { const double2 v = g[e]; z64[e] = make_double2(v.x, inverse ? -v.y : v.y); }
  __syncthreads();
  const double2* Z = fft64_rows(z64, z64 + cols * ny, count, P, tw);
  for (int e = threadIdx.x; e < total; e += blockDim.x) { const double2 v = Z[e]; g[e] = make_double2(v.x, inverse ? -v.y : v.y); }
}

// The vertical sweeps in place, a thread per mode and part (real, imaginary): forward d_k = a_k r_k - b_k d_(k-1)
// (a = 1 / pivot with the solve's factors, b = lower / pivot, from the host; `negate`: of minus the right-hand sides),
// back x_k = d_k - c_k x_(k+1). One FMA a level on the chain; eight levels' values are loaded ahead of their steps.
constexpr int SWEEP64_AHEAD = 8, SWEEP64_THREADS = 32;
__global__ void __launch_bounds__(SWEEP64_THREADS) k64_sweep(double* __restrict__ S, const double* __restrict__ a, const double* __restrict__ b,
                                                             const double* __restrict__ c, int levels, int modes, int negate,
                                                             const int* __restrict__ done, int skip) {
  if (done && (*done & skip)) return;
  const int u = blockIdx.x * SWEEP64_THREADS + threadIdx.x;
  if (u >= 2 * modes) return;
  const int g = u >> 1;
  double d = 0;
  for (int k0 = 0; k0 < levels; k0 += SWEEP64_AHEAD) {
    double r[SWEEP64_AHEAD], bb[SWEEP64_AHEAD];
#pragma unroll
    for (int q = 0; q < SWEEP64_AHEAD; q++) {
      const size_t k = min(k0 + q, levels - 1);
      const double v = a[k * modes + g] * S[2 * k * modes + u];
      r[q] = negate ? -v : v;
      bb[q] = b[k * modes + g];
    }
#pragma unroll
    for (int q = 0; q < SWEEP64_AHEAD; q++)
      if (k0 + q < levels) { d = fma(-bb[q], d, r[q]); S[2 * (size_t)(k0 + q) * modes + u] = d; }
  }
  for (int k1 = levels - 2; k1 >= 0; k1 -= SWEEP64_AHEAD) {
    double v[SWEEP64_AHEAD], cc[SWEEP64_AHEAD];
#pragma unroll
    for (int q = 0; q < SWEEP64_AHEAD; q++) {
      const size_t k = max(k1 - q, 0);
      v[q] = S[2 * k * modes + u];
      cc[q] = c[k * modes + g];
    }
#pragma unroll
    for (int q = 0; q < SWEEP64_AHEAD; q++)
      if (k1 - q >= 0) { d = fma(-cc[q], d, v[q]); S[2 * (size_t)(k1 - q) * modes + u] = d; }
  }
}

// x inverse of `levels` levels into out.
__global__ void k64_xinv(const double2* __restrict__ S, double* __restrict__ out, int nx, int ny, int pairs, Fft64 P, const double2* __restrict__ tw) {
  extern __shared__ double2 z64[];
  const int k = blockIdx.y, y0 = blockIdx.x * 2 * pairs, rows = min(2 * pairs, ny - y0);
  fft64_pack(S, z64, nx, ny, y0, rows, k);
  __syncthreads();
  const double2* Z = fft64_rows(z64, z64 + pairs * nx, (rows + 1) / 2, P, tw);
  double* o = out + (size_t)k * nx * ny + (size_t)y0 * nx;
  for (int e = threadIdx.x; e < rows * nx; e += blockDim.x) {
    const int r = e / nx, x = e - r * nx;
    const double2 v = Z[(r >> 1) * nx + x];
    o[e] = r & 1 ? -v.y : v.x;
  }
}

}  // namespace

void Spectral64::shape(int nx_, int ny_, int levels_) {
  nx = nx_; ny = ny_; levels = levels_; mh = nx / 2; modes = (mh + 1) * ny;
  px = fft64_plan(nx); py = fft64_plan(ny);
  x = x64_shape(nx, ny, levels); y = y64_shape(ny, (mh + 1) * levels);
}
void Spectral64::forward_x(const double* src, cudaStream_t st, const int* done, int skip) const {
  k64_xfwd<<<dim3(x.groups, levels), x.threads, x.smem, st>>>(src, S, nx, ny, x.pairs, px, twx, done, skip);
}
void Spectral64::forward_y(cudaStream_t st, const int* done, int skip) const {
  k64_ycols<<<y.blocks, y.threads, y.smem, st>>>(S, ny, (mh + 1) * levels, y.cols, py, twy, 0, done, skip);
}
void Spectral64::sweep(cudaStream_t st, int negate, const int* done, int skip) const {
  const int blocks = (2 * modes + SWEEP64_THREADS - 1) / SWEEP64_THREADS;
  k64_sweep<<<blocks, SWEEP64_THREADS, 0, st>>>(reinterpret_cast<double*>(S), a, b, c, levels, modes, negate, done, skip);
}
void Spectral64::inverse_y(cudaStream_t st, const int* done, int skip) const {
  k64_ycols<<<y.blocks, y.threads, y.smem, st>>>(S, ny, (mh + 1) * levels, y.cols, py, twy, 1, done, skip);
}
void Spectral64::solve(const double* src, double* out, int negate, cudaStream_t st) const {
  forward_x(src, st); forward_y(st); sweep(st, negate); inverse_y(st);
  k64_xinv<<<dim3(x.groups, levels), x.threads, x.smem, st>>>(S, out, nx, ny, x.pairs, px, twx);
}

cudaError_t spectral64_limits() {
  cudaError_t e = cudaFuncSetAttribute(k64_xfwd, cudaFuncAttributeMaxDynamicSharedMemorySize, SPECTRAL64_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k64_xinv, cudaFuncAttributeMaxDynamicSharedMemorySize, SPECTRAL64_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k64_ycols, cudaFuncAttributeMaxDynamicSharedMemorySize, SPECTRAL64_SMEM);
  return e;
}

}  // namespace sg
