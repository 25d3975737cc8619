// FP64 spectral solves on the device: the horizontal transforms and the vertical sweeps shared by the storm's electric
// potential (sg_electric.cu, sg_lightning.cu) and the terrain's conjugate gradients (sg_masked.cu). A solve is five
// launches in place on one spectrum S[k][m][y] (levels k, half-complex x-modes m <= nx / 2, y): x forward (two real rows a
// complex transform), y forward, one tridiagonal sweep per mode along k, y inverse, x inverse.
//
// GB300 issues two FP64 operations a clock and SM (one per FP64 instruction and cell costs 0.4 us on 250,000 cells over
// the whole chip, and a divide costs seven of them), so the count of FP64 instructions bounds every kernel here, not
// memory and not index arithmetic: mixed-radix transforms (the direct sums they replace took 80 to 130 multiply-adds a
// value, these 20 to 30), no divides, the normalisation and the pairing's factor 1/2 folded into the sweep's
// coefficients, and work split finely enough to reach all 152 SMs. An 80 x 64 x 49 solve took 0.42 ms by direct sums.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>

namespace sg {

// The radices of a transform of n points (n <= 2048: at most 11), fours first; any prime is a radix.
struct Fft64 {
  int n = 0, nf = 0;
  int rad[11] = {};
};
Fft64 fft64_plan(int n);

#ifdef __CUDACC__
__device__ __forceinline__ double2 z_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 z_sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a times the conjugate of w (the tables hold exp(+2 pi i t / n), the forward transform turns by the conjugates)
__device__ __forceinline__ double2 z_turn(double2 a, double2 w) { return make_double2(fma(a.x, w.x, a.y * w.y), fma(a.y, w.x, -(a.x * w.y))); }

// One butterfly of a self-sorting (Stockham) stage of radix 4, 2, 3 or 5: j in [0, n / r), Ns the product of the radices
// already applied.
__device__ __forceinline__ void fft64_butterfly(const double2* x, double2* y, int n, int r, int Ns, int j, const double2* __restrict__ tw) {
  const int nb = n / r, k = j % Ns, t = k * (n / (Ns * r)), out = (j / Ns) * Ns * r + k;
  const bool turn = Ns > 1;  // (the first stage's turns are all 1)
  if (r == 4) {
    double2 v0 = x[j], v1 = x[j + nb], v2 = x[j + 2 * nb], v3 = x[j + 3 * nb];
    if (turn) { v1 = z_turn(v1, tw[t]); v2 = z_turn(v2, tw[2 * t]); v3 = z_turn(v3, tw[3 * t]); }
    const double2 a0 = z_add(v0, v2), a1 = z_sub(v0, v2), b0 = z_add(v1, v3), b1 = z_sub(v1, v3);
    y[out] = z_add(a0, b0);
    y[out + Ns] = make_double2(a1.x + b1.y, a1.y - b1.x);
    y[out + 2 * Ns] = z_sub(a0, b0);
    y[out + 3 * Ns] = make_double2(a1.x - b1.y, a1.y + b1.x);
  } else if (r == 2) {
    double2 v0 = x[j], v1 = x[j + nb];
    if (turn) v1 = z_turn(v1, tw[t]);
    y[out] = z_add(v0, v1); y[out + Ns] = z_sub(v0, v1);
  } else if (r == 3) {
    const double s3 = 0.866025403784438646763723170752936183;  // sin(pi / 3)
    double2 v0 = x[j], v1 = x[j + nb], v2 = x[j + 2 * nb];
    if (turn) { v1 = z_turn(v1, tw[t]); v2 = z_turn(v2, tw[2 * t]); }
    const double2 s = z_add(v1, v2), d = z_sub(v1, v2), m = make_double2(fma(-.5, s.x, v0.x), fma(-.5, s.y, v0.y));
    y[out] = z_add(v0, s);
    y[out + Ns] = make_double2(fma(s3, d.y, m.x), fma(-s3, d.x, m.y));
    y[out + 2 * Ns] = make_double2(fma(-s3, d.y, m.x), fma(s3, d.x, m.y));
  } else if (r == 5) {
    // cos and sin of 2 pi / 5 and 4 pi / 5
    const double c1 = 0.309016994374947424102293417182819059, s1 = 0.951056516295153572116439333379382143;
    const double c2 = -0.809016994374947424102293417182819059, s2 = 0.587785252292473129168705954639072769;
    double2 v0 = x[j], v1 = x[j + nb], v2 = x[j + 2 * nb], v3 = x[j + 3 * nb], v4 = x[j + 4 * nb];
    if (turn) { v1 = z_turn(v1, tw[t]); v2 = z_turn(v2, tw[2 * t]); v3 = z_turn(v3, tw[3 * t]); v4 = z_turn(v4, tw[4 * t]); }
    const double2 t1 = z_add(v1, v4), t2 = z_add(v2, v3), d1 = z_sub(v1, v4), d2 = z_sub(v2, v3);
    const double2 a = make_double2(fma(c2, t2.x, fma(c1, t1.x, v0.x)), fma(c2, t2.y, fma(c1, t1.y, v0.y)));
    const double2 b = make_double2(fma(c1, t2.x, fma(c2, t1.x, v0.x)), fma(c1, t2.y, fma(c2, t1.y, v0.y)));
    const double2 e = make_double2(fma(s2, d2.x, s1 * d1.x), fma(s2, d2.y, s1 * d1.y));
    const double2 f = make_double2(fma(-s1, d2.x, s2 * d1.x), fma(-s1, d2.y, s2 * d1.y));
    y[out] = make_double2(v0.x + t1.x + t2.x, v0.y + t1.y + t2.y);
    y[out + Ns] = make_double2(a.x + e.y, a.y - e.x);
    y[out + 4 * Ns] = make_double2(a.x - e.y, a.y + e.x);
    y[out + 2 * Ns] = make_double2(b.x + f.y, b.y - f.x);
    y[out + 3 * Ns] = make_double2(b.x - f.y, b.y + f.x);
  }
}

// A stage of any other (odd prime) radix r, over all rows: the turned inputs' sums and differences s_q = v_q + v_(r-q),
// d_q = v_q - v_(r-q) take their places, then a thread forms the outputs k and r - k together from
// v_0 + sum s_q cos(2 pi q k / r) and sum d_q sin(2 pi q k / r): r - 1 FMAs an output, a quarter of a direct sum's.
__device__ __forceinline__ void fft64_prime_stage(double2* a, double2* b, int rows, int n, int r, int Ns, const double2* __restrict__ tw) {
  const int nb = n / r, h = r / 2, step = n / (Ns * r);
  for (int u = threadIdx.x; u < rows * h * nb; u += blockDim.x) {
    const int row = u / (h * nb), e = u - row * h * nb, q = 1 + e / nb, j = e - (q - 1) * nb, t = (j % Ns) * step;
    double2 *x = a + row * n + j + q * nb, *y = a + row * n + j + (r - q) * nb;
    double2 v = *x, w = *y;
    if (Ns > 1) { v = z_turn(v, tw[q * t]); w = z_turn(w, tw[(r - q) * t]); }
    *x = z_add(v, w); *y = z_sub(v, w);
  }
  __syncthreads();
  for (int u = threadIdx.x; u < rows * (h + 1) * nb; u += blockDim.x) {
    const int row = u / ((h + 1) * nb), e = u - row * (h + 1) * nb, k = e / nb, j = e - k * nb, out = (j / Ns) * Ns * r + j % Ns;
    const double2* x = a + row * n + j;
    double2* y = b + row * n + out;
    double2 A = x[0], B = make_double2(0, 0);
    if (k == 0) {
      for (int q = 1; q <= h; q++) A = z_add(A, x[q * nb]);
      y[0] = A;
      continue;
    }
    int at = 0;
    for (int q = 1; q <= h; q++) {
      at += k;
      if (at >= r) at -= r;
      const double2 w = tw[at * nb], sq = x[q * nb], dq = x[(r - q) * nb];  // exp(2 pi i q k / r)
      A = make_double2(fma(sq.x, w.x, A.x), fma(sq.y, w.x, A.y));
      B = make_double2(fma(dq.x, w.y, B.x), fma(dq.y, w.y, B.y));
    }
    y[k * Ns] = make_double2(A.x + B.y, A.y - B.x);
    y[(r - k) * Ns] = make_double2(A.x - B.y, A.y + B.x);
  }
  __syncthreads();
}

// Forward transforms of `rows` rows of P.n values in shared memory, between a and b; returns the buffer with the result.
// All threads of the block call it with the input in place and synchronised; it ends synchronised.
__device__ __forceinline__ double2* fft64_rows(double2* a, double2* b, int rows, const Fft64& P, const double2* __restrict__ tw) {
  int Ns = 1;
  for (int s = 0; s < P.nf; s++) {
    const int r = P.rad[s], nb = P.n / r, total = rows * nb;
    if (r > 5) fft64_prime_stage(a, b, rows, P.n, r, Ns, tw);
    else {
      for (int u = threadIdx.x; u < total; u += blockDim.x) {
        const int row = u / nb, j = u - row * nb;
        fft64_butterfly(a + row * P.n, b + row * P.n, P.n, r, Ns, j, tw);
      }
      __syncthreads();
    }
    double2* t = a; a = b; b = t;
    Ns *= r;
  }
  return a;
}

// The half spectra (m <= nx / 2) of the `rows` real rows y0.. of level k from their paired transforms Z, twice the
// reference's (the factor is in the sweep's coefficients).
__device__ __forceinline__ void fft64_unpack(const double2* Z, double2* __restrict__ S, int nx, int ny, int y0, int rows, int k) {
  const int mh = nx / 2;
  for (int e = threadIdx.x; e < (mh + 1) * rows; e += blockDim.x) {
    const int m = e / rows, r = e - m * rows, c = m ? nx - m : 0;
    const double2 zm = Z[(r >> 1) * nx + m], zc = Z[(r >> 1) * nx + c];
    S[((size_t)k * (mh + 1) + m) * ny + y0 + r] = (r & 1) == 0 ? make_double2(zm.x + zc.x, zm.y - zc.y) : make_double2(zm.y + zc.y, zc.x - zm.x);
  }
}

// The paired rows of level k rebuilt from the half spectra as the conjugate of A + i B (Hermitian rows A and B), whose
// forward transform is the conjugate of the two real rows.
__device__ __forceinline__ void fft64_pack(const double2* __restrict__ S, double2* Z, int nx, int ny, int y0, int rows, int k) {
  const int mh = nx / 2, pairs = (rows + 1) / 2;
  for (int e = threadIdx.x; e < (mh + 1) * pairs; e += blockDim.x) {
    const int m = e / pairs, pr = e - m * pairs;
    const double2* at = S + ((size_t)k * (mh + 1) + m) * ny + y0 + 2 * pr;
    const bool real = m == 0 || 2 * m == nx;
    double2 A = at[0], B = 2 * pr + 1 < rows ? at[1] : make_double2(0, 0);
    if (real) { A.y = 0; B.y = 0; }
    Z[pr * nx + m] = make_double2(A.x - B.y, -(A.y + B.x));
    if (!real) Z[pr * nx + nx - m] = make_double2(A.x + B.y, A.y - B.x);
  }
}

#endif

// Launch shapes: the row pairs a block of the x-transforms takes, the columns a block of the y-transforms takes.
struct X64 { int pairs = 1, threads = 64, groups = 1; size_t smem = 0; };
struct Y64 { int cols = 1, threads = 32, blocks = 1; size_t smem = 0; };

// A solve: grid, levels, plans, launch shapes and its device arrays. `done`, `skip`: the launches return at once where
// *done & skip (done may be null).
struct Spectral64 {
  int nx = 0, ny = 0, levels = 0, mh = 0, modes = 0;
  Fft64 px, py;
  X64 x;
  Y64 y;
  double2 *S = nullptr, *twx = nullptr, *twy = nullptr;  // [levels][mh + 1][ny]; exp(2 pi i t / n)
  double *a = nullptr, *b = nullptr, *c = nullptr;       // [levels][modes]: the sweep's coefficients

  void shape(int nx, int ny, int levels);
  // the factor of the sweep's coefficient a: the pairing's 1/2 and the transforms' normalisation
  double factor() const { return .5 / ((double)nx * ny); }
  void forward_x(const double* src, cudaStream_t st, const int* done = nullptr, int skip = 0) const;
  void forward_y(cudaStream_t st, const int* done = nullptr, int skip = 0) const;
  void sweep(cudaStream_t st, int negate, const int* done = nullptr, int skip = 0) const;
  void inverse_y(cudaStream_t st, const int* done = nullptr, int skip = 0) const;
  // The whole solve, of src (levels x ny x nx) into out.
  void solve(const double* src, double* out, int negate, cudaStream_t st) const;
};

// Opts the solve's kernels in to the shared memory of rows and columns of more than 1536 points (64 KB at most).
constexpr int SPECTRAL64_SMEM = 65536;
cudaError_t spectral64_limits();

}  // namespace sg
