// Lightning of an electrified run on the device (src/core/lightning.ts:135-420, driven by AtmosphereModel.discharge,
// src/core/model.ts:1537-1552): after every step, while the storm's field somewhere exceeds the breakdown threshold
// (and at most flashLimit(dt) times), one flash there; then the conduction of the small ions and the corona from the
// ground; then the vertical field for the next step's inductive charging.
//
// The work splits by its shape. Whole-grid passes (the charge density of the four carriers, the FP64 potential solve,
// the search for the strongest field, the conduction) are ordinary grid-wide kernels. A flash's channel grows one node
// at a time with a random pick among the links that exceed the propagation threshold, each pick depending on the last:
// one block grows it (k_lgt_grow), its threads weighting the growth front, which lies in shared memory, and the warp that
// holds the picked link doing the reference's sequential bookkeeping (the front's order, the neighbours appended in the
// reference's order, the running potential sum), so the channel is the reference's own for the same potential. The
// deposit of a stage is one block over the channel. The host steps through the flash's stages (a stage ends when the
// channel leaves the cloud, touches the ground or stops; the field is solved again between stages), reading a small
// state record after each: the control flow of Lightning.flash, with every array on the device.
//
// Every loop is bounded: a grow launch adds at most MAX_CHANNEL nodes, a flash has at most STROKES + 2 stages, a step
// at most flashLimit(dt) flashes.
#include <cuda_runtime.h>
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "sg_common.cuh"
#include "sg_elec_solve.cuh"
#include "sg_lightning.h"

namespace sg {

namespace {

constexpr double EPS0 = 8.8541878128e-12;                                                     // src/core/electric.ts:6
constexpr double E_INIT = 2.84e5, RHO_STANDARD = 1.225, F_CRIT = .43, RHO_MIN = 1e-10, CHANNEL_RADIUS = 1, SHIELDING = .25;  // lightning.ts:13-29
constexpr double SIGMA_GROUND = 2e-14, SIGMA_SCALE = 6000, CLOUD_SIGMA = .1, CLOUDY = 1e-5, CORONA_FIELD = 5e3, CORONA_RATE = 5e-13;  // :51-67
constexpr int GROW_THREADS = 128, DEP_THREADS = 256;

SG_D void mulberryNext(uint32_t& s) { s += 0x6D2B79F5u; }
SG_D double mulberry(uint32_t& s) {  // src/core/math.ts:7-14
  mulberryNext(s);
  uint32_t t = (s ^ (s >> 15)) * (1u | s);
  t = (t + (t ^ (t >> 7)) * (61u | t)) ^ t;
  return (double)(t ^ (t >> 14)) / 4294967296.0;
}
SG_D double lt(const LgtDev& L, int which, int z) { return L.lv[(size_t)which * L.nz + z]; }
SG_D double dmul(double a, double b) { return __dmul_rn(a, b); }
SG_D double dadd(double a, double b) { return __dadd_rn(a, b); }
// The FP64 pipe takes 64 cycles an instruction and warp on a quarter of an SM, comparisons and conversions included, so
// what only orders values goes by their bits: |v| below a bound, the sign of a product, cloud above CLOUDY (the float
// nearest 1e-5 lies below it, so the float comparison is the same).
SG_D long long bitsOf(double v) { return __double_as_longlong(v); }
SG_D bool below(double v, double bound) { return (bitsOf(v) & 0x7fffffffffffffffll) < bitsOf(bound); }  // |v| < bound, bound > 0
SG_D bool isZero(double v) { return (bitsOf(v) << 1) == 0; }
SG_D bool sameSign(double a, double b) { return (bitsOf(a) ^ bitsOf(b)) >= 0; }
SG_D bool cloudAt(float c) { return c > (float)CLOUDY; }
// sum / count to the last bit, from 1 / count correctly rounded: the product and one remainder (Markstein, IBM J. Res.
// Dev. 34, 1990); an FP64 divide's latency is that of 8.6 FMAs, this three.
SG_D double meanOf(double sum, double count, double icount) {
  const double m = dmul(sum, icount);
  return fma(fma(-m, count, sum), icount, m);
}
SG_D bool clearOf(double rho, float cloudy) { return below(rho, RHO_MIN) || !cloudAt(cloudy); }  // :343

// Block sum in a fixed order (warps by halves, then the warps), valid in every thread of warp 0; all threads call it.
SG_D double blockSum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v = dadd(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();  // (an earlier sum's sh is read)
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0;
  if (threadIdx.x < 32) for (int w = 0; w < (int)(blockDim.x >> 5); w++) v = dadd(v, sh[w]);
  return v;
}
// Whether this block is the last of its launch to arrive (a counter the caller clears then; no block waits).
SG_D bool lastBlock(unsigned* arrived) {
  __shared__ bool last;
  if (threadIdx.x == 0) { __threadfence(); last = atomicAdd(arrived, 1u) == gridDim.x - 1; }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// ---------------------------------------------------------------- grid-wide passes
// cloud(): the cloud water, ice and snow summed at each node as FP32 (:249-253).
__global__ void k_lgt_cloudy(const RunDesc R, const LgtDev L) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= R.n) return;
  L.cloudy[i] = __fadd_rn(__fadd_rn(field(R, 0, CLOUD)[i], field(R, 0, ICE)[i]), field(R, 0, SNOW)[i]);
}
// solve()'s charge density (:226-230): the four carriers summed in FP64, times the level's air density.
__global__ void k_lgt_rho(const RunDesc R, const LgtDev L) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= R.n) return;
  double s = (double)field(R, 0, CHARGE_ICE)[i];
  s = dadd(s, (double)field(R, 0, CHARGE_GRAUPEL)[i]);
  s = dadd(s, (double)field(R, 0, CHARGE_RAIN)[i]);
  s = dadd(s, (double)field(R, 0, CHARGE_AIR)[i]);
  L.rho[i] = dmul(s, lt(L, LT_AIR, i / R.layer));
}
// strongest() (:233-246): |E|^2 / Einit^2 of the interior nodes not failed at this step; the largest, first in node order.
// Each block's best goes to the partials, the block that ends last takes the best of those. Multiplying by the levels' reciprocals instead of dividing, and one pass instead of a second one for the node,
// took a search of the standard grid from 53 to 8 us.
SG_D double fieldRatio2(const RunDesc& R, const LgtDev& L, int i) {
  const int nx = R.nx, ny = R.ny, layer = R.layer, z = i / layer, y = (i - z * layer) / nx, x = i - z * layer - y * nx, row = y * nx + z * layer;
  const double* phi = L.phi;
  const int xp = x + 1 == nx ? 0 : x + 1, xm = x == 0 ? nx - 1 : x - 1, yp = y + 1 == ny ? 0 : y + 1, ym = y == 0 ? ny - 1 : y - 1;
  const double ex = dmul(phi[xp + row] - phi[xm + row], L.i2dx), ey = dmul(phi[x + yp * nx + z * layer] - phi[x + ym * nx + z * layer], L.i2dy);
  const double ez = dmul(phi[i + layer] - phi[i - layer], lt(L, LT_ISPAN, z));
  return dmul(dadd(dadd(dmul(ex, ex), dmul(ey, ey)), dmul(ez, ez)), lt(L, LT_IEINIT2, z));
}
struct Best { unsigned long long bits; int at; };  // non-negative: bits order as values
SG_D Best better(Best a, Best b) { return b.bits > a.bits || (b.bits == a.bits && b.at < a.at) ? b : a; }
SG_D Best blockBest(Best v) {
  __shared__ Best sh[32];
  for (int o = 16; o > 0; o >>= 1) v = better(v, Best{__shfl_xor_sync(0xffffffffu, v.bits, o), __shfl_xor_sync(0xffffffffu, v.at, o)});
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  v = sh[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); w++) v = better(v, sh[w]);
  return v;
}
__global__ void __launch_bounds__(256) k_lgt_strongest(const RunDesc R, const LgtDev L, int stamp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + R.layer;
  Best v{0, INT_MAX};
  if (i < R.n - R.layer && L.failed[i] != stamp) {
    const double r = fieldRatio2(R, L, i);
    if (r > 0) v = Best{(unsigned long long)bitsOf(r), i};
  }
  v = blockBest(v);
  unsigned long long* pb = reinterpret_cast<unsigned long long*>(L.part);
  int* pi = L.partAt;
  if (threadIdx.x == 0) { pb[blockIdx.x] = v.bits; pi[blockIdx.x] = v.at; }
  if (!lastBlock(&L.st->arrived)) return;
  v = Best{0, INT_MAX};
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) v = better(v, Best{__ldcg(pb + b), __ldcg(pi + b)});
  v = blockBest(v);
  if (threadIdx.x == 0) { L.st->maxBits = v.bits; L.st->best = v.at; L.st->arrived = 0; }
}

// ---------------------------------------------------------------- the channel
// The state record in shared memory for a kernel's run (a copy in, its changes out): the channel's bookkeeping reads
// and writes it every node, a round trip to L2 each time in global memory.
static_assert(sizeof(LgtState) % 4 == 0, "the state record copies as words");
SG_D void stateIn(LgtState& sh, const LgtDev& L, int t, int threads) {
  for (int k = t; k < (int)(sizeof(LgtState) / 4); k += threads) reinterpret_cast<int*>(&sh)[k] = reinterpret_cast<const int*>(L.st)[k];
}
SG_D void stateOut(const LgtState& sh, const LgtDev& L, int t, int threads) {
  for (int k = t; k < (int)(sizeof(LgtState) / 4); k += threads) reinterpret_cast<int*>(L.st)[k] = reinterpret_cast<const int*>(&sh)[k];
}

// The growth front: per link the node it reaches and its potential, the reciprocal of its reach (length times threshold),
// the channel index it starts from, and its tag: the reach's table index, whether the start's node is in clear air
// (TAG_FROM_CLEAR), whether its own is (TAG_CLEAR). The first FRONT links are in shared memory, any further ones in the
// run's buffers; L.pos holds each node's place on the front (-1: off it).
constexpr int FRONT = 5120, REACHES = 12;
constexpr unsigned TAG_CLEAR = 0x80000000u, TAG_FROM_CLEAR = 0x40000000u, TAG_REACH = 0xffffu;
struct Front {
  double *pj, *inv, *w, *reach, *ireach;  // w: the links' weights of the pick; reach, ireach: the tables [REACHES][nz]
  int *node, *from;
  unsigned* tag;
};
size_t front_bytes(int nz) { return (size_t)FRONT * (3 * 8 + 3 * 4) + (size_t)2 * REACHES * nz * 8; }
SG_D Front frontIn(double* sm, int nz) {
  Front F;
  F.pj = sm; F.inv = F.pj + FRONT; F.w = F.inv + FRONT; F.reach = F.w + FRONT; F.ireach = F.reach + REACHES * nz;
  F.node = reinterpret_cast<int*>(F.ireach + REACHES * nz); F.from = F.node + FRONT; F.tag = reinterpret_cast<unsigned*>(F.from + FRONT);
  return F;
}
SG_D double& linkPj(const Front& F, const LgtDev& L, int f) { return f < FRONT ? F.pj[f] : L.weight[f]; }
SG_D double& linkInv(const Front& F, const LgtDev& L, int f) { return f < FRONT ? F.inv[f] : L.scale[f]; }
SG_D int& linkNode(const Front& F, const LgtDev& L, int f) { return f < FRONT ? F.node[f] : L.frontier[f]; }
SG_D int& linkFrom(const Front& F, const LgtDev& L, int f) { return f < FRONT ? F.from[f] : L.link[f]; }
SG_D unsigned& linkTag(const Front& F, const LgtDev& L, int f) { return f < FRONT ? F.tag[f] : L.tag[f]; }
// The front's last link into place f (one lane).
SG_D void moveLink(const Front& F, const LgtDev& L, int f, int last) {
  if (last < FRONT) {
    const int j = F.node[last];
    F.pj[f] = F.pj[last]; F.inv[f] = F.inv[last]; F.node[f] = j; F.from[f] = F.from[last]; F.tag[f] = F.tag[last];
    L.pos[j] = f;
    return;
  }
  const int j = linkNode(F, L, last);
  linkPj(F, L, f) = linkPj(F, L, last); linkInv(F, L, f) = linkInv(F, L, last); linkNode(F, L, f) = j;
  linkFrom(F, L, f) = linkFrom(F, L, last); linkTag(F, L, f) = linkTag(F, L, last);
  L.pos[j] = f;
}
// A link's weight: how far it exceeds the threshold (:311-319), else 0. The two subtractions are all its FP64; what
// makes it zero goes by bits (after the ground contact a link into the ground or with pj before <= 0; a clear node's link
// with (pj - p) p >= 0).
SG_D double weightOf(double pj, double inv, int node, unsigned tag, int layer, int ground, double before, double potential) {
  const double d = pj - potential, w = fma(fabs(d), inv, -1.0);
  const bool grounded = ground >= 0 && (node < layer || isZero(pj) || isZero(before) || !sameSign(pj, before));
  const bool leader = (tag & TAG_CLEAR) && (isZero(d) || isZero(potential) || sameSign(d, potential));
  return !grounded && !leader && bitsOf(w) > 0 ? w : 0.0;
}

// add() of Lightning.flash (:294-304) and extend() (:389-404) by one warp, all 32 lanes, on the block's copy of the state
// record and the front: node j, the channel's nn-th. Lane l takes the l-th candidate of the reference's loop (level k from
// z - 1 up, then dj, then di); the candidates are distinct nodes, so each lane keeps its node's shorter link on its own,
// and the new links go on the front in the reference's order (a ballot over the lanes). Everything the candidates need is
// loaded before the potential's sum and its quotient, which take their latency's time.
SG_D void addNodeWarp(const RunDesc& R, const LgtDev& L, const Front& F, volatile LgtState& V, int j, int nn, int from, bool clear, double pj, int id,
                      double count, double icount) {
  const int lane = threadIdx.x & 31, nx = R.nx, ny = R.ny, nz = R.nz, layer = R.layer;
  const int z = j / layer, y = (j - z * layer) / nx, x = j - z * layer - y * nx;
  int q = -1, reach = 0, mark = 0, seen = 0, pos = -1;
  bool upward = false;
  double rho = 0, phi = 0;
  float cloudy = 0;
  if (j >= layer && lane < 27) {
    const int k = max(0, z - 1) + lane / 9, dj = (lane % 9) / 3 - 1, di = lane % 3 - 1;
    if (k <= min(nz - 2, z + 1) && x + di >= 0 && x + di < nx && y + dj >= 0 && y + dj < ny && !(k == z && di == 0 && dj == 0)) {
      q = x + di + (y + dj) * nx + k * layer;
      reach = ((k - z + 1) * 4 + abs(di) + 2 * abs(dj)) * nz + z;
      upward = k >= z;
      mark = L.mark[q]; seen = L.seen[q]; pos = L.pos[q]; rho = L.rho[q]; phi = L.phi[q]; cloudy = L.cloudy[q];
    }
  }
  if (lane == 0) {
    L.mark[j] = id; L.nodes[nn] = j; L.parent[nn] = from; V.nnodes = nn + 1;
    if (j < layer) { V.ground = j; V.before = V.potential; V.potential = 0; V.touched = 1; }
    else if (V.ground < 0) {
      const double sum = dadd(V.sum, pj);
      V.sum = sum; V.potential = meanOf(sum, count, icount);
    }
  }
  bool fresh = false;
  if (q >= 0 && !(mark == id || (upward && below(rho, RHO_MIN)))) {
    const unsigned tag = (unsigned)reach | (clear ? TAG_FROM_CLEAR : 0u);
    if (seen != id) fresh = true;
    else if (pos >= 0) {
      const unsigned old = linkTag(F, L, pos);
      if (F.reach[reach] < F.reach[old & TAG_REACH]) {
        linkInv(F, L, pos) = F.ireach[reach]; linkFrom(F, L, pos) = nn; linkTag(F, L, pos) = tag | (old & TAG_CLEAR);
      }
    }
    q = fresh ? q : -1;
    reach = (int)tag;
  }
  const unsigned mask = __ballot_sync(0xffffffffu, fresh);
  const int size = V.size;
  if (fresh) {
    const int f = size + __popc(mask & ((1u << lane) - 1));
    const unsigned tag = (unsigned)reach | (clearOf(rho, cloudy) ? TAG_CLEAR : 0u);
    const double inv = F.ireach[reach & TAG_REACH];
    if (f < FRONT) { F.node[f] = q; F.pj[f] = phi; F.inv[f] = inv; F.from[f] = nn; F.tag[f] = tag; }
    else { L.frontier[f] = q; L.weight[f] = phi; L.scale[f] = inv; L.link[f] = nn; L.tag[f] = tag; }
    L.seen[q] = id; L.pos[q] = f;
  }
  __syncwarp();
  if (lane == 0) V.size = size + __popc(mask);
  __syncwarp();
}

// One stage's growth (:309-331): until no link exceeds the threshold, the channel leaves the cloud (the first time),
// touches the ground, or has MAX_CHANNEL nodes. With a start node, first a new flash's state and that node; after a
// re-solve, first the front's potentials and the neutral channel's (:338).
// A pick: every thread weights a contiguous part of the front (an odd number of links: no bank conflicts); the warps'
// sums; one random number; the warp that holds the first position where the pick less the weights before it is no longer
// positive finds it by two scans, removes the link from the front, prunes the clear-air leader's other links (the
// reference's swap-with-last order) and adds the node; two barriers a node. One block on one SM, 3.6 us a node on a front
// of 400 links, bound by the latency of that chain: its FP64 instructions (64 cycles each on a quarter of the SM; three a
// link and three links a thread at a front of 300) are about a tenth of it, the rest the scans, the pick, the candidates'
// loads and the barriers.
__global__ void __launch_bounds__(GROW_THREADS) k_lgt_grow(const RunDesc R, const LgtDev L, int id, int start) {
  extern __shared__ double fsm[];
  constexpr int W = GROW_THREADS / 32;
  constexpr unsigned ALL = 0xffffffffu;
  __shared__ double wsum[W];
  __shared__ struct { double u, n, inv; } next[2];  // of this iteration and the next
  __shared__ int stop;
  __shared__ LgtState sh;
  volatile LgtState& V = sh;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, layer = R.layer;
  const Front F = frontIn(fsm, R.nz);
  stateIn(sh, L, t, GROW_THREADS);
  for (int e = t; e < REACHES * R.nz; e += GROW_THREADS) {
    F.reach[e] = L.lv[(size_t)LT_REACH * R.nz + e]; F.ireach[e] = L.lv[(size_t)LT_IREACH * R.nz + e];
  }
  if (t == 0) stop = 0;
  __syncthreads();
  if (start >= 0) {
    if (t == 0) {
      V.size = 0; V.nnodes = 0; V.npol = 0; V.ground = -1; V.touched = 0; V.left = 0; V.event = 0; V.strokes = 0; V.nstrokes = 0;
      V.sum = 0; V.potential = 0; V.before = 0; V.moment = 0; V.lowered = 0; V.neutralized = 0; V.stage = 0; V.needPotential = 0;
      V.start = start; V.id = id;
    }
    __syncthreads();
    if (warp == 0) addNodeWarp(R, L, F, V, start, 0, -1, clearOf(L.rho[start], L.cloudy[start]), L.phi[start], id, 1.0, 1.0);
  } else {
    for (int f = t; f < V.size; f += GROW_THREADS) {
      // the last stage's deposit changed the charge: the potentials and the clear air are the present ones
      const int j = L.frontier[f], from = L.link[f], i = L.nodes[from];
      const double pj = L.phi[j];
      const unsigned reach = L.tag[f] & TAG_REACH;
      const unsigned tag = reach | (clearOf(L.rho[j], L.cloudy[j]) ? TAG_CLEAR : 0u) | (clearOf(L.rho[i], L.cloudy[i]) ? TAG_FROM_CLEAR : 0u);
      if (f < FRONT) { F.node[f] = j; F.from[f] = from; F.tag[f] = tag; F.inv[f] = F.ireach[reach]; F.pj[f] = pj; }
      else { L.weight[f] = pj; L.tag[f] = tag; }
    }
    if (V.needPotential) {  // summed in node order
      const int nn = V.nnodes;
      double sum = 0;
      for (int c0 = 0; c0 < nn; c0 += FRONT) {
        __syncthreads();
        for (int c = c0 + t; c < min(nn, c0 + FRONT); c += GROW_THREADS) F.w[c - c0] = L.phi[L.nodes[c]];
        __syncthreads();
        if (t == 0) for (int c = c0; c < min(nn, c0 + FRONT); c++) sum = dadd(sum, F.w[c - c0]);
      }
      if (t == 0) { V.sum = sum; V.potential = sum / (double)nn; V.needPotential = 0; }
    }
  }
  __syncthreads();
  if (t == 0) { V.grown = V.nnodes; V.event = 0; }
  uint32_t rng = V.rng;  // every thread draws the same numbers
  __syncthreads();
  // What a node needs that its pick does not change, its random number, its count as a double and that's reciprocal, is
  // made an iteration ahead by a warp that does not hold the pick.
  auto ahead = [&](int slot, uint32_t r, int count) {
    const double u = mulberry(r), n = (double)count, inv = 1.0 / n;
    if (lane == 0) { next[slot].u = u; next[slot].n = n; next[slot].inv = inv; }
  };
  if (warp == 0) ahead(0, rng, V.nnodes + 1);
  __syncthreads();
  for (int iter = 0; iter < MAX_CHANNEL; iter++) {
    // what the holder changes below is read here, before the barrier: past it the holder may be ahead of any other thread
    const int size = V.size, ground = V.ground, nodes = V.nnodes, left = V.left;
    if (nodes >= MAX_CHANNEL || size == 0) break;
    const double before = V.before, potential = V.potential;
    const int C = ((size + GROW_THREADS - 1) / GROW_THREADS) | 1, f0 = min(size, t * C), f1 = min(size, f0 + C);
    double acc = 0;
    if (size <= FRONT) {
      for (int k = 0; k < C; k += 3) {  // three links' loads and subtractions side by side
        double w[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
          const int f = min(f0 + k + q, size - 1);
          w[q] = weightOf(F.pj[f], F.inv[f], F.node[f], F.tag[f], layer, ground, before, potential);
        }
#pragma unroll
        for (int q = 0; q < 3; q++)
          if (f0 + k + q < f1) { F.w[f0 + k + q] = w[q]; if (bitsOf(w[q]) != 0) acc = dadd(acc, w[q]); }
      }
    } else {
      for (int f = f0; f < f1; f++) {
        const double w = weightOf(linkPj(F, L, f), linkInv(F, L, f), linkNode(F, L, f), linkTag(F, L, f), layer, ground, before, potential);
        if (f < FRONT) F.w[f] = w;
        if (bitsOf(w) != 0) acc = dadd(acc, w);
      }
    }
    double inc = acc;  // inclusive sums of the parts in thread order
    for (int o = 1; o < 32; o <<= 1) { const double u = __shfl_up_sync(ALL, inc, o); if (lane >= o) inc = dadd(inc, u); }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    double total = wsum[0], mine = 0, upTo[W];
    upTo[0] = total;
#pragma unroll
    for (int w = 1; w < W; w++) { if (w == warp) mine = total; total = dadd(total, wsum[w]); upTo[w] = total; }
    if (bitsOf(total) == 0) break;
    const double pick = dmul(next[iter & 1].u, total);
    mulberryNext(rng);
    int holder = W - 1;
#pragma unroll
    for (int w = W - 2; w >= 0; w--) if (bitsOf(pick) <= bitsOf(upTo[w])) holder = w;
    if (warp == (holder + 1) % W) ahead((iter + 1) & 1, rng, nodes + 2);
    if (warp == holder) {
      // the part, then the link (by scans over its weights)
      const unsigned parts = __ballot_sync(ALL, bitsOf(acc) != 0 && bitsOf(pick) <= bitsOf(dadd(mine, inc)));
      const unsigned some = __ballot_sync(ALL, bitsOf(acc) != 0);
      const int p = parts ? __ffs(parts) - 1 : some ? 31 - __clz(some) : 0;
      double exc = __shfl_up_sync(ALL, inc, 1);
      if (lane == 0) exc = 0;
      double cum = dadd(mine, __shfl_sync(ALL, exc, p));
      const int g0 = __shfl_sync(ALL, f0, p), g1 = __shfl_sync(ALL, f1, p);
      int n = -1, fallback = size - 1;
      if (size <= FRONT && g1 - g0 <= 8) {  // a short part: link by link
        for (int f = g0; f < g1 && n < 0; f++) {
          const double w = F.w[f];
          if (bitsOf(w) == 0) continue;
          cum = dadd(cum, w);
          fallback = f;
          if (bitsOf(pick) <= bitsOf(cum)) n = f;
        }
      } else {
        for (int g = g0; g < g1 && n < 0; g += 32) {
          const int f = g + lane;
          double w = 0;
          if (f < FRONT && f < g1) w = F.w[f];
          else if (f < g1) w = weightOf(linkPj(F, L, f), linkInv(F, L, f), linkNode(F, L, f), linkTag(F, L, f), layer, ground, before, potential);
          double sum = w;
          for (int o = 1; o < 32; o <<= 1) { const double u = __shfl_up_sync(ALL, sum, o); if (lane >= o) sum = dadd(sum, u); }
          const double end = dadd(cum, sum);
          const unsigned hit = __ballot_sync(ALL, bitsOf(w) != 0 && bitsOf(pick) <= bitsOf(end)), any = __ballot_sync(ALL, bitsOf(w) != 0);
          if (hit) n = g + __ffs(hit) - 1;
          if (any) fallback = g + 31 - __clz(any);
          cum = __shfl_sync(ALL, end, 31);
        }
      }
      if (n < 0) n = fallback;  // (the last bits of two sums: the part's last link that counts)
      const int j = linkNode(F, L, n), from = linkFrom(F, L, n);
      const unsigned tag = linkTag(F, L, n);
      const double pj = linkPj(F, L, n);
      const bool clear = tag & TAG_CLEAR;
      __syncwarp();
      if (!left && ground < 0 && clear) {  // the first step out of the cloud
        if (lane == 0) { V.left = 1; V.event = 1; stop = 1; }
      } else {
        int m = size - 1;
        if (lane == 0) { L.pos[j] = -1; if (n != m) moveLink(F, L, n, m); }
        __syncwarp();
        if (tag & TAG_FROM_CLEAR) {
          // through clear air a leader does not branch: the other links from the same clear-air node leave the front
          for (int base = m - 1; base >= 0; base -= 32) {
            const int f = base - lane;
            unsigned match = __ballot_sync(ALL, f >= 0 && linkFrom(F, L, max(f, 0)) == from);
            for (; match; match &= match - 1) {
              const int at = base - (__ffs(match) - 1);
              m--;
              if (lane == 0) { L.pos[linkNode(F, L, at)] = -1; if (at != m) moveLink(F, L, at, m); }
              __syncwarp();
            }
          }
        }
        if (lane == 0) V.size = m;
        __syncwarp();
        addNodeWarp(R, L, F, V, j, nodes, from, clear, pj, id, next[iter & 1].n, next[iter & 1].inv);
        if (lane == 0 && V.touched) { V.touched = 0; V.event = 1; stop = 1; }
      }
    }
    __syncthreads();
    if (stop) break;
  }
  __syncthreads();
  for (int f = t; f < min(V.size, FRONT); f += GROW_THREADS) {
    L.frontier[f] = F.node[f]; L.link[f] = F.from[f]; L.tag[f] = F.tag[f]; L.scale[f] = F.inv[f];
  }
  if (t == 0) V.rng = rng;
  __syncthreads();
  stateOut(sh, L, t, GROW_THREADS);
}

// deposit() (:352-381) and neutralize() (:410-418) of one stage, one block: each channel node gets its capacitance
// times the potential difference, limited to neutralizing the charge there; before the ground contact both signs are
// scaled to the smaller (the channel stays neutral), after it the ground supplies the difference.
__global__ void __launch_bounds__(DEP_THREADS) k_lgt_deposit(const RunDesc R, const LgtDev L) {
  __shared__ double red[32];
  __shared__ double scaleP, scaleN;
  LgtState& S = *L.st;
  const int t = threadIdx.x, layer = R.layer, nn = S.nnodes, npol = S.npol;
  const bool grounded = S.ground >= 0;
  const double V = S.potential;
  const int C = (nn + DEP_THREADS - 1) / DEP_THREADS, c0 = min(nn, t * C), c1 = min(nn, c0 + C);
  double p = 0, q_ = 0, m = 0;
  for (int c = c0; c < c1; c++) {
    const int i = L.nodes[c], z = i / layer;
    double d = 0;
    if (z == 0) { if (c >= npol) L.polarity[c] = 0; }
    else {
      const double q = dmul(lt(L, LT_CAP, z), V - L.phi[i]), here = dmul(dmul(dmul(L.rho[i], L.dx), L.dy), lt(L, LT_HZ, z));
      if (c >= npol) L.polarity[c] = q > 0 ? 1 : q < 0 ? -1 : 0;
      if (dmul(q, here) < 0) {
        d = (q > 0 ? 1.0 : -1.0) * fmin(fabs(q), fabs(here));
        if (d > 0) p = dadd(p, d); else q_ = dadd(q_, -d);
      }
    }
    L.dep[c] = d;
  }
  const double P = blockSum(p, red), N = blockSum(q_, red);
  if (t == 0) {
    if (!grounded) {
      const double both = fmin(P, N);
      scaleP = P > 0 ? both / P : 0; scaleN = N > 0 ? both / N : 0;
      S.stage = both; S.neutralized = dadd(S.neutralized, both);
    } else {
      const double charge = N - P;
      scaleP = scaleN = 1;
      S.stage = charge; S.fromGround -= charge; S.lowered = dadd(S.lowered, charge);
      if (S.nstrokes < STROKES) S.strokeQ[S.nstrokes++] = charge;
    }
  }
  __syncthreads();
  for (int c = c0; c < c1; c++) {
    double d = L.dep[c];
    if (d == 0) continue;
    if (!grounded) d = dmul(d, d > 0 ? scaleP : scaleN);
    const int i = L.nodes[c], z = i / layer;
    if (grounded) m = dadd(m, dmul(d, lt(L, LT_ZS, z)));
    if (d == 0) continue;
    // neutralize: taken from the carriers of the opposite sign, in proportion to their charge
    const double perKg = d / lt(L, LT_NODEAIR, z), sq = d > 0 ? 1.0 : -1.0;
    float* cr[4] = {field(R, 0, CHARGE_ICE), field(R, 0, CHARGE_GRAUPEL), field(R, 0, CHARGE_RAIN), field(R, 0, CHARGE_AIR)};
    double opposite = 0;
    for (int k = 0; k < 4; k++) { const double v = cr[k][i]; if (dmul(v, d) < 0) opposite -= dmul(v, sq); }
    if (opposite <= 0) continue;
    for (int k = 0; k < 4; k++) {
      const double v = cr[k][i];
      if (dmul(v, d) < 0) cr[k][i] = (float)dadd(v, dmul(perKg, fabs(v)) / opposite);
    }
  }
  const double M = grounded ? blockSum(m, red) : 0;
  if (t == 0) {
    if (grounded) { S.moment -= M; S.strokes++; }
    S.npol = nn;
    S.needPotential = !grounded;  // after the next solve the neutral channel's potential is the mean of its nodes' (:338)
  }
}

// The end of a flash: the run's counts and charge budget (:1543), or, for a breakdown that neutralized nothing, the node
// left out for the rest of the step (:270).
__global__ void k_lgt_flash_end(const RunDesc R, const LgtDev L, int stamp) {
  if (threadIdx.x || blockIdx.x) return;
  LgtState& S = *L.st;
  const bool cg = S.ground >= 0;
  const double charge = cg ? S.lowered : S.neutralized;
  S.charge = charge;
  if (charge == 0) { L.failed[S.start] = stamp; return; }
  if (cg) {
    R.acc[A_CHG_GROUND] += charge; R.acc[A_FLASH_CG] += 1;
    if (charge < 0) R.acc[A_CHG_CG_NEG] += charge; else R.acc[A_CHG_CG_POS] += charge;
  } else { R.acc[A_FLASH_IC] += 1; R.acc[A_CHG_IC] += fabs(charge); }
}

// ---------------------------------------------------------------- conduction and corona (:185-223)
// Per interior node, the charge through its six faces over dt (a face's conductance the harmonic mean of its two nodes'
// in series, one of a few a level: clear air or cloud on either side; the ground and top take what reaches them) and, on
// the lowest interior level, the corona from the ground; the ion carrier takes it. And the vertical field of the last
// solve (:1550-1551). The charge the air lost to the ground, the top and the corona is summed over the blocks (in a fixed
// order, by the block that ends last) into the run's budget.
__global__ void __launch_bounds__(256) k_lgt_conduct(const RunDesc R, const LgtDev L, int corona, double dt) {
  __shared__ double red[32];
  const int nx = R.nx, ny = R.ny, nz = R.nz, layer = R.layer;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + layer;
  double lost = 0;
  if (i < R.n - layer) {
    const int z = i / layer, y = (i - z * layer) / nx, x = i - z * layer - y * nx;
    const int xp = x + 1 == nx ? 0 : x + 1, xm = x == 0 ? nx - 1 : x - 1, yp = y + 1 == ny ? 0 : y + 1, ym = y == 0 ? ny - 1 : y - 1;
    const double* phi = L.phi;
    const int ixp = xp + y * nx + z * layer, ixm = xm + y * nx + z * layer, iyp = x + yp * nx + z * layer, iym = x + ym * nx + z * layer;
    const bool here = cloudAt(L.cloudy[i]);
    auto flat = [&](int j) { return lt(L, LT_FLAT + (here ? 1 : 0) + (cloudAt(L.cloudy[j]) ? 1 : 0), z); };          // in the level
    auto step = [&](int zb, bool b, bool a) { return lt(L, LT_STEP + (b ? 1 : 0) + (a ? 2 : 0), zb); };                // level zb to the next
    const double across = lt(L, LT_ACROSS, z), along = lt(L, LT_ALONG, z), p = phi[i];
    const double qxo = dmul(dmul(flat(ixp), p - phi[ixp]), across), qyo = dmul(dmul(flat(iyp), p - phi[iyp]), along);
    const double qxi = dmul(dmul(flat(ixm), phi[ixm] - p), across), qyi = dmul(dmul(flat(iym), phi[iym] - p), along);
    const double pd = phi[i - layer], pu = phi[i + layer];
    const double qb = dmul(dmul(step(z - 1, cloudAt(L.cloudy[i - layer]), here), pd - p), lt(L, LT_UP, z - 1));
    const double qa = dmul(dmul(step(z, here, cloudAt(L.cloudy[i + layer])), p - pu), lt(L, LT_UP, z));
    double change = -dadd(qxo, qyo);
    change = dadd(dadd(change, qxi), qyi);
    change = dadd(dadd(change, qb), -qa);
    if (z == 1) {
      lost -= qb;
      if (corona) {
        const double e0 = -p / lt(L, LT_DZS, 0), over = fabs(e0) - CORONA_FIELD;
        if (over > 0) {
          const double qc = dmul(dmul(dmul(dmul((e0 > 0 ? 1.0 : -1.0) * CORONA_RATE, over), L.dx), L.dy), dt);
          change = dadd(change, qc); lost -= qc;
        }
      }
    }
    if (z == nz - 2) lost += qa;
    if (!isZero(change)) {
      float* air = field(R, 0, CHARGE_AIR);
      air[i] = (float)dadd((double)air[i], dmul(change, lt(L, LT_PERKG, z)));
    }
    R.ez[i] = (float)-dmul(pu - pd, lt(L, LT_ISPAN, z));
  }
  lost = blockSum(lost, red);
  if (threadIdx.x == 0) L.part[blockIdx.x] = lost;
  if (!lastBlock(&L.st->arrived)) return;
  double all = 0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) all = dadd(all, __ldcg(L.part + b));
  all = blockSum(all, red);
  if (threadIdx.x == 0) { L.st->arrived = 0; L.st->conducted += all; R.acc[A_CHG_GROUND] += all; R.acc[A_CHG_CONDUCTION] += all; }
}

__global__ void k_lgt_seed(const LgtDev L, uint32_t rng) {
  if (threadIdx.x == 0 && blockIdx.x == 0) { L.st->rng = rng; L.st->maxBits = 0; L.st->best = INT_MAX; }
}

inline int blocks(int n, int t) { return (n + t - 1) / t; }

}  // namespace

// ---------------------------------------------------------------- host side
size_t lightning_bytes(int nx, int ny, int nz) {
  const size_t n = (size_t)nx * ny * nz, mh = nx / 2, spec = (size_t)(nz - 2) * (mh + 1) * ny;
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  return al(sizeof(LgtState)) + 4 * al(n * 8) + al(n * 4) + 7 * al(n * 4) + 4 * al((size_t)MAX_CHANNEL * 8) +
         al((size_t)LT_COUNT * nz * 8) + al(((n + 255) / 256 + 1) * 8) + al(((n + 255) / 256 + 1) * 4) + al(spec * 16) + 3 * al(spec * 8) +
         al((size_t)nx * 16) + al((size_t)ny * 16);
}

void lightning_bind(char* base, int nx, int ny, int nz, LgtHost& H) {
  LgtDev& L = H.dev;
  const size_t n = (size_t)nx * ny * nz, mh = nx / 2, spec = (size_t)(nz - 2) * (mh + 1) * ny;
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  size_t o = 0;
  auto take = [&](size_t b) { char* p = base + o; o += al(b); return p; };
  L.nz = nz;
  L.st = (LgtState*)take(sizeof(LgtState));
  L.rho = (double*)take(n * 8); L.phi = (double*)take(n * 8);
  L.weight = (double*)take(n * 8); L.scale = (double*)take(n * 8);
  L.cloudy = (float*)take(n * 4);
  L.pos = (int*)take(n * 4); L.tag = (unsigned*)take(n * 4);
  L.mark = (int*)take(n * 4); L.seen = (int*)take(n * 4); L.link = (int*)take(n * 4); L.failed = (int*)take(n * 4); L.frontier = (int*)take(n * 4);
  L.nodes = (int*)take(MAX_CHANNEL * 8); L.parent = (int*)take(MAX_CHANNEL * 8); L.polarity = (int*)take(MAX_CHANNEL * 8);
  L.dep = (double*)take(MAX_CHANNEL * 8);
  L.lv = (double*)take((size_t)LT_COUNT * nz * 8);
  L.part = (double*)take(((n + 255) / 256 + 1) * 8); L.partAt = (int*)take(((n + 255) / 256 + 1) * 4);
  H.es.shape(nx, ny, nz - 2);
  H.es.S = (double2*)take(spec * 16);
  H.es.a = (double*)take(spec * 8); H.es.b = (double*)take(spec * 8); H.es.c = (double*)take(spec * 8);
  H.es.twx = (double2*)take((size_t)nx * 16); H.es.twy = (double2*)take((size_t)ny * 16);
}

int lightning_init(cudaStream_t st, const sg_grid* g, const double* rho, LgtHost& H) {
  const int nx = g->nx, ny = g->ny, nz = g->nz;
  LgtDev& L = H.dev;
  L.dx = g->dx; L.dy = g->dy; L.i2dx = 1 / (2 * g->dx); L.i2dy = 1 / (2 * g->dy);
  // per-level tables in FP64, each the reference's expression
  std::vector<double> lv((size_t)LT_COUNT * nz, 0.0);
  auto T = [&](int w, int z, double v) { lv[(size_t)w * nz + z] = v; };
  const double dx = g->dx, dy = g->dy;
  for (int z = 0; z < nz; z++) {
    const double h = g->hz[z], e = E_INIT * rho[z] / RHO_STANDARD, Lc = std::cbrt(dx * dy * h);
    T(LT_AIR, z, rho[z]); T(LT_ZS, z, g->zs[z]);
    T(LT_CAP, z, SHIELDING * 2 * 3.14159265358979323846 * EPS0 * Lc / std::log(Lc / CHANNEL_RADIUS));        // :179
    T(LT_NODEAIR, z, rho[z] * dx * dy * h); T(LT_PERKG, z, 1 / (rho[z] * dx * dy * h));
    T(LT_DZS, z, z < nz - 1 ? g->dzs[z] : 0);
    T(LT_HZ, z, h);
    T(LT_ISPAN, z, z > 0 && z < nz - 1 ? 1 / (g->zs[z + 1] - g->zs[z - 1]) : 1); T(LT_IEINIT2, z, 1 / std::pow(e, 2));
    // conductances in series between nodes of clear air or cloud, in the level (clear-clear, clear-cloud, cloud-cloud) and
    // to the next level (bit 1 cloud below, bit 2 cloud above)
    auto series = [](double a, double b) { return 2 * a * b / (a + b); };
    auto sigma = [&](int k, bool cloud) { const double c = SIGMA_GROUND * std::exp(g->zs[k] / SIGMA_SCALE); return cloud ? c * CLOUD_SIGMA : c; };
    for (int q = 0; q < 3; q++) T(LT_FLAT + q, z, series(sigma(z, q > 1), sigma(z, q > 0)));
    for (int q = 0; q < 4 && z < nz - 1; q++) T(LT_STEP + q, z, series(sigma(z, q & 1), sigma(z + 1, q & 2)));
    // a link's reach from level z to level z - 1, z, z + 1 by |di| + 2 |dj|: its length times the propagation threshold
    // (:389-404), each operation rounded by itself as on the device (no contraction), and its reciprocal
    for (int kk = 0; kk < 3; kk++) {
      const int k = z + kk - 1;
      if (k < 0 || k >= nz) continue;
      for (int q = 0; q < 4; q++) {
        const double hz = g->zs[k] - g->zs[z], e2 = E_INIT * rho[k] / RHO_STANDARD;
        const volatile double a2 = q & 1 ? dx * dx : 0, b2 = q & 2 ? dy * dy : 0, h2 = hz * hz, es = e + e2;
        const volatile double ab = a2 + b2, abh = ab + h2, threshold = F_CRIT * .5 * es;
        const double s = std::sqrt((double)abh) * threshold;
        T(LT_REACH + kk * 4 + q, z, s); T(LT_IREACH + kk * 4 + q, z, s > 0 ? 1 / s : 0);
      }
    }
  }
  H.conductDt = 0;
  H.tables = lv;
  std::vector<double> a, b, c;
  std::vector<double2> tx, ty;
  elec_host_tables(H.es, dx, dy, g->dzs, g->hz, a, b, c, tx, ty);
  cudaError_t e;
  if ((e = spectral64_limits()) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_lgt_grow, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)front_bytes(128))) != cudaSuccess || (e = cudaMemcpyAsync(L.lv, lv.data(), lv.size() * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(H.es.a, a.data(), a.size() * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(H.es.b, b.data(), b.size() * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(H.es.c, c.data(), c.size() * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(H.es.twx, tx.data(), tx.size() * 16, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(H.es.twy, ty.data(), ty.size() * 16, cudaMemcpyHostToDevice, st)) != cudaSuccess)
    return (int)e;
  H.dxy = dx * dy;
  return 0;
}

// The conduction tables depend on dt (across = dy hz dt / dx, along, up = dx dy dt / dzs: :192).
static cudaError_t conduct_tables(cudaStream_t st, const sg_grid* g, LgtHost& H, double dt) {
  if (H.conductDt == dt) return cudaSuccess;
  const int nz = g->nz;
  const double dx = g->dx, dy = g->dy;
  for (int z = 0; z < nz; z++) {
    H.tables[(size_t)LT_ACROSS * nz + z] = dy * g->hz[z] * dt / dx;
    H.tables[(size_t)LT_ALONG * nz + z] = dx * g->hz[z] * dt / dy;
    H.tables[(size_t)LT_UP * nz + z] = z < nz - 1 ? dx * dy * dt / g->dzs[z] : 0;
  }
  H.conductDt = dt;
  return cudaMemcpyAsync(H.dev.lv, H.tables.data(), H.tables.size() * 8, cudaMemcpyHostToDevice, st);
}

static cudaError_t read_state(cudaStream_t st, const LgtHost& H, LgtState& S) {
  cudaError_t e = cudaMemcpyAsync(&S, H.dev.st, sizeof(LgtState), cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) return e;
  return cudaStreamSynchronize(st);
}

int lightning_state(cudaStream_t st, LgtHost& H, double* out) {
  LgtState S{};
  if (read_state(st, H, S) != cudaSuccess) return SG_ERR_DEVICE;
  const double v[16] = {(double)S.id, (double)S.start, (double)S.size, (double)S.nnodes, (double)S.ground, (double)S.event, (double)S.left,
                        (double)S.strokes, (double)S.grown, S.potential, S.sum, S.neutralized, S.lowered, S.stage, S.charge, (double)H.flashId};
  for (int k = 0; k < 16; k++) out[k] = v[k];
  return SG_OK;
}

int lightning_probe(cudaStream_t st, const RunDesc& R, LgtHost& H, double* phi, double* rho, int* best, double* ratio) {
  const LgtDev& L = H.dev;
  const int nb = blocks(R.n, 256), ni = blocks(R.n - 2 * R.layer, 256);
  k_lgt_cloudy<<<nb, 256, 0, st>>>(R, L);
  k_lgt_rho<<<nb, 256, 0, st>>>(R, L);
  elec_solve_launch(H.es, L.rho, L.phi, st);
  k_lgt_strongest<<<ni, 256, 0, st>>>(R, L, -1);
  LgtState S{};
  cudaError_t e;
  if (read_state(st, H, S) != cudaSuccess) return SG_ERR_DEVICE;
  if (phi && (e = cudaMemcpyAsync(phi, L.phi, (size_t)R.n * 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return SG_ERR_DEVICE;
  if (rho && (e = cudaMemcpyAsync(rho, L.rho, (size_t)R.n * 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return SG_ERR_DEVICE;
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess) return SG_ERR_DEVICE;
  double r2;
  std::memcpy(&r2, &S.maxBits, sizeof(double));
  *best = S.maxBits ? S.best : -1;
  *ratio = S.maxBits ? std::sqrt(r2) : 0;
  return SG_OK;
}

LgtHost::~LgtHost() {
  if (st) { cudaStreamSynchronize(st); cudaStreamDestroy(st); }
  if (hs) cudaFreeHost(hs);
  if (hchan) cudaFreeHost(hchan);
}

int lightning_host_buffers(LgtHost& H) {
  if (!H.st && cudaStreamCreateWithFlags(&H.st, cudaStreamNonBlocking) != cudaSuccess) return SG_ERR_DEVICE;
  if (!H.hs && cudaMallocHost(&H.hs, sizeof(LgtState)) != cudaSuccess) return SG_ERR_DEVICE;
  if (!H.hchan && cudaMallocHost(&H.hchan, 3 * (size_t)MAX_CHANNEL * sizeof(int)) != cudaSuccess) return SG_ERR_DEVICE;
  return SG_OK;
}

namespace {

// The search of pass k of Discharge (:264-268): the charge density and its field, then the strongest field; at the pass
// after the last flash allowed, the conduction and the vertical field instead (:1547-1551).
void launch_finish(const LgtJob& J) {
  const int ni = blocks(J.R.n - 2 * J.R.layer, 256);
  k_lgt_conduct<<<ni, 256, 0, J.H->st>>>(J.R, J.H->dev, J.H->corona ? 1 : 0, J.dt);
}
void launch_search(LgtJob& J) {
  const LgtDev& L = J.H->dev;
  const int nb = blocks(J.R.n, 256), ni = blocks(J.R.n - 2 * J.R.layer, 256);
  cudaStream_t st = J.H->st;
  k_lgt_rho<<<nb, 256, 0, st>>>(J.R, L);
  elec_solve_launch(J.H->es, L.rho, L.phi, st);
  if (J.k == J.limit) { launch_finish(J); J.phase = LgtJob::FINISHING; return; }
  k_lgt_strongest<<<ni, 256, 0, st>>>(J.R, L, J.stamp);
  J.phase = LgtJob::SEARCH;
}
void launch_stage(LgtJob& J, int start) {  // start: a new flash's first node, -1 for its later stages
  k_lgt_grow<<<1, GROW_THREADS, front_bytes(J.R.nz), J.H->st>>>(J.R, J.H->dev, J.id, start);
  k_lgt_deposit<<<1, DEP_THREADS, 0, J.H->st>>>(J.R, J.H->dev);
  J.stage++;
}

// Advances a job by what its last round's state record says (Lightning.discharge and .flash, :259-340).
cudaError_t advance(LgtJob& J) {
  LgtHost& H = *J.H;
  const LgtState& S = *H.hs;
  cudaError_t e = cudaSuccess;
  if (J.pending) {  // the flash that ended last round: its record (its channel was copied behind flash_end)
    J.pending = false;
    if (S.charge != 0) {
      FlashRecord f;
      f.time = J.time; f.cg = S.ground >= 0; f.start = J.start; f.ground = S.ground; f.charge = S.charge;
      f.potential = S.ground >= 0 ? S.before : S.potential; f.moment = S.ground >= 0 ? S.moment : 0;
      f.strokes.assign(S.strokeQ, S.strokeQ + (S.ground >= 0 ? S.nstrokes : 0));
      const int m = J.copied;
      f.nodes.assign(H.hchan, H.hchan + m); f.parent.assign(H.hchan + MAX_CHANNEL, H.hchan + MAX_CHANNEL + m);
      f.polarity.assign(H.hchan + 2 * MAX_CHANNEL, H.hchan + 2 * MAX_CHANNEL + m);
      H.last.push_back(std::move(f));
    }
  }
  switch (J.phase) {
    case LgtJob::SEARCH: {
      double r2;
      std::memcpy(&r2, &S.maxBits, sizeof(double));
      if (S.maxBits == 0 || !(std::sqrt(r2) > 1)) { launch_finish(J); J.phase = LgtJob::DONE; break; }
      J.start = S.best; J.id = ++H.flashId; J.stage = 0;
      launch_stage(J, J.start);
      J.phase = LgtJob::FLASH;
      break;
    }
    case LgtJob::FLASH: {
      const bool end = (S.ground >= 0 && (S.strokes >= STROKES || (!S.event && S.nnodes == S.grown))) || (S.ground < 0 && !S.event) ||
                       S.nnodes >= MAX_CHANNEL || J.stage >= STROKES + 8;
      if (!end) {
        // the field of the charge as it now stands; before the contact the channel stays neutral on it
        k_lgt_rho<<<blocks(J.R.n, 256), 256, 0, H.st>>>(J.R, H.dev);
        elec_solve_launch(H.es, H.dev.rho, H.dev.phi, H.st);
        launch_stage(J, -1);
        break;
      }
      k_lgt_flash_end<<<1, 32, 0, H.st>>>(J.R, H.dev, J.stamp);
      J.copied = S.nnodes;
      if ((e = cudaMemcpyAsync(H.hchan, H.dev.nodes, (size_t)S.nnodes * 4, cudaMemcpyDeviceToHost, H.st)) != cudaSuccess ||
          (e = cudaMemcpyAsync(H.hchan + MAX_CHANNEL, H.dev.parent, (size_t)S.nnodes * 4, cudaMemcpyDeviceToHost, H.st)) != cudaSuccess ||
          (e = cudaMemcpyAsync(H.hchan + 2 * MAX_CHANNEL, H.dev.polarity, (size_t)S.nnodes * 4, cudaMemcpyDeviceToHost, H.st)) != cudaSuccess)
        return e;
      J.pending = true;
      J.k++;
      launch_search(J);
      break;
    }
    case LgtJob::FINISHING: J.phase = LgtJob::DONE; break;
    case LgtJob::DONE: break;
  }
  return e;
}

}  // namespace

// The discharges of several runs side by side, each on its own stream: whenever a run's stream has done its piece of work
// (a search, a flash stage, the end of a flash and the next search, the conduction) its state record is read and its next
// piece launched, so the runs' single-block channel growths overlap and no run waits for another's (in lockstep rounds
// every piece took as long as the longest run's: 6.4 ms a step for 16 storms, 4.1 now).
int lightning_discharge_many(LgtJob* jobs, int n, std::string* err) {
  cudaError_t e = cudaSuccess;
  for (int j = 0; j < n; j++) {
    LgtJob& J = jobs[j];
    LgtHost& H = *J.H;
    if ((e = conduct_tables(H.st, J.g, H, J.dt)) != cudaSuccess) { *err = cudaGetErrorString(e); return SG_ERR_DEVICE; }
    H.last.clear();
    J.stamp = ++H.flashId; J.k = 0; J.pending = false;
    // the random numbers start afresh from the seed and the model time (:263)
    const int32_t tenths = (int32_t)(int64_t)std::floor(J.time * 10 + .5);
    k_lgt_seed<<<1, 32, 0, H.st>>>(H.dev, H.seed ^ (uint32_t)((uint32_t)tenths * 0x9E3779B1u));
    k_lgt_cloudy<<<blocks(J.R.n, 256), 256, 0, H.st>>>(J.R, H.dev);
    launch_search(J);
  }
  auto read = [&](LgtJob& J) { return cudaMemcpyAsync(J.H->hs, J.H->dev.st, sizeof(LgtState), cudaMemcpyDeviceToHost, J.H->st); };
  for (int j = 0; j < n && e == cudaSuccess; j++) e = read(jobs[j]);
  if (e == cudaSuccess) e = cudaGetLastError();
  std::vector<int> pieces(n, 0);
  int left = n;
  while (left > 0 && e == cudaSuccess) {
    for (int j = 0; j < n && e == cudaSuccess; j++) {
      LgtJob& J = jobs[j];
      if (J.phase == LgtJob::DONE) continue;
      e = cudaStreamQuery(J.H->st);
      if (e == cudaErrorNotReady) { cudaGetLastError(); e = cudaSuccess; continue; }  // (not an error: cleared)
      if (e == cudaSuccess) e = advance(J);
      if (J.phase == LgtJob::DONE) left--;
      else if (e == cudaSuccess) {
        // every flash has at most STROKES + 9 stages and its end, every pass a search
        if (++pieces[j] > std::max(8, (J.limit + 2) * (STROKES + 12))) { *err = "a discharge did not end within its bound of rounds"; return SG_ERR_DEVICE; }
        e = read(J);
      }
      if (e == cudaSuccess) e = cudaGetLastError();
    }
  }
  for (int j = 0; j < n && e == cudaSuccess; j++) e = cudaStreamSynchronize(jobs[j].H->st);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) { *err = cudaGetErrorString(e); return SG_ERR_DEVICE; }
  return SG_OK;
}

int lightning_discharge(cudaStream_t, const sg_grid* g, const RunDesc& R, LgtHost& H, double time, double dt, int limit, std::string* err) {
  LgtJob J;
  J.g = g; J.R = R; J.H = &H; J.time = time; J.dt = dt; J.limit = limit;
  return lightning_discharge_many(&J, 1, err);
}

}  // namespace sg
