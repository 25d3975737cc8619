// The growth of a lightning channel (k_lgt_grow of sg_lightning.cu, cut out by the test as lightning_helpers.inc and
// lightning_grow.inc) run as one block on the CPU: see block_emulator.h.
#include <climits>
#include <map>
#include <string>
#include "block_emulator.h"
#include "../../meteolab_gb300/csrc/sg_lightning.h"

static std::vector<double> dynamic_shared;
namespace sg {
namespace {
#include "lightning_helpers.inc"
#include "lightning_grow.inc"
}  // namespace
}  // namespace sg

using namespace sg;

// `stages` stages of one flash from node `start`, stage s on the potential phi[s], with what the deposit does between two
// stages to a channel that has not touched the ground; the threads in the scheduler's order `order`. out: the channel's
// nodes, then their parents (MAX_CHANNEL each); state: nodes, front, ground, left, random state, potential, sum. The largest
// front any stage ends with, or -1 where the threads wait forever.
extern "C" int lb_flash(int nx, int ny, int nz, double dx, double dy, const double* zs, const double* air, double* rho, double* phi, float* cloudy,
                        int stages, int start, unsigned seed, int order, int* out, double* state) {
  RunDesc R{};
  R.nx = nx; R.ny = ny; R.nz = nz; R.layer = nx * ny; R.n = nx * ny * nz;
  LgtDev L;
  LgtState S{};
  const size_t n = (size_t)R.n;
  std::vector<double> weight(n), scale(n), lv((size_t)LT_COUNT * nz);
  std::vector<int> pos(n), mark(n), seen(n), link(n), frontier(n), nodes(2 * MAX_CHANNEL), parent(2 * MAX_CHANNEL);
  std::vector<unsigned> tag(n);
  for (int z = 0; z < nz; z++)
    for (int kk = 0; kk < 3; kk++) {
      const int k = z + kk - 1;
      if (k < 0 || k >= nz) continue;
      for (int q = 0; q < 4; q++) {
        const double h = zs[k] - zs[z], e = E_INIT / RHO_STANDARD * (air[z] + air[k]) * F_CRIT * .5;
        const double s = std::sqrt((q & 1 ? dx * dx : 0) + (q & 2 ? dy * dy : 0) + h * h) * e;
        lv[(size_t)(LT_REACH + kk * 4 + q) * nz + z] = s; lv[(size_t)(LT_IREACH + kk * 4 + q) * nz + z] = s > 0 ? 1 / s : 0;
      }
    }
  L.nz = nz; L.dx = dx; L.dy = dy; L.st = &S; L.rho = rho; L.weight = weight.data(); L.scale = scale.data(); L.cloudy = cloudy;
  L.pos = pos.data(); L.tag = tag.data(); L.mark = mark.data(); L.seen = seen.data(); L.link = link.data(); L.frontier = frontier.data();
  L.nodes = nodes.data(); L.parent = parent.data(); L.lv = lv.data();
  S.rng = seed;
  dynamic_shared.assign(front_bytes(nz) / 8 + 1, NAN);
  int largest = 0;
  for (int s = 0; s < stages; s++) {
    L.phi = phi + s * n;
    if (!emu::run(GROW_THREADS, order, [&] { k_lgt_grow(R, L, 7, s == 0 ? start : -1); })) return -1;
    S.npol = S.nnodes; S.needPotential = S.ground < 0;
    largest = std::max(largest, S.size);
  }
  std::copy(nodes.begin(), nodes.begin() + MAX_CHANNEL, out);
  std::copy(parent.begin(), parent.begin() + MAX_CHANNEL, out + MAX_CHANNEL);
  const double v[7] = {(double)S.nnodes, (double)S.size, (double)S.ground, (double)S.left, (double)S.rng, S.potential, S.sum};
  std::copy(v, v + 7, state);
  return largest;
}

// how many of sum[i] / (i % MAX_CHANNEL + 1) the mean from the count's reciprocal does not give to the last bit
extern "C" int lb_means(const double* sum, int n) {
  int wrong = 0;
  for (int i = 0; i < n; i++) {
    const double count = i % MAX_CHANNEL + 1;
    wrong += emu::bits(meanOf(sum[i], count, 1.0 / count)) != emu::bits(sum[i] / count);
  }
  return wrong;
}
