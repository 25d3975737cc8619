// The transport kernel's item (sg_transport.cu, cut out by the test as transport_item.inc) run block by block on the
// CPU: see block_emulator.h.
#include "block_emulator.h"
#include "../../meteolab_gb300/csrc/sg_common.cuh"

namespace sg {
constexpr int MAXNZ = 128;
enum TKind { TK_WENO = 0, TK_DYN = 1 };
#include "transport_item.inc"
}  // namespace sg

using namespace sg;

// One stage (start set 0, input set `in`, output set 2) of a run's fields `fld` (three sets of the base fields), every
// column cut into `slabs` slabs of levels, the threads of each block in the scheduler's order `order`, the copies landing
// `late` or early. 0, or -1 where a block's threads wait forever.
extern "C" int tb_transport(int kind, int G, int ew, int TX, int TY, int nx, int ny, int nz, int slabs, int order, int late, int flags, int in, int stage,
                            float* fld, float* faces, const float* lv) {
  RunDesc R{};
  R.nx = nx; R.ny = ny; R.nz = nz; R.layer = nx * ny; R.n = nx * ny * nz; R.flags = flags;
  R.dt = 3.f; R.inv_dx = 1e-3f; R.inv_dy = 9e-4f; R.fld = fld; R.faces = faces; R.lv = lv;
  const size_t floats = (size_t)tlv_rows(kind) * MAXNZ + 8 * (size_t)TX * TY + (size_t)G * 7 * (TX + 6) * (TY + 6) + 2 * (size_t)G * TY * (TX + 1) +
                        2 * (size_t)G * (TY + 1) * TX;
  std::vector<float4> shared(floats / 4 + 1);
  const int tiles = ((nx + TX - 1) / TX) * ((ny + TY - 1) / TY), threads = TX * TY + (ew ? TEDGE : 0);
  for (int tile = 0; tile < tiles; tile++)
    for (int s = 0; s < slabs; s++) {
      const int levels = (nz * s / slabs) | (nz * (s + 1) / slabs) << 16;
      float* sm = reinterpret_cast<float*>(shared.data());
      std::fill(sm, sm + floats, NAN);  // (what a block has not written is not read)
      const bool ended = emu::run(threads, order, [&] {
        if (kind == TK_DYN) transport_item<TK_DYN, 4, 0, 0, false>(R, 3, tile, levels, in, 2, .5f, stage, TX, TY, sm);
        else if (G == 3 && ew) transport_item<TK_WENO, 3, 0, 0, true>(R, 0, tile, levels, in, 2, .5f, stage, TX, TY, sm);
        else if (G == 3) transport_item<TK_WENO, 3, 0, 0, false>(R, 0, tile, levels, in, 2, .5f, stage, TX, TY, sm);
        else transport_item<TK_WENO, 1, 0, 0, false>(R, 4, tile, levels, in, 2, .5f, stage, TX, TY, sm);
      }, late != 0);
      if (!ended) return -1;
    }
  return 0;
}
