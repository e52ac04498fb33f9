// Instantiations of the float32 reverse lane loop.
#ifndef FRNN_F16  // compiled once, into the bfloat16 build, which owns the public entry points
#include "frnn_f32_lane.cuh"

namespace FRNN_NS {
namespace {
template <int CELL, int KS, int KQ, int TB, int BT> XLane make(int D, int U) {
  return XLane{reinterpret_cast<const void*>(&x32l_bwd_kernel<CELL, KS, KQ, TB, BT>), 8 * U + kXIo, BT, XBwdGeom<CELL, KS, KQ, TB, BT>::smem(U, D / U)};
}
// One CTA per head: Gr * U / 4 quads of k over 32 lanes.  Clusters (U <= 32): Gr * 8 quads at most over 8 lanes, D / 16 column tasks over
// U / 4 warps.
template <int CELL> XLane pick(int D, int U, int bt) {
  constexpr int Gr = Cell<CELL>::Gr;
  if (D == U) {
    if (Gr == 1 || Gr * U / 4 <= 32) return bt == 1 ? make<CELL, 32, 1, 1, 1>(D, U) : bt == 2 ? make<CELL, 32, 1, 1, 2>(D, U) : make<CELL, 32, 1, 1, 4>(D, U);
    if constexpr (Gr > 1) return bt == 1 ? make<CELL, 32, 2, 1, 1>(D, U) : bt == 2 ? make<CELL, 32, 2, 1, 2>(D, U) : make<CELL, 32, 2, 1, 4>(D, U);
  }
  if ((D + 15) / 16 <= U / 4) return bt <= 2 ? make<CELL, 8, Gr, 1, 2>(D, U) : make<CELL, 8, Gr, 1, 4>(D, U);
  if ((D + 15) / 16 <= 2 * (U / 4)) return make<CELL, 8, Gr, 2, 2>(D, U);
  return XLane{nullptr, 0, 0, 0};
}
}  // namespace

XLane x32_lane_bwd(int cell, int D, int U, int bt) {
  switch (cell) {
    case CELL_LSTM: return pick<CELL_LSTM>(D, U, bt);
    case CELL_GRU: return pick<CELL_GRU>(D, U, bt);
    case CELL_ELMAN: return pick<CELL_ELMAN>(D, U, bt);
    case CELL_ELMAN_CLIP: return pick<CELL_ELMAN_CLIP>(D, U, bt);
    case CELL_SLSTM: return pick<CELL_SLSTM>(D, U, bt);
  }
  return XLane{nullptr, 0, 0, 0};
}

}  // namespace FRNN_NS
#endif  // FRNN_F16
