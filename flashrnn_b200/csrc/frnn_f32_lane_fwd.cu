// Instantiations of the float32 forward lane loop.
#ifndef FRNN_F16  // compiled once, into the bfloat16 build, which owns the public entry points
#include "frnn_f32_lane.cuh"

namespace FRNN_NS {
namespace {
template <int CELL, int KQ, int BT> XLane make(int U) {
  return XLane{reinterpret_cast<const void*>(&x32l_fwd_kernel<CELL, KQ, BT>), 8 * U + kXIo, BT, XFwdGeom<CELL, KQ, BT>::smem(U)};
}
// k quads per lane: D / 32, rounded up to a power of two (padded with zeros).  Clusters take 2 rows at least, and no more from KQ = 8
// on, whose part of R leaves no registers for them.
template <int CELL> XLane pick(int D, int U, int bt) {
  if (D <= 32) return bt == 1 ? make<CELL, 1, 1>(U) : bt == 2 ? make<CELL, 1, 2>(U) : make<CELL, 1, 4>(U);
  if (D <= 64) return bt == 1 ? make<CELL, 2, 1>(U) : bt == 2 ? make<CELL, 2, 2>(U) : make<CELL, 2, 4>(U);
  if (D <= 128) return bt <= 2 ? make<CELL, 4, 2>(U) : make<CELL, 4, 4>(U);
  return make<CELL, 8, 2>(U);
}
}  // namespace

XLane x32_lane_fwd(int cell, int D, int U, int bt) {
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
