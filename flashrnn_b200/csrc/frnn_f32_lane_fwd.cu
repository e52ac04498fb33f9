// Instantiations of the float32 forward lane loop.
#ifndef FRNN_F16  // compiled once, into the bfloat16 build, which owns the public entry points
#include "frnn_f32_lane.cuh"

namespace FRNN_NS {
namespace {
template <int CELL, bool CL, int LPU, int KQ, int BT> XLane make(int U) {
  const int warps = (U * LPU + 31) / 32;
  return XLane{reinterpret_cast<const void*>(&x32l_fwd_kernel<CELL, CL, LPU, KQ, BT>), 32 * warps + kXIo, BT, XFwdGeom<CELL, CL, LPU, KQ, BT>::smem(U)};
}
// k quads per lane, from 4 * KQ * LPU units up (of which Elman's four-unit groups need a quarter)
template <int CELL, bool CL, int LPU, int KQ, int BT> XLane quads(int U) { return make<CELL, CL, LPU, (Cell<CELL>::Gr > 1 ? KQ : KQ > 4 ? KQ / 4 : 1), BT>(U); }
template <int CELL> XLane pick(int D, int U, int bt) {
  if (D <= 32) return bt == 1 ? quads<CELL, false, 2, 4, 1>(U) : bt == 2 ? quads<CELL, false, 2, 4, 2>(U) : quads<CELL, false, 4, 2, 4>(U);
  if (D <= 64) return bt == 1 ? quads<CELL, false, 2, 8, 1>(U) : bt == 2 ? quads<CELL, false, 2, 8, 2>(U) : quads<CELL, false, 4, 4, 4>(U);
  if (D <= 128) return bt <= 2 ? quads<CELL, true, 4, 8, 2>(U) : bt == 4 ? quads<CELL, true, 4, 8, 4>(U) : quads<CELL, true, 8, 4, 8>(U);
  return bt <= 2 ? quads<CELL, true, 8, 8, 2>(U) : bt == 4 || Cell<CELL>::Gr > 1 ? quads<CELL, true, 8, 8, 4>(U) : quads<CELL, true, 8, 8, (Cell<CELL>::Gr > 1 ? 4 : 8)>(U);
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
