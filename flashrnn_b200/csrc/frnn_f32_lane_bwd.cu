// Instantiations of the float32 reverse lane loop.
#ifndef FRNN_F16  // compiled once, into the bfloat16 build, which owns the public entry points
#include "frnn_f32_lane.cuh"

namespace FRNN_NS {
namespace {
template <int CELL, bool CL, int LPU, int KQ, int TB, int BT> XLane make(int D, int U) {
  const int warps = (U * LPU + 31) / 32;
  return XLane{reinterpret_cast<const void*>(&x32l_bwd_kernel<CELL, CL, LPU, KQ, TB, BT>), 32 * warps + kXIo, BT,
               XBwdGeom<CELL, CL, LPU, KQ, TB, BT>::smem(U, D / U)};
}
// One CTA per head: Gr * U / 4 quads of k over 4 LPU lanes (KQ of them each with 64 units, half of it up to 32)
template <int CELL, int LPU, int BT> XLane single(int D) {
  constexpr int KQ = Cell<CELL>::Gr == 1 ? 4 / LPU : 16 / LPU;  // (of the GRU, three quarters are not zero)
  if constexpr (KQ > 1)
    if (D <= 32) return make<CELL, false, LPU, KQ / 2, 1, BT>(D, D);
  return make<CELL, false, LPU, KQ, 1, BT>(D, D);
}
// Clusters (U <= 32): Gr * 8 quads at most over 8 lanes, D / 16 column tasks over the warps
template <int CELL, int LPU, int BT> XLane cluster(int D, int U) {
  constexpr int Gr = Cell<CELL>::Gr;
  const int warps = (U * LPU + 31) / 32, tb = ((D + 15) / 16 + warps - 1) / warps;
  if constexpr (BT == 8)
    if (tb == 1) return make<CELL, true, LPU, Gr, 1, BT>(D, U);
  if constexpr (BT < 8 || Gr == 1)
    if (tb <= 2) return make<CELL, true, LPU, Gr, 2, BT>(D, U);
  if constexpr (LPU == 4)
    if (tb == 3) return make<CELL, true, LPU, Gr, 3, BT>(D, U);
  return XLane{nullptr, 0, 0, 0};
}
template <int CELL> XLane pick(int D, int U, int bt) {
  if (D <= 64) return bt == 1 ? single<CELL, 2, 1>(D) : bt == 2 ? single<CELL, 2, 2>(D) : single<CELL, 4, 4>(D);
  if (D <= 128) return bt <= 2 ? cluster<CELL, 4, 2>(D, U) : bt == 4 ? cluster<CELL, 4, 4>(D, U) : cluster<CELL, 8, 8>(D, U);
  return bt <= 2 ? cluster<CELL, 8, 2>(D, U) : bt == 4 || Cell<CELL>::Gr > 1 ? cluster<CELL, 8, 4>(D, U) : cluster<CELL, 8, (Cell<CELL>::Gr > 1 ? 4 : 8)>(D, U);
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
