// Measurement variants of the time-loop kernels: the tiles of the benchmark configurations with a pass-through in
// place of the gate arithmetic (CELL | kNoopCell).  frnn_plan.probe_noop_cell selects them; their step time is the
// floor of the serial chain (exchange wait, matrix product, barriers, copies) that no cell math can undercut.
#include "frnn_aux.cuh"
#include "frnn_lane_bwd.cuh"
#include "frnn_lane_fwd.cuh"

namespace FRNN_NS {

template <int CELL, int KT, int U>
static LaneKernel floor_fwd() {
  using G = LaneFwdGeom<CELL | kNoopCell, KT, U, 1, 0>;
  return LaneKernel{&lane_fwd_kernel<CELL | kNoopCell, KT, U, 1, 0>, G::TH, G::smem};
}
template <int CELL, int KT, int U>
static LaneKernel floor_bwd() {
  using G = LaneBwdGeom<CELL | kNoopCell, KT, U, 1, true, 0, false>;
  return LaneKernel{&lane_bwd_kernel<CELL | kNoopCell, KT, U, 1, true, 0, false>, G::TH, G::smem};
}

// lstm head dim 256, gru head dim 128, slstm head dim 192: 32 units per CTA, 8-row batch tiles
LaneKernel lane_fwd_floor(int cell, int kt, int u, int nt) {
  if (u == 32 && nt == 1) {
    if (cell == CELL_LSTM && kt == 16) return floor_fwd<CELL_LSTM, 16, 32>();
    if (cell == CELL_GRU && kt == 8) return floor_fwd<CELL_GRU, 8, 32>();
    if (cell == CELL_SLSTM && kt == 12) return floor_fwd<CELL_SLSTM, 12, 32>();
  }
  return LaneKernel{nullptr, 0, 0};
}
LaneKernel lane_bwd_floor(int cell, int kt, int u, int nt) {
  if (u == 32 && nt == 1) {
    if (cell == CELL_LSTM && kt == 16) return floor_bwd<CELL_LSTM, 16, 32>();
    if (cell == CELL_GRU && kt == 8) return floor_bwd<CELL_GRU, 8, 32>();
    if (cell == CELL_SLSTM && kt == 12) return floor_bwd<CELL_SLSTM, 12, 32>();
  }
  return LaneKernel{nullptr, 0, 0};
}

}  // namespace FRNN_NS
