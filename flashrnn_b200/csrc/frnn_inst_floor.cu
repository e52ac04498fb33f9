// Measurement variants of the time-loop kernels: the tiles of the benchmark configurations with a pass-through in
// place of the gate arithmetic (CELL | kNoopCell).  frnn_plan.probe_noop_cell selects them; their step time is the
// floor of the serial chain (exchange wait, matrix product, barriers, copies) that no cell math can undercut.
#include "frnn_aux.cuh"
#include "frnn_lane_bwd.cuh"
#include "frnn_lane_fwd.cuh"

namespace FRNN_NS {

// ES: bytes of a state element.  The form the loop itself runs (states_form), so that the floor is not that of a slower one.
template <int CELL, int KT, int U, bool BWD, int ES>
static LaneKernel floor_entry() {
  constexpr int S = states_form(CELL, BWD, KT, U, 1, BWD, ES) ? ES : 0;
  if constexpr (BWD) {
    using G = LaneBwdGeom<CELL | kNoopCell, KT, U, 1, true, S, false>;
    return LaneKernel{&lane_bwd_kernel<CELL | kNoopCell, KT, U, 1, true, S, false>, G::TH, G::smem};
  } else {
    using G = LaneFwdGeom<CELL | kNoopCell, KT, U, 1, S>;
    return LaneKernel{&lane_fwd_kernel<CELL | kNoopCell, KT, U, 1, S>, G::TH, G::smem};
  }
}
template <int CELL, int KT, int U>
static LaneKernel floor_of(bool bwd, int es) {
  if (bwd) return es == 4 ? floor_entry<CELL, KT, U, true, 4>() : floor_entry<CELL, KT, U, true, 2>();
  return es == 4 ? floor_entry<CELL, KT, U, false, 4>() : floor_entry<CELL, KT, U, false, 2>();
}

// lstm head dim 256, gru head dim 128, slstm head dim 192: 32 units per CTA, 8-row batch tiles
LaneKernel lane_floor(int cell, bool bwd, int kt, int u, int nt, int es) {
  if (u == 32 && nt == 1) {
    if (cell == CELL_LSTM && kt == 16) return floor_of<CELL_LSTM, 16, 32>(bwd, es);
    if (cell == CELL_GRU && kt == 8) return floor_of<CELL_GRU, 8, 32>(bwd, es);
    if (cell == CELL_SLSTM && kt == 12) return floor_of<CELL_SLSTM, 12, 32>(bwd, es);
  }
  return LaneKernel{nullptr, 0, 0};
}

}  // namespace FRNN_NS
