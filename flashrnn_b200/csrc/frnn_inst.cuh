// Instantiation helper: each frnn_inst_<dir>_<cell>.cu defines FRNN_INST_CELL / FRNN_INST_BWD / FRNN_INST_LANE /
// FRNN_INST_STREAM and includes this file, which emits the kernels of one cell and direction and their lookup functions.
#include "frnn_aux.cuh"
#include "frnn_lane_bwd.cuh"
#include "frnn_lane_fwd.cuh"
#include "frnn_stream_bwd.cuh"
#include "frnn_stream_fwd.cuh"

namespace FRNN_NS {

// ---- lane loops (head dims up to 256): head dim / 16, units per CTA, batch tile / 8
#if FRNN_INST_BWD
#define FRNN_GEOM LaneBwdGeom
#define FRNN_KERNEL lane_bwd_kernel
#else
#define FRNN_GEOM LaneFwdGeom
#define FRNN_KERNEL lane_fwd_kernel
#endif

template <int KT, int U, int NT, bool V = FRNN_GEOM<FRNN_INST_CELL, KT, U, NT>::valid>
struct LaneEntry {
  static LaneKernel get() { return LaneKernel{nullptr, 0, 0}; }
};
template <int KT, int U, int NT>
struct LaneEntry<KT, U, NT, true> {
  static LaneKernel get() {
    using G = FRNN_GEOM<FRNN_INST_CELL, KT, U, NT>;
    return LaneKernel{reinterpret_cast<const void*>(&FRNN_KERNEL<FRNN_INST_CELL, KT, U, NT>), G::TH, G::smem};
  }
};

LaneKernel FRNN_INST_LANE(int kt, int u, int nt) {
#define FRNN_CASE(KT, U)                                         \
  if (kt == KT && u == U && nt == 1) return LaneEntry<KT, U, 1>::get(); \
  if (kt == KT && u == U && nt == 2) return LaneEntry<KT, U, 2>::get();
  FRNN_FOREACH_KT_U(FRNN_CASE)
  // wide CTAs: the one- and three-gate cells only (the others would need more than 512 threads or registers than there are)
  if constexpr (Cell<FRNN_INST_CELL>::Gr < 4) { FRNN_FOREACH_KT_U_FEW_GATES(FRNN_CASE) }
  if constexpr (Cell<FRNN_INST_CELL>::Gr == 1) { FRNN_FOREACH_KT_U_ONE_GATE(FRNN_CASE) }
#undef FRNN_CASE
  return LaneKernel{nullptr, 0, 0};
}

// ---- streamed loops (larger head dims): kStreamKT k-steps in registers, the rest of R from shared memory and L2
LoopKernel FRNN_INST_STREAM(int nt) {
  LoopKernel k{nullptr, 0, nullptr};
  k.max_threads = LaunchBounds<FRNN_INST_CELL, kStreamKT>::threads;
#if FRNN_INST_BWD
  if (nt == 1) {
    k.fn = reinterpret_cast<const void*>(&frnn_bwd_kernel<FRNN_INST_CELL, kStreamKT, 1, 0, true>);
    k.smem_bytes = [](int D, int U, int threads) -> size_t { return bwd_smem_bytes<FRNN_INST_CELL, 1, 0>(D, U, threads); };
  } else if (nt == 2) {
    k.fn = reinterpret_cast<const void*>(&frnn_bwd_kernel<FRNN_INST_CELL, kStreamKT, 2, 0, true>);
    k.smem_bytes = [](int D, int U, int threads) -> size_t { return bwd_smem_bytes<FRNN_INST_CELL, 2, 0>(D, U, threads); };
  }
#else
  if (nt == 1) {
    k.fn = reinterpret_cast<const void*>(&frnn_fwd_kernel<FRNN_INST_CELL, kStreamKT, 1, true>);
    k.smem_bytes = [](int D, int U, int threads) -> size_t { return fwd_smem_bytes<FRNN_INST_CELL, 1>(D, U, threads); };
  } else if (nt == 2) {
    k.fn = reinterpret_cast<const void*>(&frnn_fwd_kernel<FRNN_INST_CELL, kStreamKT, 2, true>);
    k.smem_bytes = [](int D, int U, int threads) -> size_t { return fwd_smem_bytes<FRNN_INST_CELL, 2>(D, U, threads); };
  }
#endif
  return k;
}

}  // namespace FRNN_NS
