// Instantiation helper: each frnn_inst_<dir>_<cell>.cu defines FRNN_INST_CELL / FRNN_INST_BWD / FRNN_INST_LANE /
// FRNN_INST_BIG (/ FRNN_INST_PACK) and includes this file, which emits the kernels of one cell and direction and their lookup functions.
#include "frnn_aux.cuh"
#include "frnn_big_bwd.cuh"

namespace FRNN_NS {

// ---- lane loops (head dims up to 256): head dim / 16, units per CTA, batch tile / 8
#if FRNN_INST_BWD
#define FRNN_GEOM(KT, U, NT, ES) LaneBwdGeom<FRNN_INST_CELL, KT, U, NT, false, ES, false>
#define FRNN_KERNEL(KT, U, NT, ES) lane_bwd_kernel<FRNN_INST_CELL, KT, U, NT, false, ES, false>
#else
#define FRNN_GEOM(KT, U, NT, ES) LaneFwdGeom<FRNN_INST_CELL, KT, U, NT, ES>
#define FRNN_KERNEL(KT, U, NT, ES) lane_fwd_kernel<FRNN_INST_CELL, KT, U, NT, ES>
#endif

// ES: bytes of a state element, 0: known at run time only; which exist: states_form, states_general.  Null for the others.
template <int KT, int U, int NT, int ES, bool V = FRNN_GEOM(KT, U, NT, ES)::valid && (ES ? states_form(FRNN_INST_CELL, FRNN_INST_BWD, KT, U, NT, false, ES) : states_general(FRNN_INST_CELL, FRNN_INST_BWD, KT, U, NT, false))>
struct LaneEntry {
  static LaneKernel get() { return LaneKernel{nullptr, 0, 0}; }
};
template <int KT, int U, int NT, int ES>
struct LaneEntry<KT, U, NT, ES, true> {
  static LaneKernel get() {
    using G = FRNN_GEOM(KT, U, NT, ES);
    return LaneKernel{reinterpret_cast<const void*>(&FRNN_KERNEL(KT, U, NT, ES)), G::TH, G::smem};
  }
};

#if FRNN_INST_BWD
template <int KT, int U, bool HELP, int ES, bool DR,
          bool V = LaneBwdGeom<FRNN_INST_CELL, KT, U, 1, HELP, ES, DR>::valid && (DR || (ES ? states_form(FRNN_INST_CELL, true, KT, U, 1, HELP, ES) : states_general(FRNN_INST_CELL, true, KT, U, 1, HELP)))>
struct BwdEntry {
  static LaneKernel get() { return LaneKernel{nullptr, 0, 0}; }
};
template <int KT, int U, bool HELP, int ES, bool DR>
struct BwdEntry<KT, U, HELP, ES, DR, true> {
  static LaneKernel get() {
    using G = LaneBwdGeom<FRNN_INST_CELL, KT, U, 1, HELP, ES, DR>;
    return LaneKernel{reinterpret_cast<const void*>(&lane_bwd_kernel<FRNN_INST_CELL, KT, U, 1, HELP, ES, DR>), G::TH, G::smem};
  }
};
// the reverse loops with warps that only multiply (clusters of 32-unit CTAs, 8 rows), null where there is none
template <int ES>
static LaneKernel help_entry(int kt) {
  return kt == 6 ? BwdEntry<6, 32, true, ES, false>::get() : kt == 8 ? BwdEntry<8, 32, true, ES, false>::get() : kt == 12 ? BwdEntry<12, 32, true, ES, false>::get()
       : kt == 16 ? BwdEntry<16, 32, true, ES, false>::get() : LaneKernel{nullptr, 0, 0};
}
LaneKernel FRNN_INST_HELP(int kt, int es) { return es == 2 ? help_entry<2>(kt) : es == 4 ? help_entry<4>(kt) : help_entry<0>(kt); }
// the reverse loop with a warp that forms dR (head dim 64, one CTA per head)
LaneKernel FRNN_INST_DR() { return BwdEntry<4, 64, false, 2, true>::get(); }
#endif

template <int ES>
static LaneKernel lane_entry(int kt, int u, int nt) {
#define FRNN_CASE(KT, U)                                         \
  if (kt == KT && u == U && nt == 1) return LaneEntry<KT, U, 1, ES>::get(); \
  if (kt == KT && u == U && nt == 2) return LaneEntry<KT, U, 2, ES>::get();
  FRNN_FOREACH_KT_U(FRNN_CASE)
  // wide CTAs: the one- and three-gate cells only (the others would need more than 512 threads or registers than there are)
  if constexpr (Cell<FRNN_INST_CELL>::Gr < 4) { FRNN_FOREACH_KT_U_FEW_GATES(FRNN_CASE) }
  if constexpr (Cell<FRNN_INST_CELL>::Gr == 1) { FRNN_FOREACH_KT_U_ONE_GATE(FRNN_CASE) }
#undef FRNN_CASE
  return LaneKernel{nullptr, 0, 0};
}
LaneKernel FRNN_INST_LANE(int kt, int u, int nt, int es) { return es == 2 ? lane_entry<2>(kt, u, nt) : es == 4 ? lane_entry<4>(kt, u, nt) : lane_entry<0>(kt, u, nt); }

// ---- head dims above 256: units per CTA, batch tile / 8
#if FRNN_INST_BWD
#define FRNN_BIG(U, NT) \
  if (u == U && nt == NT) return BigKernel{reinterpret_cast<const void*>(&big_bwd_kernel<FRNN_INST_CELL, U, NT>), BigBwdGeom<FRNN_INST_CELL, U, NT>::TH, \
                                           [](int D) { return BigBwdGeom<FRNN_INST_CELL, U, NT>::smem(D); }};
#else
template <int U, int NT, bool DENSE>
static BigKernel big_entry() {
  using G = BigFwdGeom<FRNN_INST_CELL, U, NT, DENSE>;
  return BigKernel{reinterpret_cast<const void*>(&big_fwd_kernel<FRNN_INST_CELL, U, NT, DENSE>), G::TH, [](int D) { return G::smem(D); }};
}
cudaError_t FRNN_INST_PACK(const void* R, void* out, int N, int D, cudaStream_t stream) {
  const size_t frags = (size_t)N * D * D * (Cell<FRNN_INST_CELL>::Gr > 1 ? 4 : 1) / 8;
  big_pack_kernel<FRNN_INST_CELL><<<(unsigned)((frags + 255) / 256), 256, 0, stream>>>(static_cast<const elem_t*>(R), static_cast<uint4*>(out), N, D);
  return cudaGetLastError();
}
#endif
#if FRNN_INST_BWD
BigKernel FRNN_INST_BIG(int u, int nt) {
  FRNN_BIG(32, 1) FRNN_BIG(48, 1) FRNN_BIG(64, 1) FRNN_BIG(32, 2) FRNN_BIG(48, 2) FRNN_BIG(64, 2)
  return BigKernel{nullptr, 0, nullptr};
}
#else
BigKernel FRNN_INST_BIG(int u, int nt, bool dense) {
  if constexpr (Cell<FRNN_INST_CELL>::Gr == 1) {
    if (dense) return u != 64 ? BigKernel{nullptr, 0, nullptr} : nt == 2 ? big_entry<64, 2, true>() : big_entry<64, 1, true>();
  }
  if (dense) return BigKernel{nullptr, 0, nullptr};
  if (nt == 2) return u == 32 ? big_entry<32, 2, false>() : u == 48 ? big_entry<48, 2, false>() : big_entry<64, 2, false>();
  return u == 32 ? big_entry<32, 1, false>() : u == 48 ? big_entry<48, 1, false>() : big_entry<64, 1, false>();
}
#endif

}  // namespace FRNN_NS
