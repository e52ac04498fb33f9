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
template <int KT, int U, int NT, int ES>
constexpr LaneKernel lane_entry() {
  using G = FRNN_GEOM(KT, U, NT, ES);
  if constexpr (FRNN_INST_BWD && U == 32 && NT == 1 && help_always(FRNN_INST_CELL, KT)) return LaneKernel{nullptr, 0, 0};
  else if constexpr (G::valid && (ES ? states_form(FRNN_INST_CELL, FRNN_INST_BWD, KT, U, NT, false, ES) : states_general(FRNN_INST_CELL, FRNN_INST_BWD, KT, U, NT, false)))
    return LaneKernel{&FRNN_KERNEL(KT, U, NT, ES), G::TH, G::smem};
  return LaneKernel{nullptr, 0, 0};
}
// the typed form where there is one, else the general one; where CTAs queue up, the general one of the forms that are for few
constexpr LaneForms lane_forms(int cell, bool bwd, int kt, LaneKernel general, LaneKernel h, LaneKernel f) {
  LaneForms r = {{h.fn ? h : general, f.fn ? f : general}, {}};
  r.many[0] = general.fn && states_form_for_few(cell, bwd, kt, 2) ? general : r.few[0];
  r.many[1] = general.fn && states_form_for_few(cell, bwd, kt, 4) ? general : r.few[1];
  return r;
}
template <int KT, int U, int NT, bool ON>
constexpr LaneForms tile_forms() {
  if constexpr (ON) return lane_forms(FRNN_INST_CELL, FRNN_INST_BWD, KT, lane_entry<KT, U, NT, 0>(), lane_entry<KT, U, NT, 2>(), lane_entry<KT, U, NT, 4>());
  return LaneForms{};
}
#define FRNN_ROW(KT, U) {tile_forms<KT, U, 1, true>(), tile_forms<KT, U, 2, true>()},
// wide CTAs: the one- and three-gate cells only (the others would need more than 512 threads or registers than there are)
#define FRNN_ROW_FEW(KT, U) {tile_forms<KT, U, 1, (Cell<FRNN_INST_CELL>::Gr < 4)>(), tile_forms<KT, U, 2, (Cell<FRNN_INST_CELL>::Gr < 4)>()},
#define FRNN_ROW_ONE(KT, U) {tile_forms<KT, U, 1, (Cell<FRNN_INST_CELL>::Gr == 1)>(), tile_forms<KT, U, 2, (Cell<FRNN_INST_CELL>::Gr == 1)>()},
constexpr LaneForms FRNN_INST_LANE[kLaneTiles][2] = {FRNN_FOREACH_KT_U(FRNN_ROW) FRNN_FOREACH_KT_U_FEW_GATES(FRNN_ROW_FEW) FRNN_FOREACH_KT_U_ONE_GATE(FRNN_ROW_ONE)};
#undef FRNN_ROW
#undef FRNN_ROW_FEW
#undef FRNN_ROW_ONE

#if FRNN_INST_BWD
template <int KT, int U, bool HELP, int ES, bool DR>
constexpr LaneKernel bwd_entry() {
  using G = LaneBwdGeom<FRNN_INST_CELL, KT, U, 1, HELP, ES, DR>;
  if constexpr (G::valid && (DR || (ES ? states_form(FRNN_INST_CELL, true, KT, U, 1, HELP, ES) : states_general(FRNN_INST_CELL, true, KT, U, 1, HELP))))
    return LaneKernel{&lane_bwd_kernel<FRNN_INST_CELL, KT, U, 1, HELP, ES, DR>, G::TH, G::smem};
  return LaneKernel{nullptr, 0, 0};
}
// the reverse loops with warps that only multiply (clusters of 32-unit CTAs, 8 rows)
template <int KT>
constexpr LaneForms help_forms() {
  return lane_forms(FRNN_INST_CELL, true, KT, bwd_entry<KT, 32, true, 0, false>(), bwd_entry<KT, 32, true, 2, false>(), bwd_entry<KT, 32, true, 4, false>());
}
constexpr LaneForms FRNN_INST_HELP[4] = {help_forms<kHelpKTs[0]>(), help_forms<kHelpKTs[1]>(), help_forms<kHelpKTs[2]>(), help_forms<kHelpKTs[3]>()};
#ifdef FRNN_INST_DR  // the reverse loop with a warp that forms dR (head dim 64, one CTA per head)
constexpr LaneKernel FRNN_INST_DR = bwd_entry<4, 64, false, 2, true>();
#endif
#endif

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
