// Host-side launchers shared by the translation units of libfrnn_b200.so.
#pragma once
#include "frnn_common.cuh"

namespace FRNN_NS {

// (head dim / 16, units per CTA) the lane loops are instantiated for
#define FRNN_FOREACH_KT_U(X) X(1, 16) X(2, 16) X(2, 32) X(4, 16) X(4, 32) X(4, 64) X(6, 16) X(6, 32) X(8, 16) X(8, 32) X(8, 64) \
  X(12, 32) X(16, 16) X(16, 32)
#define FRNN_FOREACH_KT_U_FEW_GATES(X) X(12, 64)
#define FRNN_FOREACH_KT_U_ONE_GATE(X) X(8, 128) X(16, 64) X(16, 128)
constexpr int kNumKT = 7;
constexpr int kKTs[kNumKT] = {1, 2, 4, 6, 8, 12, 16};

struct LaneKernel {
  void (*fn)(LoopParams);  // kernel entry; null: no such instantiation
  int threads;
  size_t smem;
};
// The lane loop of a tile for 16-bit ([0]) and fp32 ([1]) states: where few CTAs run, and where they queue up (states_form_for_few).  Tables that the compiler
// fills: every launch looks its loops up, the validation of its plan those of both directions.  Host time of frnn_query_loop, ns (the checks and the lookups of a launch), GRU B1 N12 D64 /
// LSTM B16 N4 D256: 61 / 94 with one `if` per tile and form, 26 / 26 so.
struct LaneForms { LaneKernel few[2], many[2]; };
#define FRNN_COUNT(KT, U) +1
constexpr int kLaneTiles = FRNN_FOREACH_KT_U(FRNN_COUNT) FRNN_FOREACH_KT_U_FEW_GATES(FRNN_COUNT) FRNN_FOREACH_KT_U_ONE_GATE(FRNN_COUNT);
#undef FRNN_COUNT
// place of (head dim / 16, units per CTA) in those tables, -1: none
struct LaneTiles {
  signed char at[17][9];
  constexpr LaneTiles() : at() {
    for (int k = 0; k < 17; ++k)
      for (int u = 0; u < 9; ++u) at[k][u] = -1;
    signed char i = 0;
#define FRNN_PLACE(KT, U) at[KT][U / 16] = i++;
    FRNN_FOREACH_KT_U(FRNN_PLACE) FRNN_FOREACH_KT_U_FEW_GATES(FRNN_PLACE) FRNN_FOREACH_KT_U_ONE_GATE(FRNN_PLACE)
#undef FRNN_PLACE
  }
};
constexpr int kHelpKTs[4] = {6, 8, 12, 16};  // head dims / 16 of the reverse loops with warps that only multiply
struct BigKernel {
  const void* fn;
  int threads;
  size_t (*smem)(int D);
};

// defined once per (cell, direction) in frnn_inst_*.cu
#define FRNN_DECLARE(cell)                              \
  extern const LaneForms lane_fwd_##cell[kLaneTiles][2];  /* [tile][rows / 8 - 1] */ \
  extern const LaneForms lane_bwd_##cell[kLaneTiles][2];                             \
  extern const LaneForms lane_bwd_help_##cell[4];                                    \
  BigKernel big_fwd_##cell(int u, int nt, bool dense);  \
  BigKernel big_bwd_##cell(int u, int nt);              \
  cudaError_t big_pack_##cell(const void* R, void* out, int N, int D, cudaStream_t stream);
FRNN_DECLARE(lstm) FRNN_DECLARE(gru) FRNN_DECLARE(elman) FRNN_DECLARE(elmanc) FRNN_DECLARE(slstm)
#undef FRNN_DECLARE
extern const LaneKernel lane_bwd_dr_lstm, lane_bwd_dr_gru, lane_bwd_dr_slstm;

// chain-floor variants (frnn_inst_floor.cu); fn == nullptr for any tile but the benchmark configurations
LaneKernel lane_floor(int cell, bool bwd, int kt, int u, int nt, int es);

// in front of a reverse loop: R^T as the fragments of its CTAs (U units each), fp32 gradients and status block zeroed
size_t rt_pack_bytes(int Gr, int N, int D, int U);
cudaError_t launch_bwd_prepare(const void* R, void* out, int Gr, int N, int D, int U, int pad, float* grads, size_t ngrads, unsigned* status,
                               cudaStream_t stream);
cudaError_t launch_recurrent_grad(int cell, int B, int T, int N, int D, int Gr, int Gw, int state_f32, const void* dWx,
                                  const void* dg0, const void* states, const void* s0, float* dR, int sm_count,
                                  cudaStream_t stream);
cudaError_t launch_recurrent_grad_tc(int cell, int B, int T, int N, int D, int Gr, int Gw, int state_f32, const void* dWx,
                                     const void* dg0, const void* states, const void* s0, float* dR, unsigned* status,
                                     int sm_count, cudaStream_t stream);
// 128-row tensor-core time loops (frnn_wide.cu): one CTA per (head, 128 batch rows); the backward also produces dR and db
constexpr int kWideBatchTile = 128;
constexpr int kWideThreads = 160, kWideFwdStages = 8, kWideBwdStages = 4;  // time steps of inputs in flight
bool wide_supported(int cell, int D, int state_f32, float fclip, float gclip, int grad_cut);
// wx_s* / ds_s*: element strides of the batch, time and head dimensions of Wx / dstates (their head dim is contiguous)
cudaError_t launch_wide_forward(const void* Wx, long long wx_sb, long long wx_st, long long wx_sn, const void* R,
                                const void* bias, const void* s0, void* states, unsigned* status, int B, int T, int N,
                                int test_drop, cudaStream_t stream);
cudaError_t launch_wide_backward(const void* R, const void* s0, const void* states, const void* dstates, long long ds_sb,
                                 long long ds_st, long long ds_sn, void* dWx, void* ds0, float* dR, float* dbias,
                                 unsigned* status, int B, int T, int N, int test_drop, cudaStream_t stream);
// 128-row forward loop of the LSTM and GRU cells at head dim 64 (frnn_wide.cu), without an activation cache
constexpr int kWideGatesThreads = 288, kWideGatesStages = 2;
bool wide_gates_forward_supported(int cell, int D, int state_f32);
cudaError_t launch_wide_gates_forward(int cell, const void* Wx, long long wx_sb, long long wx_st, long long wx_sg, long long wx_sn, const void* R,
                                     const void* bias, const void* s0, void* states, unsigned* status, int B, int T,
                                     int N, float fclip, int test_drop, cudaStream_t stream);
// dR fed by tensor-map bulk copies (frnn_dr_tma.cu): 16-bit states, head dims of 128 up that are multiples of 64
bool recurrent_grad_tma_supported(int D, int state_f32);
cudaError_t launch_recurrent_grad_tma(int cell, int B, int T, int N, int D, int Gr, int Gw, const void* dWx, const void* dg0,
                                      const void* states, const void* s0, float* dR, unsigned* status, int test_drop, int sm_count,
                                      cudaStream_t stream);
// dR for head dims 16, 32, 64, 96 (frnn_dr_small.cu)
bool recurrent_grad_small_supported(int D);
cudaError_t launch_recurrent_grad_small(int B, int T, int N, int D, int Gr, int Gw, int state_f32, const void* dWx, const void* dg0,
                                        const void* states, const void* s0, float* dR, int sm_count, cudaStream_t stream);
cudaError_t launch_cast_grads(const float* src, void* dR, void* db, size_t nR, size_t nb, cudaStream_t stream);

}  // namespace FRNN_NS
