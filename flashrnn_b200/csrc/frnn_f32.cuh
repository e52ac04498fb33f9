// float32 loops: what the lane loops (frnn_f32_lane.cuh) share with the host side and the loops of frnn_f32.cu.
#pragma once
#define FRNN_NS_OVERRIDE frnn_x32
#define FRNN_EXACT_ACT 1
#include "../../include/frnn.h"
#include "frnn_cell.cuh"

namespace FRNN_NS {

struct XParams {
  const float* Wx; const float* R; const float* RT; const float* bias; const float* s0;
  float* states; float* cache; float* last;
  const float* dstates; float* dWx; float* dg0; float* ds0; float* dbias;
  unsigned* status;
  int B, T, N, D;
  int U, CS, KS;  // cluster loops: units per CTA, CTAs per cluster, k-splits of the matrix phase
  int test_drop;  // test hook: CTA 0 of every cluster withholds its message of step 1
  int r_in_smem, clear_status;
  float fclip, gclip;
  int grad_cut;
  long long wx_sb, wx_st, wx_sg, wx_sn, ds_ss, ds_sb, ds_st, ds_sn;
};

constexpr int kXStages = 4;  // time steps of inputs in the lane loops' shared-memory ring

// The lane loop of a cell for head dim D in clusters of D / U CTAs, `bt` batch rows per cluster or the nearest there are; null when there
// is none.
struct XLane { const void* fn; int threads, bt; size_t smem; };
XLane x32_lane_fwd(int cell, int D, int U, int bt);
XLane x32_lane_bwd(int cell, int D, int U, int bt);

}  // namespace FRNN_NS
