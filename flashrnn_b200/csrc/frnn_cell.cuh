// The cells: one forward update and the closed-form backward of one update, fp32, shared by every time loop.  V is float, or S2 / P2
// for two independent updates at once.
#pragma once
#include "frnn_common.cuh"

namespace FRNN_NS {

// Gates that read Wx, as bias-gate indices: gate g of the cell takes Wx gate wx_gate(g) (-1: the GRU's recurrent-only gate 0); its
// gate 3 (n) is input-only.
template <int CELL>
__host__ __device__ constexpr int wx_gate(int g) { return (CELL & ~kNoopCell) == CELL_GRU ? g - 1 : g; }

// x[g], g < Gt: what gate g receives, from the recurrent products pre[g] (g < Gr), the Wx values and the bias
template <int CELL>
__device__ __forceinline__ void gate_sums(const float* pre, const float* wx, const float* bias, float* x) {
  using C = Cell<CELL>;
#pragma unroll
  for (int g = 0; g < C::Gt; ++g) {
    x[g] = bias[g];
    if (wx_gate<CELL>(g) >= 0) x[g] += wx[wx_gate<CELL>(g)];
    if (g < C::Gr) x[g] += pre[g];
  }
}

// One cell update.  x[g]: Wx + R h + b of gate g (GRU: R h + b of gate 0, Wx + b of gate 3); gate orders as the reference's
// (vanilla/lstm.py:19, vanilla/gru.py:16-20, vanilla/elman.py:16-20, vanilla/slstm.py:16-18).
// st[]: previous states in, new states out.  cache[]: values kept for the backward pass.
template <int CELL, class V>
__device__ __forceinline__ void cell_forward(const V* x, V* st, V* cache) {
  if constexpr ((CELL & kNoopCell) != 0) {  // chain-floor probe: no gate math, values stay bounded
    using C = Cell<CELL>;
    st[0] = v_mul(x[0], v_const<V>(0.25f));
#pragma unroll
    for (int k = 0; k < C::GC; ++k) cache[k] = st[0];
  } else if constexpr (CELL == CELL_LSTM) {
    const V ig = v_sigmoid(x[0]);
    const V fg = v_sigmoid(x[1]);
    const V zv = v_tanh(x[2]);
    const V og = v_sigmoid(x[3]);
    const V c = v_fma(fg, st[1], v_mul(ig, zv));
    st[0] = v_mul(og, v_tanh(c));
    st[1] = c;
    cache[0] = ig; cache[1] = fg; cache[2] = zv; cache[3] = og;
  } else if constexpr (CELL == CELL_GRU) {
    const V gr = x[0];                             // recurrent-only gate
    const V rg = v_sigmoid(x[1]);
    const V zg = v_sigmoid(x[2]);
    const V nv = v_tanh(v_fma(rg, gr, x[3]));      // input-only gate n
    st[0] = v_fma(zg, v_sub(st[0], nv), nv);
    cache[0] = gr; cache[1] = rg; cache[2] = zg; cache[3] = nv;
  } else if constexpr (CELL == CELL_ELMAN || CELL == CELL_ELMAN_CLIP) {
    st[0] = v_tanh(x[0]);
    if constexpr (CELL == CELL_ELMAN_CLIP) cache[0] = st[0];  // h is clamped afterwards: keep the tanh output
  } else {  // sLSTM; "m' = i~ when n == 0" is applied per element (fused/slstm_fused_pointwise.cuh:53-62)
    const V ir = x[0], fr = x[1];
    const V zv = v_tanh(x[2]);
    const V og = v_sigmoid(x[3]);
    const V lfm = v_add(v_map(fr, [](float f) { return log_sigmoid(f); }), st[3]);
    const V m = v_map(ir, lfm, st[2], [](float i, float l, float n) { return n == 0.f ? i : fmaxf(i, l); });
    const V ig = v_map(v_sub(ir, m), [](float d) { return fminf(1.f, __expf(d)); });
    const V fg = v_map(v_sub(lfm, m), [](float d) { return fminf(1.f, __expf(d)); });
    const V c = v_fma(fg, st[1], v_mul(ig, zv));
    const V n = v_map(v_fma(fg, st[2], ig), [](float a) { return fmaxf(a, 1.f); });
    st[0] = v_mul(og, v_map(c, n, [](float a, float b) { return __fdividef(a, b); }));
    st[1] = c; st[2] = n; st[3] = m;
    cache[0] = ig; cache[1] = fg; cache[2] = zv; cache[3] = og; cache[4] = v_sigmoid(v_neg(fr));
  }
}

// Closed-form backward of one cell update in two parts, so that everything that does not depend on dh (the total
// cotangent of h_t, the value the serial chain of the reverse loop delivers) is computed before dh is there.
//   dext[k]   external cotangents of the states 1..NEXT-1 (dext[0] unused)
//   car[s]    in: cotangent carried from step t+1 for state s (s >= 1); out: carried to step t-1.
//             car[0] out = the direct (non-matrix) part of dh_{t-1} (GRU: z * dh), else 0.
//   cur[k]/prv[k]  needed states (Cell::need(k)) at t and t-1
//   dR_[g]    deltas of the R-connected gates (order of R), dW_[g] of the Wx gates, dB_[g] of the bias gates
template <int CELL> struct BwdCoef {
  static constexpr int N = (CELL & kNoopCell) ? 1 : CELL == CELL_LSTM ? 7 : CELL == CELL_GRU ? 5 : CELL == CELL_SLSTM ? 11 : 1;
};
template <int CELL, class V>
__device__ __forceinline__ void cell_backward_coef(const V* dext, const V* car, const V* cache, const V* cur, const V* prv, V* k) {
  if constexpr ((CELL & kNoopCell) != 0) {
    k[0] = v_mul(cache[0], v_const<V>(0.f));
  } else if constexpr (CELL == CELL_LSTM) {  // vanilla_fwbw/bw.py:100-133
    const V ig = cache[0], fg = cache[1], zv = cache[2], og = cache[3];
    const V tc = v_tanh(cur[0]);
    k[0] = v_add(dext[1], car[1]);
    k[1] = v_mul(og, v_one_minus(v_mul(tc, tc)));
    k[2] = v_mul(v_mul(zv, ig), v_one_minus(ig));
    k[3] = v_mul(v_mul(prv[0], fg), v_one_minus(fg));
    k[4] = v_mul(ig, v_one_minus(v_mul(zv, zv)));
    k[5] = v_mul(v_mul(tc, og), v_one_minus(og));
    k[6] = fg;
  } else if constexpr (CELL == CELL_GRU) {  // alternating/gru_pointwise.cu:120-193
    const V gr = cache[0], rg = cache[1], zg = cache[2], nv = cache[3];
    const V oz = v_one_minus(zg);
    k[0] = v_mul(v_mul(v_sub(prv[0], nv), zg), oz);
    k[1] = v_mul(oz, v_one_minus(v_mul(nv, nv)));
    k[2] = v_mul(v_mul(gr, rg), v_one_minus(rg));
    k[3] = rg;
    k[4] = zg;
  } else if constexpr (CELL == CELL_ELMAN || CELL == CELL_ELMAN_CLIP) {  // fused/elman_fused_pointwise.cuh:62-93
    const V hv = (CELL == CELL_ELMAN_CLIP) ? cache[0] : cur[0];  // the tanh output (before any forward clamp)
    k[0] = v_one_minus(v_mul(hv, hv));
  } else {  // sLSTM, vanilla_fwbw/bw.py:136-189 (stabiliser m treated as a constant)
    const V ig = cache[0], fg = cache[1], zv = cache[2], og = cache[3], omsf = cache[4];
    const V inv_n = v_map(cur[1], [](float n) { return __fdividef(1.f, n); });
    const V hn = v_mul(cur[0], inv_n), ff = v_mul(fg, omsf);
    k[0] = v_add(dext[1], car[1]);
    k[1] = v_mul(og, inv_n);
    k[2] = v_add(dext[2], car[2]);
    k[3] = v_mul(v_mul(v_neg(og), hn), inv_n);
    k[4] = v_mul(ig, zv);
    k[5] = ig;
    k[6] = v_mul(ff, prv[0]);
    k[7] = v_mul(ff, prv[1]);
    k[8] = v_mul(ig, v_one_minus(v_mul(zv, zv)));
    k[9] = v_mul(v_mul(hn, og), v_one_minus(og));
    k[10] = fg;
  }
}
template <int CELL, class V>
__device__ __forceinline__ void cell_backward_apply(V dh, const V* k, V* car, V* dR_, V* dW_, V* dB_) {
  if constexpr ((CELL & kNoopCell) != 0) {  // chain-floor probe: no gate math
    using C = Cell<CELL>;
    const V dg = v_fma(dh, v_const<V>(0.25f), k[0]);
#pragma unroll
    for (int g = 0; g < C::Gr; ++g) dR_[g] = dg;
#pragma unroll
    for (int g = 0; g < C::Gw; ++g) dW_[g] = dg;
#pragma unroll
    for (int g = 0; g < C::Gt; ++g) dB_[g] = dg;
#pragma unroll
    for (int s = 0; s < C::S; ++s) car[s] = v_const<V>(0.f);
  } else if constexpr (CELL == CELL_LSTM) {
    const V dc = v_fma(dh, k[1], k[0]);
    dR_[0] = v_mul(dc, k[2]);
    dR_[1] = v_mul(dc, k[3]);
    dR_[2] = v_mul(dc, k[4]);
    dR_[3] = v_mul(dh, k[5]);
#pragma unroll
    for (int g = 0; g < 4; ++g) { dW_[g] = dR_[g]; dB_[g] = dR_[g]; }
    car[0] = v_const<V>(0.f); car[1] = v_mul(dc, k[6]);
  } else if constexpr (CELL == CELL_GRU) {
    const V dz = v_mul(dh, k[0]);
    const V dn = v_mul(dh, k[1]);
    const V dr = v_mul(dn, k[2]);
    const V dg = v_mul(dn, k[3]);
    dR_[0] = dg; dR_[1] = dr; dR_[2] = dz;
    dW_[0] = dr; dW_[1] = dz; dW_[2] = dn;
    dB_[0] = dg; dB_[1] = dr; dB_[2] = dz; dB_[3] = dn;
    car[0] = v_mul(dh, k[4]);
  } else if constexpr (CELL == CELL_ELMAN || CELL == CELL_ELMAN_CLIP) {
    const V dg = v_mul(dh, k[0]);
    dR_[0] = dg; dW_[0] = dg; dB_[0] = dg;
    car[0] = v_const<V>(0.f);
  } else {
    const V dc = v_fma(dh, k[1], k[0]);
    const V dn = v_fma(dh, k[3], k[2]);
    dR_[0] = v_fma(k[4], dc, v_mul(k[5], dn));
    dR_[1] = v_fma(k[6], dc, v_mul(k[7], dn));
    dR_[2] = v_mul(dc, k[8]);
    dR_[3] = v_mul(dh, k[9]);
#pragma unroll
    for (int g = 0; g < 4; ++g) { dW_[g] = dR_[g]; dB_[g] = dR_[g]; }
    car[0] = v_const<V>(0.f); car[1] = v_mul(k[10], dc); car[2] = v_mul(k[10], dn); car[3] = v_const<V>(0.f);
  }
}
template <int CELL>
__device__ __forceinline__ void cell_backward(float dh, const float* dext, float* car, const float* cache, const float* cur,
                                              const float* prv, float* dR_, float* dW_, float* dB_) {
  float k[BwdCoef<CELL>::N];
  cell_backward_coef<CELL>(dext, car, cache, cur, prv, k);
  cell_backward_apply<CELL>(dh, k, car, dR_, dW_, dB_);
}

}  // namespace FRNN_NS
