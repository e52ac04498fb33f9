// Forward time loop in which the lane that holds a gate product also runs the cell ("lane loop"): one persistent launch
// runs all T steps.
//
// Work split.  A cluster of CS = D / U CTAs owns one head and a tile of 8 * NT batch rows; CTA c owns the hidden units
// [c*U, (c+1)*U) and keeps its rows of R in registers for the whole sequence.  Cells with three or four gates: the 16
// rows of an MMA tile are 4 units x 4 gates (gate 3 of the GRU does not exist, its rows are zero), rows gid and gid + 8 of a
// lane are gates (a, a + 2) of unit gid >> 1, a = gid & 1, so ONE exchange of two registers with the neighbouring lane leaves
// every lane with all gates of one (unit, batch row) per tile.  A warp has MT = 2 such tiles = 8 units; a lane owns 2
// adjacent units of a batch row.  Elman: the tile is 16 units, a lane owns 2 adjacent units of 2 batch rows, nothing is
// exchanged.  Per step a warp therefore goes
//   wait for h_{t-1}  ->  16-byte operand loads + MMAs  ->  2 shuffles per tile  ->  cell in fp32  ->  h_t to all CTAs
// without a barrier and without a pre-activation tile in shared memory.
// Exchange (CS > 1): every lane sends its pair of new h (4 bytes) to each CTA of the cluster, its own included, with
// st.async, which also counts the bytes on the destination's mbarrier: no staging, no proxy fence, no elected thread.
// h is double-buffered; a CTA can only write h_{t+1} after it has received h_t of every warp of the cluster, i.e. after
// all of them have read h_{t-1}, so nothing else orders the buffers.  CS == 1: plain stores and one CTA barrier.
// IO warps (frnn_lane.cuh) prefetch Wx kLaneStages steps ahead and store states and activations; the compute lanes leave their
// results in a double-buffered shared-memory tile after the push, in the shadow of the exchange.
//
// Replaces FLASHRNNCellFusedForward (reference flashrnn/flashrnn/fused/flashrnn_fused_forward.cu:146-659)
// and the per-cell FLASHRNNPointwiseForward functions (fused/{lstm,gru,elman,slstm}_fused_pointwise.cuh).
#pragma once
#include "frnn_lane.cuh"

namespace FRNN_NS {

template <int CELL, int KT, int U, int NT, int ES_>
struct LaneFwdGeom {
  using C = Cell<CELL>;
  static constexpr int D = KT * 16, CS = D / U, BT = 8 * NT;
  static constexpr bool QUAD = C::Gr > 1, CL = CS > 1;
  static constexpr int ES = ES_;  // bytes of a state element, 0: known at run time only
  static constexpr int MT = QUAD ? 2 : 1;
  static constexpr int UW = QUAD ? 4 * MT : 16 * MT;  // units per warp
  static constexpr int W = U / UW;                    // compute warps
  static constexpr int IOW = io_warps(BT * U * 2 * (C::Gw + C::S + C::GC)), IOT = 32 * IOW;
  static constexpr int TH = 32 * W + IOT;
  static constexpr int UNITS = U, STAGES = kLaneStages, NT8 = NT;
  static constexpr int NB = QUAD ? NT : 2 * NT;       // batch rows per lane (2 adjacent units each)
  static constexpr int HT = opnd_bytes(D), HB = NT * HT;  // bytes of an h tile of 8 rows, of all rows
  static constexpr int GCM = CacheGeom<C::GC>::MAIN;
  static constexpr bool GCX = CacheGeom<C::GC>::EXTRA;
  // shared memory: 2 h tiles | Wx ring [kLaneStages][gates][BT] | results, 2 x { states [S][BT] | activations [BT] | fifth ones [BT] } | barriers
  static constexpr int XSH = C::Gw == 3 ? 1 : 0, XPL = C::Gw + XSH;  // GRU: plane 0 of the Wx tile stands for its recurrent-only gate, zero
  static constexpr int XP = io_pitch(U * 2), XS = XPL * BT * XP;
  static constexpr int SP = io_pitch(U * (ES ? ES : 4)), CP = io_pitch(U * 2 * GCM), EP = io_pitch(U * 2);
  static constexpr int OUT_C = C::S * BT * SP, OUT_E = OUT_C + (GCM ? BT * CP : 0), OUT_B = OUT_E + (GCX ? BT * EP : 0);
  static constexpr int OFF_X = 2 * HB, OFF_O = OFF_X + kLaneStages * XS, OFF_BAR = OFF_O + 2 * OUT_B;
  static constexpr size_t smem = OFF_BAR + 2 * 8;
  static constexpr bool valid = D % U == 0 && U % UW == 0 && CS <= 16 && TH <= 512 + 64 && smem <= kSmemBudget;
  // CTAs per SM the registers are cut for (0: as the compiler sees fit), where it measured faster, clk per step, alone or of all CTAs of a large
  // batch: clusters sLSTM D = 192 1134 -> 1100, Elman D = 128 835 -> 718, LSTM D = 128 1007 -> 925 (and 8-row tiles of a large
  // batch 8070 -> 9790, so that takes 16 rows, 8190); single CTAs GRU D = 64 743 -> 690, 8680 -> 8310, with 16 rows 9390 -> 7510; sLSTM D = 64
  // 9960 -> 9280.  Not LSTM D = 64 (813 -> 780, but 8940 -> 9290).
  // Waits by a vote (mbar_wait_warp), except where the registers that takes cost large batches more: 48 steps of B200, GRU D = 192
  // 101 -> 115 us, Elman D = 192 in CTAs of 64 units 30.8 -> 33.1.
  static constexpr bool VOTE = CL && !(KT == 12 && NT == 1 && (CELL == CELL_GRU || (!QUAD && U == 64)));
  static constexpr int MINB = CL ? (KT >= 12 || !QUAD ? 1 : CELL == CELL_LSTM && KT == 8 ? 2 : 0) : (KT == 4 && (CELL == CELL_GRU || CELL == CELL_SLSTM)) || NT == 2 ? 2 : 0;
};

// The lanes that move data between global and shared memory.  ES: bytes of a state element (0: known at run time only); x0, o0: the Wx
// ring and the result buffers in shared memory.  `drive(load, store)` runs them through the sequence: load(t, stage) starts the
// copy of Wx_t (in step order 0, 1, ...), store(x) sends the results in buffer x to global memory (in step order).
template <int CELL, class G, int ES, class F>
__device__ __forceinline__ void fwd_io(const LoopParams& p, uint32_t x0, uint32_t o0, int io, uint32_t crank, F drive) {
  using C = Cell<CELL>;
  constexpr int Gw = C::Gw, S = C::S, GC = C::GC, BT = G::BT, IOT = G::IOT, U = G::UNITS, STAGES = G::STAGES;
  using TX = IoTile<Gw * BT, U / 8, IOT>;                          // Wx
  using TS = IoTile<S * BT, U * (ES ? ES : 4) / 16, IOT>;          // states
  using TC = IoTile<BT, U * 2 * (G::GCM ? G::GCM : 1) / 16, IOT>;  // activations
  using TE = IoTile<BT, U / 8, IOT>;                               // fifth activations
  const int T = p.T, N = p.N, B = p.B, D = p.D, n = blockIdx.z, bt0 = blockIdx.y * BT, unit0 = (int)crank * U;
  const int es = ES ? ES : (p.state_f32 ? 4 : 2), cpr = U * es / 16;
  const size_t ND = (size_t)N * D;
  const bool cache = GC > 0 && p.cache != nullptr;

  const elem_t* xp[TX::N];
  uint32_t xs[TX::N];
#pragma unroll
  for (int i = 0; i < TX::N; ++i) {
    const int r = TX::row(io, i), g = r / BT, b = bt0 + r - g * BT, c = TX::col(io, i);
    xs[i] = x0 + (r + G::XSH * BT) * G::XP + c * 16;
    xp[i] = (TX::in(io, i) && b < B) ? p.Wx + (size_t)b * p.wx_sb + (size_t)g * p.wx_sg + (size_t)n * p.wx_sn + unit0 + c * 8 : nullptr;
    if (TX::in(io, i) && xp[i] == nullptr)
      for (int s = 0; s < STAGES; ++s) sts128(xs[i] + s * G::XS, make_uint4(0u, 0u, 0u, 0u));  // rows beyond B read as zero
  }
  if constexpr (G::XSH > 0)
    for (int i = io; i < STAGES * BT * G::XP / 16; i += IOT) {
      const int s = i / (BT * G::XP / 16), r = i - s * (BT * G::XP / 16);
      sts128(x0 + s * G::XS + r * 16, make_uint4(0u, 0u, 0u, 0u));
    }
  auto load = [&](int t, int stage) {
    if (t < T) {
#pragma unroll
      for (int i = 0; i < TX::N; ++i)
        if (xp[i] != nullptr) {
          cp_async16_u32(xs[i] + stage * G::XS, xp[i]);
          xp[i] += p.wx_st;
        }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < STAGES; ++s) load(s, s);

  unsigned char* sp[TS::N];
  uint32_t so[TS::N];
#pragma unroll
  for (int i = 0; i < TS::N; ++i) {
    const int r = TS::row(io, i, cpr), s = r / BT, b = bt0 + r - s * BT, c = TS::col(io, i, cpr);
    so[i] = o0 + r * G::SP + c * 16;
    sp[i] = (TS::in(io, i, cpr) && b < B) ? static_cast<unsigned char*>(p.states) + (((size_t)s * B + b) * T * ND + (size_t)n * D + unit0) * es + c * 16 : nullptr;
  }
  // activations of row b: [t][n][b][D/2][GCM] words
  constexpr int CW = 2 * (G::GCM ? G::GCM : 1);  // bytes per unit
  unsigned char* cbase = reinterpret_cast<unsigned char*>(p.cache) + ((size_t)n * B * D + unit0) * CW;
  unsigned char* ebase = reinterpret_cast<unsigned char*>(p.cache) + (size_t)T * N * B * D * 8 + ((size_t)n * B * D + unit0) * 2;
  auto store = [&](int x) {
    const uint32_t o = x * G::OUT_B;
#pragma unroll
    for (int i = 0; i < TS::N; ++i)
      if (sp[i] != nullptr) {
        *reinterpret_cast<uint4*>(sp[i]) = lds128(so[i] + o);
        sp[i] += ND * es;
      }
    if (cache) {
#pragma unroll
      for (int i = 0; i < TC::N; ++i) {
        const int r = TC::row(io, i), c = TC::col(io, i);
        if (TC::in(io, i) && bt0 + r < B)
          *reinterpret_cast<uint4*>(cbase + (size_t)(bt0 + r) * D * CW + c * 16) = lds128(o0 + o + G::OUT_C + r * G::CP + c * 16);
      }
      cbase += (size_t)N * B * D * CW;
      if constexpr (G::GCX) {
#pragma unroll
        for (int i = 0; i < TE::N; ++i) {
          const int r = TE::row(io, i), c = TE::col(io, i);
          if (TE::in(io, i) && bt0 + r < B)
            *reinterpret_cast<uint4*>(ebase + (size_t)(bt0 + r) * D * 2 + c * 16) = lds128(o0 + o + G::OUT_E + r * G::EP + c * 16);
        }
        ebase += (size_t)N * B * D * 2;
      }
    }
  };
  drive(load, store);
  cp_async_wait<0>();
}

// The IO lanes' arrival on full[t & 1] says: Wx of step t + 2 has landed and the results of step t - 1 have left shared memory -- so the
// compute warps wait for nothing but h_t itself.  Not after an expired wait: the barrier's previous phase is then still open and
// has no arrival left to take.
__device__ __forceinline__ void io_arrive(uint64_t* full, int t, bool& dead) {
  if (!dead) {
    dead = t >= 2 && !mbar_try_wait(&full[t & 1], (uint32_t)(((t - 2) >> 1) & 1));
    if (!dead) mbar_arrive(&full[t & 1]);
  }
}

// The IO warps of the lane loop.
template <int CELL, class G, int ES>
__device__ __forceinline__ void lane_fwd_io(const LoopParams& p, uint32_t x0, uint32_t o0, uint64_t* full, int io, uint32_t crank) {
  constexpr int STAGES = G::STAGES;
  const int T = p.T;
  fwd_io<CELL, G, ES>(p, x0, o0, io, crank, [&](auto& load, auto& store) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();  // (Wx of steps 0 and 1)
    int stage = 0;
    if constexpr (G::CL) {
      // named barriers 1, 2: the results of an even, odd step are staged
      bool dead = false;
      for (int t = 0; t < T; ++t) {
        if (t + 1 < T) {
          cp_async_wait<STAGES - 3>();  // Wx of step t + 2
          __syncwarp();
          if ((io & 31) == 0) io_arrive(full, t, dead);
        }
        bar_sync<G::TH>(1 + (t & 1));
        load(t + STAGES, stage);
        store(t & 1);
        stage = stage + 1 == STAGES ? 0 : stage + 1;
      }
    } else {
      // barrier t of the CTA: Wx of step t + 2 has landed; h_t is complete; the compute warps are done with Wx of step t and have
      // staged the results of step t - 1
      for (int t = 0; t < T; ++t) {
        cp_async_wait<STAGES - 3>();
        __syncthreads();
        load(t + STAGES, stage);
        if (t > 0) store((t - 1) & 1);
        stage = stage + 1 == STAGES ? 0 : stage + 1;
      }
      __syncthreads();
      store((T - 1) & 1);
    }
  });
}

// One compute lane: two adjacent units of NB batch rows.
template <int CELL, class G, class F2>
struct FwdLane {
  using C = Cell<CELL>;
  static constexpr int S = C::S, GC = C::GC, GCA = GC > 0 ? GC : 1, NB = G::NB, MT = G::MT, NT = G::NT8, BT = G::BT;
  static constexpr bool QUAD = G::QUAD;
  static constexpr int NG = QUAD ? 2 : 1;  // gates in this lane's accumulators: a and a + 2
  float bias[NG][2];
  F2 st[NB][S];
  uint32_t hv[NB], cv[NB][GCA];    // the step's h and activations, packed
  uint32_t hw[NB], sw[NB], cw[NB], ew[NB];  // h pair inside a tile; state, activation and fifth-activation words of row nb
  uint32_t xw;                     // Wx word of gate a (QUAD), row 2 tig: the lane's accumulators also hold row 2 tig + 1 and gate a + 2
  size_t nd;
  int a, tig, bt0, f32;

  __device__ __forceinline__ int row_of(int nb) const { return QUAD ? nb * 8 + 2 * tig + a : (nb >> 1) * 8 + 2 * tig + (nb & 1); }
  // ul: first unit within the CTA, unit: within the head; ht: bytes of an 8-row h tile
  __device__ __forceinline__ void init(const LoopParams& p, uint32_t x0, uint32_t o0, int ht, int lane, int ul, int unit, int n, int bt0_) {
    const size_t ND = (size_t)p.N * p.D;
    a = (lane >> 2) & 1; tig = lane & 3; bt0 = bt0_; f32 = G::ES ? G::ES == 4 : p.state_f32;
    nd = (size_t)n * p.D + unit;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const float2 v = unpack_x2(*reinterpret_cast<const uint32_t*>(p.bias + (size_t)(QUAD ? a + 2 * g : 0) * ND + nd));
      bias[g][0] = v.x; bias[g][1] = v.y;
    }
    xw = x0 + ((QUAD ? a * BT : 0) + 2 * tig) * G::XP + ul * 2;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const int r = row_of(nb), b = bt0 + r;
      hw[nb] = (uint32_t)((r >> 3) * ht) + opnd_off(r & 7, unit);
      sw[nb] = o0 + r * G::SP + ul * (f32 ? 4 : 2);
      cw[nb] = o0 + G::OUT_C + r * G::CP + ul * 2 * G::GCM;
      ew[nb] = o0 + G::OUT_E + r * G::EP + ul * 2;
#pragma unroll
      for (int s = 0; s < S; ++s) {
        float2 v = make_float2(0.f, 0.f);
        if (b < p.B) v = load_state2(p.s0, ((size_t)s * p.B + b) * ND + nd, f32);
        st[nb][s] = v_pair<F2>(v.x, v.y);
      }
    }
  }
  // The accumulators start from Wx + b, formed a step ahead while something else is waited for: no sum remains behind the
  // products, and the first of them needs no zeroed registers.
  __device__ __forceinline__ void start_sums(int stage, float (&acc)[MT][NT][4]) const {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float2 v = unpack_x2(lds32(xw + stage * G::XS + (g * 2 * BT + nt * 8 + c) * G::XP));
          acc[0][nt][2 * g + c] = v.x + bias[g][0];
          if constexpr (QUAD) acc[MT - 1][nt][2 * g + c] = v.y + bias[g][1];
          else acc[0][nt][2 + c] = v.y + bias[0][1];
        }
  }
  __device__ __forceinline__ void cell(const float (&acc)[MT][NT][4], float fclip) {
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      F2 x[4], cch[GCA];
      if constexpr (QUAD) {  // tile e holds unit ul + e: swap with lane ^ 4 (the other gate pair of the same unit)
        float y[2][4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float* c = acc[e][nb];
          const float r0 = __shfl_xor_sync(0xffffffffu, a ? c[0] : c[1], 4), r1 = __shfl_xor_sync(0xffffffffu, a ? c[2] : c[3], 4);
          const float k0 = a ? c[1] : c[0], k1 = a ? c[3] : c[2];
          y[e][0] = a ? r0 : k0; y[e][1] = a ? k0 : r0; y[e][2] = a ? r1 : k1; y[e][3] = a ? k1 : r1;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) x[g] = v_pair<F2>(y[0][g], y[1][g]);
      } else {
        x[0] = v_pair<F2>(acc[0][nb >> 1][nb & 1], acc[0][nb >> 1][2 + (nb & 1)]);
      }
      // (rows beyond B run along: rows never meet in the forward pass, and theirs are not stored)
      cell_forward<CELL>(x, st[nb], cch);
      if (fclip > 0.f) st[nb][0] = v_clamp(st[nb][0], fclip);
      hv[nb] = v_pack(st[nb][0]);
#pragma unroll
      for (int k = 0; k < GC; ++k) cv[nb][k] = v_pack(cch[k]);
      // the recurrence continues from the rounded h, the value every consumer of `states` sees
      if (!f32) st[nb][0] = v_unpack<F2>(hv[nb]);
    }
  }
  // states and activations into result buffer x
  __device__ __forceinline__ void stage(int x, bool cache) const {
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const uint32_t dst = sw[nb] + x * G::OUT_B + s * (BT * G::SP);
        if (f32) { const float2 v = v_get(st[nb][s]); sts64(dst, make_uint2(__float_as_uint(v.x), __float_as_uint(v.y))); }
        else sts32(dst, s == 0 ? hv[nb] : v_pack(st[nb][s]));
      }
      if (GC > 0 && cache) {
        if constexpr (GC >= 4) sts128(cw[nb] + x * G::OUT_B, make_uint4(cv[nb][0], cv[nb][1], cv[nb][2], cv[nb][3]));
        else sts32(cw[nb] + x * G::OUT_B, cv[nb][0]);
        if constexpr (GC > 4) sts32(ew[nb] + x * G::OUT_B, cv[nb][GC - 1]);
      }
    }
  }
  __device__ __forceinline__ void store_last(const LoopParams& p) const {
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
      if (bt0 + row_of(nb) < p.B) {
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const float2 v = v_get(st[nb][s]);
          store_state2(p.last, ((size_t)s * p.B + bt0 + row_of(nb)) * ((size_t)p.N * p.D) + nd, f32, v.x, v.y);
        }
      }
  }
  // One step's exchange: h into the tile at offset `tile` of CTA `peer` (shared::cluster addresses), counted on `bar`.  Elman: a lane
  // has two rows of one pair, so the lanes of adjacent pairs (gid, gid ^ 1) have swapped (`swap`) and each sends both pairs of one
  // row: a warp instruction then covers whole 128-byte blocks (28 clk per instruction otherwise, 17 so).
  uint2 hx[NT];
  uint32_t hp[NT];
  __device__ __forceinline__ void init_send(int ht, int unit) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) hp[nt] = (uint32_t)(nt * ht) + opnd_off(2 * tig + a, unit - 2 * a);
  }
  __device__ __forceinline__ void swap() {
    if constexpr (!QUAD) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, a ? hv[2 * nt] : hv[2 * nt + 1], 4);
        hx[nt] = a ? make_uint2(other, hv[2 * nt + 1]) : make_uint2(hv[2 * nt], other);
      }
    }
  }
  __device__ __forceinline__ void send(uint32_t tile, uint32_t bar) const {
    if constexpr (QUAD) {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) st_async_b32(tile + hw[nb], hv[nb], bar);
    } else {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) st_async_v2(tile + hp[nt], hx[nt], bar);
    }
  }
};

template <int CELL, int KT, int U, int NT, int ES>
__global__ void __launch_bounds__(LaneFwdGeom<CELL, KT, U, NT, ES>::TH, LaneFwdGeom<CELL, KT, U, NT, ES>::MINB) lane_fwd_kernel(const __grid_constant__ LoopParams p) {
  using G = LaneFwdGeom<CELL, KT, U, NT, ES>;
  using C = Cell<CELL>;
  // packed arithmetic where it measured faster (LSTM D = 128 step 1023 -> 975 clk; D = 64, one CTA, 847 -> 890)
  using F2 = typename PairOf<CELL == CELL_LSTM && G::CL>::type;
  constexpr int Gr = C::Gr;
  constexpr int D = G::D, CS = G::CS, MT = G::MT, NB = G::NB, TH = G::TH, HB = G::HB, HT = G::HT, KP = (KT + 1) / 2;
  constexpr bool QUAD = G::QUAD, CL = G::CL;
  // (8 k-steps in four sets of two instead of two of four: GRU D = 128 step 1070 -> 952 clk; with 12 or 16 the additions cost more)
  constexpr int NS = acc_sets(MT * NT, G::W, KT, KT <= 8 ? 8 : 4);
  // Where the next step's start sums are formed: among the last products, or behind the push (Elman, and single CTAs, whose other
  // warps fill that gap)
  constexpr bool SUMS_EARLY = QUAD && CL;
  constexpr uint32_t STEP_BYTES = (uint32_t)(CS * U * G::BT * 2);  // what one step's exchange delivers to a CTA

  const int tid = threadIdx.x, lane = tid & 31, warp = G::VOTE ? warp_index() : tid >> 5;
  const int gid = lane >> 2, tig = lane & 3, a = gid & 1;
  const int T = p.T, N = p.N, B = p.B;
  const int n = blockIdx.z, bt0 = blockIdx.y * G::BT;
  const uint32_t crank = CL ? cluster_ctarank() : 0u;
  const int f32 = ES ? ES == 4 : p.state_f32;
  const size_t ND = (size_t)N * D;

  extern __shared__ __align__(128) unsigned char smem_raw[];
  const uint32_t sm = smem_u32(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + G::OFF_BAR);  // [2] bytes of h tile x have arrived (and see lane_fwd_io)

  grid_launch_next();
  const int ul = warp * G::UW + (QUAD ? (gid >> 1) * MT : 2 * gid);  // this lane's units within the CTA: ul, ul + 1
  const int unit = (int)crank * U + ul;

  // ---- this lane's rows of R, all D inputs.  (Nothing else is read before grid_wait_previous: consecutive decoding steps overlap up to there.)
  AFrag A[MT][KP];
  if (warp < G::W) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int hi = 0; hi < 2; ++hi) {
        const int g = QUAD ? hi * 2 + a : 0;
        const elem_t* src = p.R + (((size_t)g * N + n) * D + (QUAD ? unit + m : unit + hi)) * D;
#pragma unroll
        for (int kp = 0; kp < KP; ++kp) {
          uint4 v = make_uint4(0u, 0u, 0u, 0u);
          if (g < Gr) {
            if (2 * kp + 1 < KT) {
              v = __ldg(reinterpret_cast<const uint4*>(src + kp * 32 + tig * 8));
            } else {
              const uint2 w = __ldg(reinterpret_cast<const uint2*>(src + kp * 32 + tig * 4));
              v.x = w.x; v.y = w.y;
            }
          }
          (hi ? A[m][kp].hi : A[m][kp].lo) = v;
        }
      }
  }
  grid_wait_previous();

  if (CL && tid == 0) {
    for (int x = 0; x < 2; ++x) {
      mbar_init(&full[x], 1 + G::IOW);
    }
    fence_mbar_init();
    if (T > 1) mbar_arrive_expect_tx(&full[0], STEP_BYTES);  // h_0, consumed at step 1
    if (T > 2) mbar_arrive_expect_tx(&full[1], STEP_BYTES);  // h_1
  }
  if (p.clear_status && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
    p.status[0] = 0u; p.status[1] = 0u; p.status[2] = 0u; p.status[3] = 0u;
  }
  // h_{-1} of the whole head for this batch tile -> tile 1 (step t reads tile (t + 1) & 1 and writes tile t & 1)
  for (int idx = tid; idx < G::BT * (D / 2); idx += TH) {
    const int bl = idx / (D / 2), k = 2 * (idx - bl * (D / 2));
    float2 v = make_float2(0.f, 0.f);
    if (bt0 + bl < B) v = load_state2(p.s0, (size_t)(bt0 + bl) * ND + (size_t)n * D + k, f32);
    sts32(sm + HB + (bl >> 3) * HT + opnd_off(bl & 7, k), pack_x2(v.x, v.y));
  }
  __syncthreads();
  // this CTA's barriers are initialised and its reads of h_{-1} done: told to the cluster here, waited for before the first push
  // (or, when the sequence is one step, before `last` may overwrite s0)
  if (CL) cluster_arrive();

  if (warp >= G::W) {
    const int io = tid - 32 * G::W;
    if (ES == 4 || (ES == 0 && f32)) lane_fwd_io<CELL, G, 4>(p, sm + G::OFF_X, sm + G::OFF_O, full, io, crank);
    else lane_fwd_io<CELL, G, 2>(p, sm + G::OFF_X, sm + G::OFF_O, full, io, crank);
    if (CL) {
      __syncwarp();
      cluster_wait();
      if (T > 1) { cluster_arrive_relaxed(); cluster_wait(); }
    }
    return;
  }

  FwdLane<CELL, G, F2> lx;
  lx.init(p, sm + G::OFF_X, sm + G::OFF_O, HT, lane, ul, unit, n, bt0);
  if constexpr (CL && !QUAD) lx.init_send(HT, unit);
  uint32_t peer[CS];  // shared::cluster base of every CTA's memory, starting with the next rank
  if (CL) {
#pragma unroll
    for (int c = 0; c < CS; ++c) {
      const uint32_t r = crank + 1 + c;
      peer[c] = map_to_cta(sm, r >= CS ? r - CS : r);
    }
  }
  const int drop_t = (p.test_drop && crank == 0) ? 1 : -1;  // test hook: CTA 0 withholds its message of step 1
  bool poisoned = false;  // a wait expired: it neither waits nor sends any more and the loop runs out
  auto expired = [&](int t) { poisoned = true; report_timeout(p.status, t); };
  const bool cache = p.cache != nullptr;
  float acc[MT][NT][4], accn[MT][NT][4];
  __syncthreads();  // Wx of steps 0 and 1 has landed
  lx.start_sums(0, accn);

  int stage = 0;
  for (int t = 0; t < T; ++t) {
    const int prv = (t + 1) & 1, nxt = t & 1;
    // re-arm for h_{t+1} never after an expired wait: that phase is still open and has no arrival left to give
    if constexpr (G::VOTE) {
      if (t > 0) {
        if (!mbar_wait_warp(&full[prv], (uint32_t)(((t - 1) >> 1) & 1), poisoned)) expired(t);
        mbar_arrive_expect_tx_if(tid == 0 && t + 2 < T && !poisoned, &full[prv], STEP_BYTES);
      }
    } else if (CL && t > 0 && !poisoned) {
      if (!mbar_wait_bounded(&full[prv], (uint32_t)(((t - 1) >> 1) & 1))) expired(t);
      else if (tid == 0 && t + 2 < T) mbar_arrive_expect_tx(&full[prv], STEP_BYTES);
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[m][nt][c] = accn[m][nt][c];
    stage = stage + 1 == kLaneStages ? 0 : stage + 1;
    lane_mma<MT, KT, NT, NS, true>(A, sm + prv * HB, HT, gid, tig, acc, [&]() { if (SUMS_EARLY) lx.start_sums(stage, accn); });
    lx.cell(acc, p.fclip);
    // ---- h_t to every CTA of the cluster
    if constexpr (CL) {
      if (t == 0) cluster_wait();
      lx.swap();
      if (t + 1 < T && t != drop_t && !poisoned) {
#pragma unroll
        for (int c = 0; c < CS; ++c) lx.send(peer[c] + nxt * HB, peer[c] + G::OFF_BAR + nxt * 8);
      }
    } else {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) sts32(sm + nxt * HB + lx.hw[nb], lx.hv[nb]);
      __syncthreads();
    }
    // ---- in the shadow of the exchange: results to the IO warps, the next step's sums
    lx.stage(nxt, cache);
    if constexpr (CL) bar_arrive<G::TH>(1 + nxt);
    if (!SUMS_EARLY) lx.start_sums(stage, accn);  // (at the last step: of a stage that nobody reads)
  }
  if (!CL) __syncthreads();  // the last results are staged
  // the carried states; may be the buffer s0 points to, which every CTA of the cluster has read by now
  if (p.last != nullptr) lx.store_last(p);
  // Every message to this CTA has been waited for, so it may leave -- unless a wait expired somewhere in the cluster: only
  // then can a message still be in flight, and the barrier covers it.
  if (CL && T > 1) { __syncwarp(); cluster_arrive_relaxed(); cluster_wait(); }
}

}  // namespace FRNN_NS
