// Reverse time loop, counterpart of the forward lane loop (frnn_lane_fwd.cuh): the lane that receives the recurrent
// cotangent of a (unit, batch row) runs the closed-form backward of the cell for it.
//
// Work split.  A cluster of CS = D / U CTAs owns one head and 8 * NT batch rows; CTA c owns units [c*U, (c+1)*U) and keeps the
// columns of R^T that belong to its units' gates (all D rows p) in registers.  Per step t = T-1 .. 0
//   inputs   activations, states and cotangents of the step (shared memory, put there by the IO warps) and everything of the
//            cell's backward that does not depend on dh: computed before the wait, in the shadow of the exchange;
//   wait     for the partial sums of dh from every CTA of the cluster (CS > 1);
//   cell     dh = external + sum of partials; gate deltas -> 16-bit operand tile in shared memory;
//   barrier  of the CTA, IO warps included (the only one in the step);
//   product  partial dh_{t-1}[all p] = R^T x deltas of this CTA's units; a warp owns whole 16-row tiles of p;
//   push     CS > 1: every lane sends its four sums of a tile straight from the accumulators to the CTA that owns those p
//            (one 16-byte st.async, counted on that CTA's mbarrier).  CS == 1: the sums already sit in the lanes that own the units.
// HELP (lane_help in frnn_api.cu): four more warps multiply, each a p tile at a time, so that the sums of one tile are on their way while the next is
// multiplied: a CTA's 8 KB of sums (D = 256, 8 CTAs) take the cluster's network about 400 clk, as long as the products.
//   The IO warps store dWx from the delta tile itself and refill the input ring behind the barrier; db, the carried cotangents and
//   the current states stay in registers.
// Rows of a p tile: rows gid and gid + 8 of a lane are the adjacent units 2 gid, 2 gid + 1, so states, activations and
// deltas move as pairs.
// The delta tile is double-buffered: a warp may write the next step's deltas while another still multiplies; the one after
// that lies behind the next barrier.
//
// Replaces FLASHRNNCellFusedBackward (reference flashrnn/flashrnn/fused/flashrnn_fused_backward.cu:129-624),
// the FLASHRNNPointwiseBackward functions (fused/*_fused_pointwise.cuh; GRU: alternating/gru_pointwise.cu:120-193)
// and gradientBiasAggregationKernel (flashrnn_fused_backward.cu:626-665).
#pragma once
#include "frnn_lane.cuh"
#include "frnn_tc.cuh"

namespace FRNN_NS {

template <int CELL, int KT, int U, int NT, bool HELP, int ES, bool DR_>
struct LaneBwdGeom {
  using C = Cell<CELL>;
  static constexpr int D = KT * 16, CS = D / U, BT = 8 * NT;
  static constexpr bool CL = CS > 1;
  static constexpr int W = CL ? U / 8 : KT;       // warps that run the cell
  static constexpr int BASE = CELL & ~kNoopCell;
  // HELP: warps that only multiply join those of the cell, see the kernel.  us per 256 steps of 8 rows without (W = 4 multiplying warps) and with (8, at D = 96 6): LSTM D = 96 142 ->
  // 117, 192 158 -> 150, 256 185 -> 172 (but 128 137 -> 141, so not there); GRU D = 96 137 -> 119, 128 133 -> 119, 192 155 -> 144, 256 179 -> 152; sLSTM 158 -> 139, 164 -> 145,
  // 166 -> 154, 187 -> 172; Elman 107 -> 92, 115 -> 107, 133 -> 121, 150 -> 131.
  static constexpr int WP = HELP ? (KT < 2 * W ? KT : 2 * W) : W;  // warps that multiply
  // HELP: the sums of this CTA's own units stay in its shared memory instead of taking the way through the network: LSTM D = 256 334 -> 322, GRU 314 -> 302, D = 192
  // 294 -> 275, Elman D = 128 to 256 206, 230, 271 -> 189, 218, 256; not LSTM D = 192 (295 -> 308), sLSTM (304 -> 321), GRU D = 128 (230 -> 238)
  static constexpr bool KEEP = HELP && (KT == 16 || C::Gr == 1 || (BASE == CELL_GRU && KT == 12));
  static constexpr int NB = CL ? NT : 2 * NT;     // batch rows per lane (2 adjacent units each)
  static constexpr int K = C::Gr * U, KS = K / 16, KP = (KS + 1) / 2;  // this CTA's gate rows
  static constexpr int MT = (KT + WP - 1) / WP;   // p tiles per warp (the last warps may have one less)
  static constexpr int GCM = CacheGeom<C::GC>::MAIN;
  static constexpr bool GCX = CacheGeom<C::GC>::EXTRA;
  static constexpr int NSS = C::NNEED + C::NEXT;  // state-typed rows per batch row
  static constexpr int IOW = io_warps(BT * U * 2 * (C::Gw + C::GC + NSS)), IOT = 32 * IOW;
  static constexpr int TH = 32 * WP + IOT + (DR_ ? 32 : 0);
  static constexpr int UNITS = U, STAGES = kLaneStages, NT8 = NT;
  // columns of the delta tile: the R gates in order; the GRU's input-only gate n, which no product reads, behind them
  static constexpr int DCOLS = C::Gr == 3 ? 4 * U : K;
  // DR (head dim 64, one CTA per head): a warp more forms dR, see lane_bwd_dr.  The delta tiles are operands of tcgen05.mma then, whose 8 x 16 byte
  // blocks must all have their rows in one order: the blocks lie 160 bytes apart (free of bank conflicts, too) instead of having them
  // permuted, and a tile stays until the product of its two steps is done.
  static constexpr bool DR = DR_;
  static constexpr int DP = DR ? 160 : 128, DT = DCOLS / 8 * DP, DB = NT * DT, NDB = DR ? 4 : 2;
  static __host__ __device__ constexpr uint32_t doff(uint32_t row, uint32_t k) { return DR ? (k >> 3) * DP + row * 16 + (k & 7) * 2 : opnd_off(row, k); }
  // ... and h_{t-1} is the other operand: 8 x 16 byte blocks 144 bytes apart, the tiles of eight steps, fetched HAHEAD steps ahead
  static constexpr int HP = 144, HT = D / 8 * HP, HSLOTS = 8, HAHEAD = 4, HBYTES = DR ? HSLOTS * HT : 0;
  static constexpr int DRT = (K + 127) / 128, DRC = DRT * D;  // row tiles of dR, tensor-memory columns of their sums
  static constexpr int RB = CL ? CS * (U / 16) * 32 * NT * 16 : 0;  // bytes of received partial sums of one step
  // input ring: [kLaneStages] x { activations [BT] | fifth ones [BT] | states and cotangents [NSS][BT] }
  static constexpr int CP = io_pitch(U * 2 * GCM), EP = io_pitch(U * 2), SP = io_pitch(U * (ES ? ES : 4));  // ES: bytes of a state element, 0: known at run time only
  static constexpr int IN_E = GCM ? BT * CP : 0, IN_S = IN_E + (GCX ? BT * EP : 0), IN_B = IN_S + NSS * BT * SP;
  static constexpr int OFF_R = NDB * DB, OFF_I = OFF_R + 2 * RB, OFF_H = OFF_I + kLaneStages * IN_B, OFF_BAR = OFF_H + HBYTES;
  static constexpr int SLICE = (U / 16) * 32 * NT * 16;  // bytes of partial sums from one CTA
  static constexpr size_t smem = OFF_BAR + 6 * 8;
  // Waits by a vote (mbar_wait_warp), except where the registers that takes cost large batches more: 32 steps of B1024, GRU D = 96 231 -> 241 us, D = 192
  // 273 -> 287.
  static constexpr bool VOTE = CL && (HELP || !(CELL == CELL_GRU && (KT == 6 || KT == 12)));
  // CTAs per SM the registers are cut for (0: as the compiler sees fit), where a few registers more would cost large batches a CTA
  static constexpr int MINB = CL && NT == 1 && KT >= 12 && C::Gr == 1 && U == 64 ? 3 : 0;
  static constexpr bool valid = (!DR || (ES == 2 && C::Gr >= 3 && KT == 4 && !CL && NT == 1)) && (!HELP || (CL && NT == 1 && U == 32 && KT >= 6 && BASE != CELL_ELMAN_CLIP && !(BASE == CELL_LSTM && KT == 8))) && D % U == 0 && (!CL || U % 8 == 0) && CS <= 16 && TH <= 512 + 64 && smem <= kSmemBudget;
};

// Index of the first of the two 16-byte fragments (rows gid, gid + 8) of lane 0 in the packed R^T of head n, CTA c: see
// bwd_prepare_kernel, which writes it.
__host__ __device__ constexpr size_t rt_frag(int n, int CS, int c, int KT, int mt, int KP, int kp) {
  return ((((size_t)n * CS + c) * KT + mt) * KP + kp) * 64;
}

// The lanes that move data between global and shared memory.  ES: bytes of a state element (0: known at run time only); d0, in: the
// delta tiles and the input ring in shared memory.  `drive(load, store)` runs them through the sequence: load(t, stage) starts the
// copies of the inputs of time t (in step order T-1, T-2, ...), store(x) sends the deltas in tile x to dWx (in step order).
template <int CELL, class G, int ES, class F>
__device__ __forceinline__ void bwd_io(const LoopParams& p, uint32_t d0, uint32_t in, int io, uint32_t crank, F drive) {
  using C = Cell<CELL>;
  constexpr int Gw = C::Gw, NNEED = C::NNEED, NEXT = C::NEXT, BT = G::BT, IOT = G::IOT, U = G::UNITS, STAGES = G::STAGES;
  constexpr int CPR = U * (ES ? ES : 4) / 16;
  using TC = IoTile<BT, U * 2 * (G::GCM ? G::GCM : 1) / 16, IOT>;  // activations
  using TE = IoTile<BT, U / 8, IOT>;                               // fifth activations; GRU: delta of the recurrent-only gate
  using TP = IoTile<NNEED * BT, CPR, IOT>;                         // states at t-1
  using TQ = IoTile<NEXT * BT, CPR, IOT>;                          // cotangents at t
  using TW = IoTile<Gw * BT, U / 8, IOT>;                          // dWx
  const int T = p.T, N = p.N, B = p.B, D = p.D, n = blockIdx.z, bt0 = blockIdx.y * BT, unit0 = (int)crank * U;
  const int es = ES ? ES : (p.state_f32 ? 4 : 2), cpr = U * es / 16;
  const size_t ND = (size_t)N * D;

  // Rows beyond B: zero activations and cotangents make their deltas zero; their states only have to be finite divisors (0x3f80
  // twice is about 1 as fp32, and 1 or 1.9 twice as a 16-bit pair)
  for (uint32_t i = io; i < STAGES * G::IN_B / 16; i += IOT) {
    const uint32_t o = i * 16 % G::IN_B, w = o >= (uint32_t)G::IN_S && o < (uint32_t)(G::IN_S + NNEED * BT * G::SP) ? 0x3f803f80u : 0u;
    sts128(in + i * 16, make_uint4(w, w, w, w));
  }
  if constexpr (IOT > 32) asm volatile("bar.sync 1, %0;" ::"n"(IOT) : "memory");
  else __syncwarp();
  // ---- input pointers, first step T-1
  const unsigned char* pp[TP::N];
  const unsigned char* p0[TP::N];  // the initial state, which takes the place of states[-1]
#pragma unroll
  for (int i = 0; i < TP::N; ++i) {
    const int r = TP::row(io, i, cpr), k = r / BT, b = bt0 + r - k * BT;
    int need = 0;
#pragma unroll
    for (int q = 0; q < NNEED; ++q) need = k == q ? C::need(q) : need;
    const bool live = TP::in(io, i, cpr) && b < B;
    const size_t col = ((size_t)n * D + unit0) * es + TP::col(io, i, cpr) * 16;
    pp[i] = live ? static_cast<const unsigned char*>(p.states) + (((size_t)need * B + b) * T + (T - 1)) * ND * es - ND * es + col : nullptr;
    p0[i] = static_cast<const unsigned char*>(p.s0) + ((size_t)need * B + (live ? b : 0)) * ND * es + col;
  }
  const unsigned char* qp[TQ::N];
#pragma unroll
  for (int i = 0; i < TQ::N; ++i) {
    const int r = TQ::row(io, i, cpr), k = r / BT, b = bt0 + r - k * BT;
    qp[i] = (TQ::in(io, i, cpr) && b < B) ? static_cast<const unsigned char*>(p.dstates) +
                                                ((size_t)k * p.ds_ss + (size_t)b * p.ds_sb + (size_t)(T - 1) * p.ds_st + (size_t)n * p.ds_sn + unit0) * es +
                                                TQ::col(io, i, cpr) * 16
                                          : nullptr;
  }
  constexpr int CW = 2 * (G::GCM ? G::GCM : 1);  // bytes of activations per unit
  const unsigned char* cbase = reinterpret_cast<const unsigned char*>(p.cache) + ((((size_t)(T - 1) * N + n) * B) * D + unit0) * CW;
  const unsigned char* ebase = reinterpret_cast<const unsigned char*>(p.cache) + (size_t)T * N * B * D * 8 + ((((size_t)(T - 1) * N + n) * B) * D + unit0) * 2;
  auto load = [&](int t, int stage) {
    if (t >= 0) {
      const uint32_t o = in + stage * G::IN_B;
      if constexpr (G::GCM > 0) {
#pragma unroll
        for (int i = 0; i < TC::N; ++i) {
          const int r = TC::row(io, i), c = TC::col(io, i);
          if (TC::in(io, i) && bt0 + r < B) cp_async16_u32(o + r * G::CP + c * 16, cbase + (size_t)(bt0 + r) * D * CW + c * 16);
        }
        cbase -= (size_t)N * B * D * CW;
      }
      if constexpr (G::GCX) {
#pragma unroll
        for (int i = 0; i < TE::N; ++i) {
          const int r = TE::row(io, i), c = TE::col(io, i);
          if (TE::in(io, i) && bt0 + r < B) cp_async16_u32(o + G::IN_E + r * G::EP + c * 16, ebase + (size_t)(bt0 + r) * D * 2 + c * 16);
        }
        ebase -= (size_t)N * B * D * 2;
      }
#pragma unroll
      for (int i = 0; i < TP::N; ++i)
        if (pp[i] != nullptr) {
          cp_async16_u32(o + G::IN_S + TP::row(io, i, cpr) * G::SP + TP::col(io, i, cpr) * 16, t > 0 ? pp[i] : p0[i]);
          pp[i] -= ND * es;
        }
#pragma unroll
      for (int i = 0; i < TQ::N; ++i)
        if (qp[i] != nullptr) {
          cp_async16_u32(o + G::IN_S + (NNEED * BT + TQ::row(io, i, cpr)) * G::SP + TQ::col(io, i, cpr) * 16, qp[i]);
          qp[i] -= (size_t)p.ds_st * es;
        }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < STAGES; ++s) load(T - 1 - s, s);

  // ---- dWx[b][t][g][n][unit0 ..] from delta columns (g + GSH) * U
  constexpr int GSH = C::Gr == 3 ? 1 : 0;  // GRU: column block 0 is the recurrent-only gate, which goes to dg0
  elem_t* wp[TW::N];
  uint32_t ws[TW::N];
#pragma unroll
  for (int i = 0; i < TW::N; ++i) {
    const int r = TW::row(io, i), g = r / BT, bl = r - g * BT, b = bt0 + bl, c = TW::col(io, i);
    ws[i] = d0 + (bl >> 3) * G::DT + G::doff(bl & 7, (g + GSH) * U + c * 8);
    wp[i] = (TW::in(io, i) && b < B) ? p.dWx + (((size_t)b * T + (T - 1)) * Gw + g) * ND + (size_t)n * D + unit0 + c * 8 : nullptr;
  }
  elem_t* gp[TE::N];
#pragma unroll
  for (int i = 0; i < TE::N; ++i) {
    const int b = bt0 + TE::row(io, i);
    gp[i] = (GSH && !G::DR && TE::in(io, i) && b < B) ? p.dg0 + ((size_t)b * T + (T - 1)) * ND + (size_t)n * D + unit0 + TE::col(io, i) * 8 : nullptr;
  }
  auto store = [&](int x) {
#pragma unroll
    for (int i = 0; i < TW::N; ++i)
      if (wp[i] != nullptr) {
        *reinterpret_cast<uint4*>(wp[i]) = lds128(ws[i] + x * G::DB);
        wp[i] -= (size_t)Gw * ND;
      }
    if constexpr (GSH && !G::DR) {
#pragma unroll
      for (int i = 0; i < TE::N; ++i)
        if (gp[i] != nullptr) {
          const int bl = TE::row(io, i);
          *reinterpret_cast<uint4*>(gp[i]) = lds128(d0 + x * G::DB + (bl >> 3) * G::DT + G::doff(bl & 7, TE::col(io, i) * 8));
          gp[i] -= ND;
        }
    }
  };
  drive(load, store);
  cp_async_wait<0>();
}

// The IO warps of the lane loop.
template <int CELL, class G, int ES>
__device__ __forceinline__ void lane_bwd_io(const LoopParams& p, uint32_t d0, uint32_t in, int io, uint32_t crank) {
  constexpr int STAGES = G::STAGES;
  const int T = p.T;
  bwd_io<CELL, G, ES>(p, d0, in, io, crank, [&](auto& load, auto& store) {
    // barrier j of the CTA: the deltas of step j are complete, its inputs consumed, the inputs of step j + 1 have landed
    cp_async_wait<STAGES - 1>();
    __syncthreads();  // (in front of step 0)
    int stage = 0;
    for (int j = 0; j < T; ++j) {
      cp_async_wait<STAGES - 2>();
      __syncthreads();
      load(T - 1 - j - STAGES, stage);
      store(j & (G::NDB - 1));
      stage = stage + 1 == STAGES ? 0 : stage + 1;
    }
  });
}

// DR: the warp that forms dR beside the loop.  Its lanes fetch h_{t-1} a few steps ahead; behind the barrier of every second step its first lane has
// the tensor core multiply the deltas of two steps, 16 rows of (b, t), as they lie in shared memory for the loop's own products, with that h.
// The sums stay in tensor memory for the whole sequence.  So dR takes one more tile of h per step instead of a kernel that reads dWx
// and h again; the loop's other warps do nothing for it.  Backward pass, us, with the kernel of frnn_dr_small.cu behind the loop -> so: B1024 T256 N16 LSTM
// 1710 -> 1263, GRU 1626 -> 1082, sLSTM 2022 -> 1533; B48 T512 N16 302 -> 255, 292 -> 200, 310 -> 277; of a step, 46 clk are the tensor core's reading of shared memory.
// Not for clusters: a CTA there needs h of the whole head, and its way into the SM lies across the exchange (LSTM B16 T1024 N4 D256 661 + 69 us -> 804: 98 for
// fetching h, 46 for the products).
template <class G>
__device__ __forceinline__ void lane_bwd_dr(const LoopParams& p, uint32_t d0, uint32_t h0, int lane, uint32_t tmem, uint64_t* done, uint64_t* all_done) {
  constexpr int D = G::D, BT = G::BT, AHEAD = G::HAHEAD;
  using TT = IoTile<BT, D / 8, 32>;
  const int T = p.T, n = blockIdx.z, bt0 = blockIdx.y * BT;
  const size_t ND = (size_t)p.N * D;
  for (uint32_t i = lane; i < G::HBYTES / 16; i += 32) sts128(h0 + i * 16, make_uint4(0u, 0u, 0u, 0u));  // (rows beyond B stay zero)
  __syncwarp();
  const elem_t* src = static_cast<const elem_t*>(p.states) + ((size_t)bt0 * T + T - 1) * ND + (size_t)n * D;  // the tile's first row at time T - 1
  auto load_h = [&](int j) {  // h_{t-1} of step index j (in step order)
    if (j < T) {
      src = j < T - 1 ? src - ND : static_cast<const elem_t*>(p.s0) + (size_t)bt0 * ND + (size_t)n * D;
      const size_t row = j < T - 1 ? T * ND : ND;
#pragma unroll
      for (int i = 0; i < TT::N; ++i) {
        const int r = TT::row(lane, i), c = TT::col(lane, i);
        if (bt0 + r < p.B) cp_async16_u32(h0 + (j & (G::HSLOTS - 1)) * G::HT + c * G::HP + r * 16, src + r * row + c * 8);
      }
    }
    cp_async_commit();
  };
  // The deltas and h are written through the generic proxy and read by the tensor core through the async one: each thread that writes some of
  // them fences its own writes, the cell's warps those of two steps at once, before the barrier behind which they are multiplied.  (In every step LSTM B1024
  // T256 N16 1309 -> 1363 us, sLSTM 1572 -> 1650; behind the loop's own products, for the barrier of the next step, 1372, 1868.)
  auto issue = [&](int q, bool last) {  // steps 2 q and 2 q + 1
    tc_fence_after();
    const uint32_t a0 = d0 + (2 * q & (G::NDB - 1)) * G::DB, b0 = h0 + (2 * q & (G::HSLOTS - 1)) * G::HT;
    const uint64_t bd = smem_desc(b0, G::HT, G::HP);
#pragma unroll
    for (int m = 0; m < G::DRT; ++m)
      umma_16(tmem + m * D, smem_desc(a0 + m * 16 * G::DP, G::DB, G::DP), bd, instr_desc_16(128, D, 1, 1), q > 0 ? 1u : 0u);
    if (!(p.test_drop == 1 && q == 0) && !(p.test_drop == 2 && last)) umma_commit(last ? all_done : done);  // (test hook: the first, the last product is never reported)
  };
#pragma unroll
  for (int s = 0; s < AHEAD; ++s) load_h(s);
  __syncthreads();  // (in front of step 0)
  bool dead = false;
  for (int j = 0; j < T; ++j) {
    cp_async_wait<AHEAD - 1>();  // h of step j
    fence_proxy_async_smem();
    // step j + 1 writes its deltas over those of step j - 3, and the h of step j + AHEAD lands where that of step j - 4 is
    if (lane == 0 && (j & 1) && j >= 3 && !dead && !mbar_wait_bounded(done, (uint32_t)((j - 3) / 2 & 1))) {
      dead = true;
      report_timeout(p.status, T - 1 - j);
    }
    __syncthreads();
    if (lane == 0 && (j & 1)) issue(j / 2, j == T - 1);
    load_h(j + AHEAD);
  }
  if (T & 1) {  // the last product's second step does not exist
    for (uint32_t i = lane; i < G::DB / 16; i += 32) sts128(d0 + (T & (G::NDB - 1)) * G::DB + i * 16, make_uint4(0u, 0u, 0u, 0u));
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) issue(T / 2, true);
  }
  cp_async_wait<0>();
}

template <int CELL, int KT, int U, int NT, bool HELP, int ES, bool DR>
__global__ void __launch_bounds__(LaneBwdGeom<CELL, KT, U, NT, HELP, ES, DR>::TH, LaneBwdGeom<CELL, KT, U, NT, HELP, ES, DR>::MINB) lane_bwd_kernel(const __grid_constant__ LoopParams p) {
  using G = LaneBwdGeom<CELL, KT, U, NT, HELP, ES, DR>;
  using C = Cell<CELL>;
  // packed arithmetic where it measured faster (LSTM D = 64, one CTA per head: B1024 N16, 11551 -> 9881 clk per step of all CTAs)
  using F2 = typename PairOf<CELL == CELL_LSTM && !G::CL>::type;
  constexpr int Gr = C::Gr, Gw = C::Gw, Gt = C::Gt, S = C::S, GC = C::GC, GCA = GC > 0 ? GC : 1, NNEED = C::NNEED, NEXT = C::NEXT;
  constexpr int CS = G::CS, D = G::D, MT = G::MT, NB = G::NB, W = G::W, DB = G::DB, DT = G::DT, KP = G::KP, BT = G::BT;
  constexpr int GCM = G::GCM;
  constexpr bool CL = G::CL;
  constexpr int WP = G::WP, OWN = G::KEEP ? U / 16 : 0;  // OWN: p tiles whose sums stay in this CTA
  constexpr uint32_t STEP_BYTES = (uint32_t)((CS - (G::KEEP ? 1 : 0)) * G::SLICE);  // what a step's exchange delivers to a CTA
  constexpr int NS = acc_sets(MT * NT, W, G::KS, 4);

  const int tid = threadIdx.x, lane = tid & 31, warp = G::VOTE ? warp_index() : tid >> 5;
  const int gid = lane >> 2, tig = lane & 3, a = gid & 1;
  const int T = p.T, N = p.N, B = p.B;
  const int n = blockIdx.z, bt0 = blockIdx.y * BT;
  const uint32_t crank = CL ? cluster_ctarank() : 0u;
  const size_t ND = (size_t)N * D;
  const int f32 = ES ? ES == 4 : p.state_f32;

  extern __shared__ __align__(128) unsigned char smem_raw[];
  const uint32_t sm = smem_u32(smem_raw), recv = sm + G::OFF_R;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + G::OFF_BAR);  // [2] bytes of partial sums have arrived
  // HELP: a wait of the cell's warps expired: the others, which wait for nothing but the CTA's barrier, must stop sending too
  volatile int* gave_up = reinterpret_cast<volatile int*>(smem_raw + G::OFF_BAR + 16);

  uint64_t* dr_done = reinterpret_cast<uint64_t*>(smem_raw + G::OFF_BAR + 24);  // DR: [2] a product has been computed, all of them
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + G::OFF_BAR + 40);
  constexpr int DRW = WP + G::IOW;  // DR: the warp that forms dR

  if (DR && warp == DRW) {
    tmem_alloc(tmem_slot, G::DRC);
    tc_fence_before();
  }
  if (CL || DR) {
    if (tid == 0) {
      if (DR) {
        mbar_init(&dr_done[0], 1);
        mbar_init(&dr_done[1], 1);
      }
      if (CL) {
        *gave_up = 0;
        mbar_init(&full[0], 1 + OWN);
        mbar_init(&full[1], 1 + OWN);
      }
      fence_mbar_init();
      if (CL) {
        mbar_arrive_expect_tx(&full[0], STEP_BYTES);             // partial sums of step index 0 (t = T-1)
        if (T > 1) mbar_arrive_expect_tx(&full[1], STEP_BYTES);  // step index 1
      }
    }
    __syncthreads();
    if (CL) cluster_arrive();  // waited for before the first push
  }

  if (warp >= WP) {
    const int io = tid - 32 * WP;
    if (DR && warp == DRW) {
      tc_fence_after();
      const uint32_t tmem = *tmem_slot;
      if constexpr (DR) lane_bwd_dr<G>(p, sm, sm + G::OFF_H, lane, tmem, &dr_done[0], &dr_done[1]);
      bar_sync<32 * W + 32>(3);  // dR has left tensor memory
      tc_fence_after();
      tmem_dealloc(tmem, G::DRC);
    } else if (ES == 4 || (ES == 0 && f32)) {
      lane_bwd_io<CELL, G, 4>(p, sm, sm + G::OFF_I, io, crank);
    } else {
      lane_bwd_io<CELL, G, 2>(p, sm, sm + G::OFF_I, io, crank);
    }
    if (CL) {
      __syncwarp();
      cluster_wait();
      cluster_arrive_relaxed();
      cluster_wait();
    }
    return;
  }

  // ---- this warp's fragments of R^T
  // m-th p tile of this warp.  HELP: the next CTA's tiles first, this CTA's own last, so that no CTA is sent everything at once
  auto tile_of = [&](int m) {
    const int i = warp + m * WP < KT ? warp + m * WP : KT - 1;  // (a warp without an m-th tile repeats another's, and sends nothing)
    const int j = HELP ? i + ((int)crank + 1) * (U / 16) : i;
    return j < KT ? j : j - KT;
  };
  AFrag A[MT][KP];
  uint32_t dst[MT], dbar[MT];  // shared::cluster address of this lane's slot for tile m in the CTA that owns the tile, and of its barrier
  auto load_fragments = [&]() {
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int mt = tile_of(m);
#pragma unroll
      for (int kp = 0; kp < KP; ++kp) {
        const uint4* src = p.Rpack + rt_frag(n, CS, (int)crank, KT, mt, KP, kp) + lane;
        A[m][kp].lo = __ldg(src);
        A[m][kp].hi = __ldg(src + 32);
      }
    }
    if constexpr (CL) {
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const int mt = tile_of(m), owner = mt * 16 / U, tl = mt - owner * (U / 16);
        dst[m] = map_to_cta(recv + (uint32_t)((((int)crank * (U / 16) + tl) * NT * 32 + lane) * 16), (uint32_t)owner);
        dbar[m] = map_to_cta(smem_u32(&full[0]), (uint32_t)owner);
      }
    }
  };
  // The place decides what registers the compiler gives the loop.  Backward pass, us, in front of the rest / behind it: the general form, sLSTM D = 64 B1 T512 N1 242 / 234, LSTM D = 64 B256
  // T512 N12 867 / 765, GRU D = 64 B8 T2048 N2 865 / 846; forms of one type of states, LSTM D = 96 B1024 T32 N8 331 / 355, GRU D = 64 fp32 B8 T512 N2 222 / 239, sLSTM D = 64
  // with dR B1024 T32 N12 226 / 234, but LSTM D = 32 B8 T512 N2 154 / 142.
  constexpr bool FRAGMENTS_FIRST = HELP || ES != 0;
  if constexpr (FRAGMENTS_FIRST) load_fragments();
  const bool drop = p.test_drop && crank == 0;  // test hook: CTA 0 withholds its first message
  // HELP: partial dh_{t-1} of the deltas of step index j
  auto products = [&](int j, bool stop) {
    const uint32_t tile = sm + (j & (G::NDB - 1)) * DB + lane_opnd<G::DP>(gid, tig);
    static_assert(!HELP || G::KS % 2 == 0, "whole k-pairs");
    uint4 b[KP];
#pragma unroll
    for (int kp = 0; kp < KP; ++kp) b[kp] = lds128(tile + (uint32_t)(kp * 4 * G::DP));
    const bool send = !stop && !*gave_up && !(drop && j == 0);
    constexpr int NSP = G::KS >= 4 ? 2 : 1;  // sums of a tile in two chains: with two warps per quadrant, four
    float part[MT][2][4];
    auto push = [&](int m) {
      const int i = warp + m * WP;
      if (!send || (KT % WP != 0 && i >= KT)) return;
      float v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) v[c] = NSP == 2 ? part[m][0][c] + part[m][1][c] : part[m][0][c];
      if (OWN > 0 && i >= KT - OWN) {
        sts128(recv + (j & 1) * G::RB + (uint32_t)((int)crank * G::SLICE + ((i - (KT - OWN)) * 32 + lane) * 16),
               make_uint4(__float_as_uint(v[0]), __float_as_uint(v[2]), __float_as_uint(v[1]), __float_as_uint(v[3])));
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[j & 1]);
      } else {
        st_async_v4(dst[m] + (j & 1) * G::RB, v[0], v[2], v[1], v[3], dbar[m] + (j & 1) * 8);
      }
    };
#pragma unroll
    for (int m = 0; m < MT; ++m) {
#pragma unroll
      for (int k = 0; k < G::KS; ++k) {
        const AFrag& f = A[m][k / 2];
        const uint4 a4 = k & 1 ? make_uint4(f.lo.z, f.hi.z, f.lo.w, f.hi.w) : make_uint4(f.lo.x, f.hi.x, f.lo.y, f.hi.y);
        const uint32_t b0 = k & 1 ? b[k / 2].z : b[k / 2].x, b1 = k & 1 ? b[k / 2].w : b[k / 2].y;
        if (k < NSP) mma_16816_zero(part[m][k % NSP], a4, b0, b1);
        else mma_16816(part[m][k % NSP], a4, b0, b1);
      }
      if (m > 0) push(m - 1);
    }
    push(MT - 1);
  };
  if (HELP && warp >= W) {  // a warp that only multiplies; barriers as in lane_bwd_io
    __syncthreads();
    for (int j = 0; j < T; ++j) {
      __syncthreads();
      if (j == 0) cluster_wait();
      products(j, false);
    }
    __syncwarp();
    cluster_arrive_relaxed();
    cluster_wait();
    return;
  }

  const int ul = CL ? warp * 8 + (gid >> 1) * 2 : warp * 16 + 2 * gid;  // this lane's units within the CTA: ul, ul + 1
  const int unit = (int)crank * U + ul;
  const size_t nd = (size_t)n * D + unit;
  auto row_of = [&](int nb) { return CL ? nb * 8 + 2 * tig + a : (nb >> 1) * 8 + 2 * tig + (nb & 1); };

  bool ok[NB];
  uint32_t cw[NB], sw[NB], dloc[NB];  // activation and state words of row nb in the input ring, delta words in the tile
  F2 car[NB][S], cur[NB][NNEED], dbacc[Gt];  // this lane's two units of row nb
#pragma unroll
  for (int g = 0; g < Gt; ++g) dbacc[g] = v_pair<F2>(0.f, 0.f);
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    const int r = row_of(nb), b = bt0 + r;
    ok[nb] = b < B;
    cw[nb] = sm + G::OFF_I + r * G::CP + ul * 2 * GCM;
    sw[nb] = sm + G::OFF_I + G::IN_S + r * G::SP + ul * (f32 ? 4 : 2);
    dloc[nb] = sm + (r >> 3) * DT + G::doff(r & 7, ul);
#pragma unroll
    for (int s = 0; s < S; ++s) car[nb][s] = v_pair<F2>(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < NNEED; ++k) {
      float2 v = make_float2(1.f, 1.f);
      if (ok[nb]) v = load_state2(p.states, (((size_t)C::need(k) * B + b) * T + (T - 1)) * ND + nd, f32);
      cur[nb][k] = v_pair<F2>(v.x, v.y);
    }
  }
  // gate g's word of a lane lies g * U columns on: a constant distance when U / 8 blocks leave the permutation unchanged
  auto dgate = [&](int nb, int g) -> uint32_t {
    if constexpr (DR || U % 32 == 0) return dloc[nb] + g * (U / 8 * G::DP);
    else return sm + (row_of(nb) >> 3) * DT + opnd_off(row_of(nb) & 7, g * U + ul);
  };

  if constexpr (!FRAGMENTS_FIRST) load_fragments();
  // where this lane's partial sums arrive: source c at + c * (U/16) * NT * 512, batch tile nt at + nt * 512
  const uint32_t rsrc = recv + (uint32_t)((ul >> 4) * NT * 512 + (((ul & 15) >> 1) * 4 + tig) * 16 + a * 8);
  bool poisoned = false;  // a wait expired: it neither waits nor sends any more and the loop runs out
  F2 rec[NB];             // matrix part of dh of the step about to run (CS == 1: handed over in registers)
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) rec[nb] = v_pair<F2>(0.f, 0.f);

  auto wait_partials = [&](int j, int t) {  // sums produced in step index j
    auto expired = [&]() {
      poisoned = true;
      if (HELP) *gave_up = 1;
      report_timeout(p.status, t);
    };
    // re-arm for step index j + 2, never after an expired wait: that phase is still open, no arrival left to give
    if constexpr (G::VOTE) {
      if (!mbar_wait_warp(&full[j & 1], (uint32_t)((j >> 1) & 1), poisoned)) expired();
      mbar_arrive_expect_tx_if(tid == 0 && j + 2 < T && !poisoned, &full[j & 1], STEP_BYTES);
    } else if (!poisoned) {
      if (!mbar_wait_bounded(&full[j & 1], (uint32_t)((j >> 1) & 1))) expired();
      else if (tid == 0 && j + 2 < T) mbar_arrive_expect_tx(&full[j & 1], G::RB);
    }
  };
  auto sum_partials = [&](int j) {
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      F2 v[CS];
#pragma unroll
      for (int c = 0; c < CS; ++c) {
        const uint2 w = lds64(rsrc + (uint32_t)((j & 1) * G::RB + (c * (U / 16) * NT + nb) * 512));
        v[c] = v_pair<F2>(__uint_as_float(w.x), __uint_as_float(w.y));
      }
      // all loads first, then two short addition chains
      F2 x = v[0], y = v[CS > 1 ? 1 : 0];
#pragma unroll
      for (int c = 2; c < CS; ++c) {
        F2& r = (c & 1) ? y : x;
        r = v_add(r, v[c]);
      }
      rec[nb] = v_add(x, y);
    }
  };

  // ---- a step's inputs and what follows from them alone
  uint4 in_c[NB];
  uint32_t in_x[NB];
  uint2 in_s[NB][G::NSS];
  F2 co[NB][BwdCoef<CELL>::N], dext0[NB];
  auto load_inputs = [&](int stage) {
    const uint32_t so = stage * G::IN_B;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      if constexpr (GCM == 4) in_c[nb] = lds128(cw[nb] + so);
      else if constexpr (GCM == 1) in_c[nb].x = lds32(cw[nb] + so);
      if constexpr (GC > 4) in_x[nb] = lds32(sm + G::OFF_I + G::IN_E + row_of(nb) * G::EP + ul * 2 + so);
#pragma unroll
      for (int k = 0; k < G::NSS; ++k) {
        if (f32) in_s[nb][k] = lds64(sw[nb] + so + k * (BT * G::SP));
        else in_s[nb][k].x = lds32(sw[nb] + so + k * (BT * G::SP));
      }
    }
  };
  auto form_coefs = [&]() {
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      F2 chv[GCA], ss[G::NSS];
      if constexpr (GCM > 0) {
        const uint32_t ww[4] = {in_c[nb].x, in_c[nb].y, in_c[nb].z, in_c[nb].w};
#pragma unroll
        for (int k = 0; k < GCM; ++k) chv[k] = v_unpack<F2>(ww[k]);
        if constexpr (GC > 4) chv[GC - 1] = v_unpack<F2>(in_x[nb]);
      }
#pragma unroll
      for (int k = 0; k < G::NSS; ++k)
        ss[k] = f32 ? v_pair<F2>(__uint_as_float(in_s[nb][k].x), __uint_as_float(in_s[nb][k].y)) : v_unpack<F2>(in_s[nb][k].x);
      cell_backward_coef<CELL>(ss + NNEED, car[nb], chv, cur[nb], ss, co[nb]);
      dext0[nb] = ss[NNEED];
#pragma unroll
      for (int k = 0; k < NNEED; ++k) cur[nb][k] = ss[k];
    }
  };

  __syncthreads();  // the inputs of the first step have landed
  int stage = 0;
  for (int j = 0; j < T; ++j) {  // j-th step of the reverse loop, time index t = T-1-j
    const int t = T - 1 - j, buf = j & 1, dbuf = j & (G::NDB - 1);
    load_inputs(stage);
    form_coefs();
    if constexpr (HELP) {  // (left to itself the compiler moves part of this behind the wait: sLSTM D = 256 174 -> 197 us per 256 steps)
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
#pragma unroll
        for (int i = 0; i < BwdCoef<CELL>::N; ++i) v_pin(co[nb][i]);
        v_pin(dext0[nb]);
      }
    }
    if constexpr (CL) {
      if (j > 0) {
        wait_partials(j - 1, t);
        sum_partials(j - 1);
      }
    }
    // ---- gate deltas
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      F2 dR_[Gr], dW_[Gw], dB_[Gt];
      F2 r = car[nb][0];
      if (!p.grad_cut) r = v_add(r, rec[nb]);
      if (p.gclip > 0.f) r = v_clamp(r, p.gclip);
      cell_backward_apply<CELL>(v_add(dext0[nb], r), co[nb], car[nb], dR_, dW_, dB_);
#pragma unroll
      for (int g = 0; g < Gr; ++g) sts32(dgate(nb, g) + dbuf * DB, v_pack(dR_[g]));
      if constexpr (Gr == 3) sts32(dgate(nb, 3) + dbuf * DB, v_pack(dW_[2]));
#pragma unroll
      for (int g = 0; g < Gt; ++g) dbacc[g] = v_add(dbacc[g], dB_[g]);
    }
    if constexpr (DR) {  // the deltas of this step and the one before, see lane_bwd_dr
      if ((j & 1) || j == T - 1) fence_proxy_async_smem();
    }
    __syncthreads();
    // ---- partial dh_{t-1}
    float acc[MT][NT][4];
    if constexpr (!HELP) lane_mma<MT, G::KS, NT, NS, false, G::DP>(A, sm + dbuf * DB, DT, gid, tig, acc, []() {});
    if constexpr (HELP) {
      if (j == 0) cluster_wait();
      products(j, poisoned);
    } else if constexpr (CL) {
      if (j == 0) cluster_wait();
      if (!poisoned && !(drop && j == 0)) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
          if (KT % W == 0 || warp + m * W < KT) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
              st_async_v4(dst[m] + buf * G::RB + nt * 512, acc[m][nt][0], acc[m][nt][2], acc[m][nt][1], acc[m][nt][3], dbar[m] + buf * 8);
          }
      }
    } else {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) rec[nb] = v_pair<F2>(acc[0][nb >> 1][nb & 1], acc[0][nb >> 1][2 + (nb & 1)]);
    }
    stage = stage + 1 == kLaneStages ? 0 : stage + 1;
  }
  if constexpr (CL) {
    wait_partials(T - 1, -1);
    sum_partials(T - 1);
  }

  // ---- cotangent of the initial states, bias gradient
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    if (!ok[nb]) continue;
    const size_t off = (size_t)(bt0 + row_of(nb)) * ND + nd;
    if (!p.grad_cut) car[nb][0] = v_add(car[nb][0], rec[nb]);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const float2 v = v_get(car[nb][s]);
      store_state2(p.ds0, off + (size_t)s * B * ND, f32, v.x, v.y);
    }
  }
#pragma unroll
  for (int g = 0; g < Gt; ++g) {
    const float2 v = v_get(dbacc[g]);
    atomicAdd(p.dbias + (size_t)g * ND + nd, v.x);
    atomicAdd(p.dbias + (size_t)g * ND + nd + 1, v.y);
  }
  if constexpr (DR) {  // dR: row 128 m + 32 warp + lane of the CTA's gate rows lies in this lane's columns [m D, (m + 1) D)
    if (!mbar_wait_bounded(&dr_done[1], 0)) report_timeout(p.status, -1);
    tc_fence_after();
    const uint32_t tcol = *tmem_slot + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
    for (int m = 0; m < G::DRT; ++m) {
      const int row = m * 128 + warp * 32 + lane, g = row / U;
      float* out = p.dR + (((size_t)g * N + n) * D + (int)crank * U + (row - g * U)) * D;
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t r[32];
        tmem_ld32(tcol + m * D + c, r);
        if (row < G::K) {
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            red_add_f32x4(out + c + i, __uint_as_float(r[i]), __uint_as_float(r[i + 1]), __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
        }
      }
    }
    tc_fence_before();
    bar_sync<32 * W + 32>(3);
  }
  // every message to this CTA has been waited for; only after an expired wait can one still be in flight, and then the barrier
  // covers it
  if (CL) { __syncwarp(); cluster_arrive_relaxed(); cluster_wait(); }
}

}  // namespace FRNN_NS
