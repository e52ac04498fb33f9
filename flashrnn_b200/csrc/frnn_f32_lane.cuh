// float32 lane loops (head dims up to 256): one persistent launch runs all T steps; the lane that ends up with a unit's gate sums runs
// its cell.  All products and sums are FFMA in fp32.
//
// Work split.  A cluster of CS = D / U CTAs owns one head and BT = 1, 2, 4 or 8 batch rows; CTA c owns the hidden units [c*U, (c+1)*U), LPU
// lanes each.  Up to head dim 64 CS is 1.
//   Forward: the lanes of a unit split k in interleaved quads; a lane keeps its part of the unit's Gr rows of R in registers (Elman: of
//   the rows of four units, k split over their 4 LPU lanes), so one 16-byte read of h, which costs four wavefronts of shared memory
//   whatever its lanes share, feeds 16 products.  The sums meet through shuffles that scatter the batch rows over the lanes.
//   Reverse: a lane keeps a part of four columns of R.  CS == 1: a warp's own columns, k = (gate, unit) split over 4 LPU lanes, so
//   that dh ends up in the lane that needs it; CS > 1: 16 columns per task, k split over 8 lanes, and the sums go to the CTA that
//   owns the columns.
// LPU is as small as the registers for R allow: the cell is issued once per warp whatever its lanes are worth (LSTM D = 64, one row, 8 lanes
// per unit 1048 clk per step).
// Operand tiles (h, deltas): quads of four consecutive k, [quad][row][4 floats], rows XOR-permuted so that the 8 lanes of a read hit
// different banks; a warp's four units of a row are one quad, so its results and messages are blocks of BT * 16 bytes.
// Exchange: st.async counted on the destination's mbarrier, as in frnn_lane_fwd.cuh.  Four IO warps move everything between global
// memory and shared memory, one CTA barrier per step.
//
// What bounds a step: the chain operand reads -> 8 KQ BT FFMA pairs -> three levels of shuffles -> cell with exact activations, at
// small batches; the FFMA rate at large ones.  See frnn_f32.cu for what it measured against the loops with R in shared memory.
#pragma once
#include "frnn_f32.cuh"

namespace FRNN_NS {

constexpr int kXIoWarps = 4, kXIo = 32 * kXIoWarps;

// byte offset of (quad q, row b) in an operand tile
template <int BT> __host__ __device__ __forceinline__ constexpr uint32_t xq_off(int q, int b) {
  return (uint32_t)(q * BT + (b ^ ((q * BT >> 3) & (BT - 1)))) * 16u;
}
__device__ __forceinline__ void x_unpack(uint4 v, P2& lo, P2& hi) {
  lo = v_pair<P2>(__uint_as_float(v.x), __uint_as_float(v.y));
  hi = v_pair<P2>(__uint_as_float(v.z), __uint_as_float(v.w));
}
// v[i][b], b < BT: sums over the lanes that differ in the bits below LANES; lane l ends up with row l & (BT - 1) in v[i][0]
template <int LANES, int BT, int NV> __device__ __forceinline__ void x_reduce(float (&v)[NV][BT], int lane) {
#pragma unroll
  for (int m = BT / 2; m > 0; m /= 2) {
    const bool hi = (lane & m) != 0;
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int b = 0; b < m; ++b) {
        const float got = __shfl_xor_sync(0xffffffffu, hi ? v[i][b] : v[i][b + m], m);
        v[i][b] = (hi ? v[i][b + m] : v[i][b]) + got;
      }
  }
#pragma unroll
  for (int m = BT; m < LANES; m *= 2)
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i][0] += __shfl_xor_sync(0xffffffffu, v[i][0], m);
}
// v[c][b]: unit c of four, row b; sums over the lanes that differ in the bits below 4 LPU.  Lane bits 2 LPU, LPU <- unit, those below <- row
template <int LPU, int BT> __device__ __forceinline__ float x_reduce_units(const float (&v)[4][BT], int lane) {
  float h[2][BT], o[1][BT];
  const bool hi2 = (lane & (2 * LPU)) != 0, hi1 = (lane & LPU) != 0;
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int e = 0; e < BT; ++e) h[c][e] = (hi2 ? v[c + 2][e] : v[c][e]) + __shfl_xor_sync(0xffffffffu, hi2 ? v[c][e] : v[c + 2][e], 2 * LPU);
#pragma unroll
  for (int e = 0; e < BT; ++e) o[0][e] = (hi1 ? h[1][e] : h[0][e]) + __shfl_xor_sync(0xffffffffu, hi1 ? h[0][e] : h[1][e], LPU);
  x_reduce<LPU, BT, 1>(o, lane);
  return o[0][0];
}
// chunk idx of a [plane][row][quad] walk, quads fastest: idx = (plane * BT + b) * Q + q (inv = 65536 / Q + 1; idx < 65536 / Q)
template <int BT> __device__ __forceinline__ void x_chunk(int idx, int Q, int inv, int& pl, int& b, int& q) {
  const int r = (idx * inv) >> 16;
  q = idx - r * Q;
  b = r & (BT - 1);
  pl = r / BT;
}

// LPU lanes per unit, KQ quads of k per lane
template <int CELL, bool CL, int LPU, int KQ, int BT>
struct XFwdGeom {
  using C = Cell<CELL>;
  static constexpr int KS = C::Gr == 1 ? 4 * LPU : LPU;  // lanes that split k for the same rows of R
  static constexpr int HB = KQ * KS * BT * 16;           // bytes of an h tile
  static constexpr int MAXQ = CL ? 8 : 16, MAXTH = 4 * LPU * MAXQ + kXIo;  // unit quads per CTA, threads, at most
  static constexpr int NR = C::Gr == 1 ? 4 : C::Gr;  // rows of R per lane: a unit's gates, Elman: four units
  static constexpr int GP = NR * KQ * BT > 128 ? 1 : NR * KQ * BT > 64 && KQ == 8 ? 2 : NR;  // of them, those multiplied in one pass over h (registers)
  // Waits by a vote (mbar_wait_warp), except with 2 rows of three or four gates up to head dim 128: us of T256, a vote / a branch per lane, LSTM B8 N2 D = 100 173 / 167, GRU B1 N1 D = 128 164 /
  // 160; with more rows it is the other way round, GRU B64 N4 T64 D = 128 89 / 91.
  static constexpr bool VOTE = CL && !(C::Gr > 1 && LPU == 4 && BT == 2);
  static constexpr int NL = (C::Gw * BT * MAXQ + kXIo - 1) / kXIo, NS = ((C::S + C::GC) * BT * MAXQ + kXIo - 1) / kXIo;  // chunks per IO lane
  static __host__ __device__ constexpr int plane(int U) { return U / 4 * BT * 16; }
  static __host__ __device__ constexpr int off_x() { return 128 + 2 * HB; }
  static __host__ __device__ constexpr int off_o(int U) { return off_x() + kXStages * C::Gw * plane(U); }
  static __host__ __device__ constexpr size_t smem(int U) { return (size_t)off_o(U) + 2 * (size_t)(C::S + C::GC) * plane(U); }
};

template <int CELL, bool CL, int LPU, int KQ, int BT>
__global__ void __launch_bounds__(XFwdGeom<CELL, CL, LPU, KQ, BT>::MAXTH, 1) x32l_fwd_kernel(const __grid_constant__ XParams p) {
  using G = XFwdGeom<CELL, CL, LPU, KQ, BT>;
  using C = Cell<CELL>;
  constexpr int Gr = C::Gr, Gw = C::Gw, Gt = C::Gt, S = C::S, GC = C::GC, GCA = GC > 0 ? GC : 1, HB = G::HB, UW = 32 / LPU, GP = G::GP, NR = G::NR, KS = G::KS;
  const int tid = threadIdx.x, lane = tid & 31, warp = G::VOTE ? warp_index() : tid >> 5;
  const int D = p.D, U = p.U, Q = U >> 2, CS = p.CS, T = p.T, B = p.B, N = p.N;
  const int n = blockIdx.z, b0 = blockIdx.y * BT;
  const uint32_t crank = CL ? cluster_ctarank() : 0u;
  const int unit0 = (int)crank * U, TH = blockDim.x, W = (TH - kXIo) >> 5;  // W compute warps
  const size_t ND = (size_t)N * D;
  const uint32_t step_bytes = (uint32_t)(D * BT * 4);

  extern __shared__ __align__(128) unsigned char xsm[];
  const uint32_t sm = smem_u32(xsm), ht = sm + 128, ring = sm + G::off_x(), out = sm + G::off_o(U);
  const int plane = G::plane(U), xs = Gw * plane, ob = (S + GC) * plane;
  uint64_t* full = reinterpret_cast<uint64_t*>(xsm);  // [2] bytes of h tile x have arrived
  grid_launch_next();
  const int kk = lane & (KS - 1), b = lane & (BT - 1), ul = warp * UW + lane / LPU;  // this lane's unit within the CTA
  const int unit = unit0 + (ul < U ? ul : U - 1);
  // (the other lanes of a unit run the same rows, lanes beyond the last unit run it, and neither stores anything)
  const bool own = (lane & (LPU - 1)) < BT && ul < U, live = b0 + b < B;
  P2 w[NR][KQ][2];  // (nothing else is read before grid_wait_previous: consecutive decoding steps overlap up to there)
  if (warp < W) {
#pragma unroll
    for (int g = 0; g < NR; ++g) {
      const int first = warp * UW + lane / KS * 4 + g, row = Gr == 1 ? unit0 + (first < U ? first : U - 1) : unit;
#pragma unroll
      for (int i = 0; i < KQ; ++i) {
        const int q = i * KS + kk;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (4 * q < D) v = __ldg(reinterpret_cast<const uint4*>(p.R + (((size_t)(Gr == 1 ? 0 : g) * N + n) * D + row) * D + 4 * q));
        x_unpack(v, w[g][i][0], w[g][i][1]);
      }
    }
  }
  grid_wait_previous();
  if (CL && tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    fence_mbar_init();
    if (T > 1) mbar_arrive_expect_tx(&full[0], step_bytes);  // h_0, consumed at step 1
    if (T > 2) mbar_arrive_expect_tx(&full[1], step_bytes);  // h_1
  }
  if (p.clear_status && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
    p.status[0] = 0u; p.status[1] = 0u; p.status[2] = 0u; p.status[3] = 0u;
  }
  // h_{-1} -> tile 1 (step t reads tile (t + 1) & 1 and writes tile t & 1); quads beyond D stay zero in both
  for (int i = tid; i < KQ * KS * BT; i += TH) {
    const int b = i / (KQ * KS), q = i - b * (KQ * KS);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    sts128(ht + xq_off<BT>(q, b), v);
    if (4 * q < D && b0 + b < B) v = *reinterpret_cast<const uint4*>(p.s0 + (size_t)(b0 + b) * ND + (size_t)n * D + 4 * q);
    sts128(ht + HB + xq_off<BT>(q, b), v);
  }
  __syncthreads();
  if (CL) cluster_arrive();  // barriers initialised, h_{-1} read; waited for before the first push, or before `last` may overwrite s0

  if (warp >= W) {
    const int io = tid - 32 * W, inv = 65536 / Q + 1;
    const bool cache = GC > 0 && p.cache != nullptr;
    for (int i = io; i < kXStages * xs / 16; i += kXIo) sts128(ring + i * 16, make_uint4(0u, 0u, 0u, 0u));  // rows beyond B read as zero
    asm volatile("bar.sync 1, %0;" ::"n"(kXIo) : "memory");
    // this lane's chunks: fixed places, pointers that advance by a time step (formed anew in every step, they were what a step waited for)
    const float* lp[G::NL];
    uint32_t ls[G::NL];
#pragma unroll
    for (int i = 0; i < G::NL; ++i) {
      const int idx = io + i * kXIo;
      int g, b, q;
      x_chunk<BT>(idx, Q, inv, g, b, q);
      ls[i] = ring + (uint32_t)((g * Q + q) * BT + b) * 16u;
      lp[i] = idx < Gw * BT * Q && b0 + b < B ? p.Wx + (size_t)(b0 + b) * p.wx_sb + (size_t)g * p.wx_sg + (size_t)n * p.wx_sn + unit0 + 4 * q : nullptr;
    }
    float* sp[G::NS];
    uint32_t ss[G::NS], act = 0;  // bit i: chunk i is an activation
#pragma unroll
    for (int i = 0; i < G::NS; ++i) {
      const int idx = io + i * kXIo;
      int pl, b, q;
      x_chunk<BT>(idx, Q, inv, pl, b, q);
      const size_t bg = b0 + b, col = (size_t)n * D + unit0 + 4 * q;
      ss[i] = out + (uint32_t)((pl * Q + q) * BT + b) * 16u;
      sp[i] = idx >= (S + (cache ? GC : 0)) * BT * Q || b0 + b >= B ? nullptr
              : pl < S                                              ? p.states + ((size_t)pl * B + bg) * T * ND + col
                                                                    : p.cache + (bg * T * GCA + (pl - S)) * ND + col;
      if (pl >= S) act |= 1u << i;
    }
    auto load = [&](int t, int stage) {  // in step order
      if (t < T) {
#pragma unroll
        for (int i = 0; i < G::NL; ++i)
          if (lp[i] != nullptr) {
            cp_async16_u32(ls[i] + stage * xs, lp[i]);
            lp[i] += p.wx_st;
          }
      }
      cp_async_commit();
    };
    auto store = [&](int t) {  // in step order
#pragma unroll
      for (int i = 0; i < G::NS; ++i)
        if (sp[i] != nullptr) {
          *reinterpret_cast<uint4*>(sp[i]) = lds128(ss[i] + (t & 1) * ob);
          sp[i] += (act >> i & 1u) ? GCA * ND : ND;
        }
    };
#pragma unroll 1
    for (int s = 0; s < kXStages; ++s) load(s, s);
    cp_async_wait<kXStages - 2>();
    __syncthreads();  // Wx of steps 0 and 1
    int stage = 0;
    // barrier t of the CTA: Wx of step t + 1 has landed; that of step t has been read and its results are staged
    for (int t = 0; t < T; ++t) {
      cp_async_wait<kXStages - 2>();
      __syncthreads();
      load(t + kXStages, stage);
      store(t);
      stage = stage + 1 == kXStages ? 0 : stage + 1;
    }
    cp_async_wait<0>();
    if (CL) {
      __syncwarp();
      cluster_wait();
      cluster_arrive_relaxed();
      cluster_wait();
    }
    return;
  }

  const size_t nd = (size_t)n * D + unit;
  float bias[Gt], st[S], cch[GCA];
#pragma unroll
  for (int g = 0; g < Gt; ++g) bias[g] = p.bias[(size_t)g * ND + nd];
#pragma unroll
  for (int s = 0; s < S; ++s) st[s] = live ? p.s0[((size_t)s * B + b0 + b) * ND + nd] : 0.f;
  const int uc = unit - unit0;
  const uint32_t word = (uint32_t)((uc >> 2) * BT + b) * 16u + (uint32_t)(uc & 3) * 4u;  // this lane's word in a plane of the ring, of the results
  const uint32_t hw = xq_off<BT>(unit >> 2, b) + (uint32_t)(unit & 3) * 4u;              // ... in an h tile
  const uint32_t hr = ht + (uint32_t)(kk * BT) * 16u, sw = (uint32_t)(kk * BT >> 3) & (BT - 1);
  const int drop_t = (p.test_drop && crank == 0) ? 1 : -1;  // test hook: CTA 0 withholds its message of step 1
  const bool cache = GC > 0 && p.cache != nullptr;
  bool poisoned = false;  // a wait expired: it neither waits nor sends any more and the loop runs out
  __syncthreads();        // Wx of steps 0 and 1 has landed
  int stage = 0;
  for (int t = 0; t < T; ++t) {
    const int prv = (t + 1) & 1, nxt = t & 1;
    float wx[Gw];
#pragma unroll
    for (int g = 0; g < Gw; ++g) wx[g] = __uint_as_float(lds32(ring + stage * xs + g * plane + word));
    if constexpr (G::VOTE) {
      if (t > 0) {
        if (!mbar_wait_warp(&full[prv], (uint32_t)(((t - 1) >> 1) & 1), poisoned)) {
          poisoned = true;
          if (lane == 0) report_timeout(p.status, t);
        }
        mbar_arrive_expect_tx_if(tid == 0 && t + 2 < T && !poisoned, &full[prv], step_bytes);
      }
    } else if (CL && t > 0 && !poisoned) {
      if (!mbar_wait_bounded(&full[prv], (uint32_t)(((t - 1) >> 1) & 1))) {
        poisoned = true;
        report_timeout(p.status, t);
      }
      else if (tid == 0 && t + 2 < T) mbar_arrive_expect_tx(&full[prv], step_bytes);
    }
    float v[NR][BT], pre[Gr], gx[Gt];
#pragma unroll
    for (int g0 = 0; g0 < NR; g0 += GP) {
      P2 acc[GP][BT];
#pragma unroll
      for (int i = 0; i < KQ; ++i) {
        P2 lo[BT], hi[BT];
        constexpr int kRow = KS * BT;
#pragma unroll
        for (int r = 0; r < BT; ++r)  // quad i * KS + kk; the row's place splits into a part of i and one of kk
          x_unpack(lds128(hr + prv * HB + (uint32_t)(i * kRow) * 16u + (((uint32_t)(r ^ ((i * kRow >> 3) & (BT - 1))) ^ sw) << 4)), lo[r], hi[r]);
#pragma unroll
        for (int g = 0; g < GP; ++g)
          if (g0 + g < NR)
#pragma unroll
            for (int r = 0; r < BT; ++r) acc[g][r] = i == 0 ? v_mul(w[g0 + g][i][0], lo[r]) : v_fma(w[g0 + g][i][0], lo[r], acc[g][r]);
#pragma unroll
        for (int g = 0; g < GP; ++g)
          if (g0 + g < NR)
#pragma unroll
            for (int r = 0; r < BT; ++r) acc[g][r] = v_fma(w[g0 + g][i][1], hi[r], acc[g][r]);
      }
#pragma unroll
      for (int g = 0; g < GP; ++g)
        if (g0 + g < NR)
#pragma unroll
          for (int r = 0; r < BT; ++r) { const float2 s = v_get(acc[g][r]); v[g0 + g][r] = s.x + s.y; }
    }
    if constexpr (Gr == 1) {
      pre[0] = x_reduce_units<LPU, BT>(v, lane);
    } else {
      x_reduce<LPU, BT, Gr>(v, lane);
#pragma unroll
      for (int g = 0; g < Gr; ++g) pre[g] = v[g][0];
    }
    gate_sums<CELL>(pre, wx, bias, gx);
    cell_forward<CELL>(gx, st, cch);
    if (p.fclip > 0.f) st[0] = clampf(st[0], p.fclip);
    if constexpr (CL) {
      if (t == 0) cluster_wait();
      if (own && t + 1 < T && t != drop_t && !poisoned) {
#pragma unroll 1
        for (int c = 0; c < CS; ++c) {
          const uint32_t r = crank + 1 + c, peer = map_to_cta(sm, r >= (uint32_t)CS ? r - CS : r);
          st_async_b32(peer + 128u + nxt * HB + hw, __float_as_uint(st[0]), peer + nxt * 8);
        }
      }
    } else {
      if (own) sts32(ht + nxt * HB + hw, __float_as_uint(st[0]));
    }
    if (own) {
#pragma unroll
      for (int s = 0; s < S; ++s) sts32(out + nxt * ob + s * plane + word, __float_as_uint(st[s]));
      if (cache) {
#pragma unroll
        for (int k = 0; k < GC; ++k) sts32(out + nxt * ob + (S + k) * plane + word, __float_as_uint(cch[k]));
      }
    }
    __syncthreads();
    stage = stage + 1 == kXStages ? 0 : stage + 1;
  }
  if (p.last != nullptr && own && live) {
#pragma unroll
    for (int s = 0; s < S; ++s) p.last[((size_t)s * B + b0 + b) * ND + nd] = st[s];
  }
  // every message has been waited for; only after an expired wait can one still be in flight, and the barrier covers it
  if (CL) { __syncwarp(); cluster_arrive_relaxed(); cluster_wait(); }
}

// LPU lanes per unit.  k is split over KS = 4 LPU lanes with one CTA per head (a warp's own columns, so that dh ends up in the lane that runs
// the unit), over 8 in clusters; KQ quads of k per lane, TB tasks of 128 / KS columns per warp
template <int CELL, bool CL, int LPU, int KQ, int TB, int BT>
struct XBwdGeom {
  using C = Cell<CELL>;
  static constexpr int PL = C::Gr == 3 ? 4 : C::Gr;  // planes of the delta tile: the R gates; the GRU's input-only gate behind them
  static constexpr int NIN = C::GC + C::NNEED + C::NEXT;
  // Waits by a vote (mbar_wait_warp), except with three column tasks per warp (head dims 100 and 120) and four gates: us, a vote / a branch per lane, sLSTM D = 100 B8
  // T256 N2 329 / 316, LSTM D = 100 B256 T32 N6 945 / 920; elsewhere 2 to 4 % the other way round, LSTM B8 T256 N2 D = 128 241 / 249.
  static constexpr bool VOTE = CL && !(TB == 3 && C::Gr == 4);
  static constexpr int KS = CL ? 8 : 4 * LPU;
  static constexpr int MAXQ = CL ? 8 : 16, MAXTH = 4 * LPU * MAXQ + kXIo;
  static constexpr int NL = (NIN * BT * MAXQ + kXIo - 1) / kXIo, NS = ((C::Gw + (C::Gr == 3 ? 1 : 0)) * BT * MAXQ + kXIo - 1) / kXIo;
  static __host__ __device__ constexpr int plane(int U) { return U / 4 * BT * 16; }
  static __host__ __device__ constexpr int db(int U) { return PL * plane(U) > KS * KQ * BT * 16 ? PL * plane(U) : KS * KQ * BT * 16; }
  static __host__ __device__ constexpr int off_i(int U) { return 128 + 2 * db(U); }
  static __host__ __device__ constexpr int off_r(int U) { return off_i(U) + kXStages * NIN * plane(U); }
  static __host__ __device__ constexpr size_t smem(int U, int CS) { return (size_t)off_r(U) + (CS > 1 ? 2 * (size_t)CS * plane(U) : 0); }
};

template <int CELL, bool CL, int LPU, int KQ, int TB, int BT>
__global__ void __launch_bounds__(XBwdGeom<CELL, CL, LPU, KQ, TB, BT>::MAXTH, 1) x32l_bwd_kernel(const __grid_constant__ XParams p) {
  using G = XBwdGeom<CELL, CL, LPU, KQ, TB, BT>;
  using C = Cell<CELL>;
  constexpr int Gr = C::Gr, Gw = C::Gw, Gt = C::Gt, S = C::S, GC = C::GC, GCA = GC > 0 ? GC : 1, NNEED = C::NNEED, NEXT = C::NEXT, NIN = G::NIN, KS = G::KS, UW = 32 / LPU;
  constexpr int GSH = Gr == 3 ? 1 : 0;  // GRU: plane 0 is the recurrent-only gate, which goes to dg0
  const int tid = threadIdx.x, lane = tid & 31, warp = G::VOTE ? warp_index() : tid >> 5;
  const int D = p.D, U = p.U, Q = U >> 2, CS = p.CS, T = p.T, B = p.B, N = p.N;
  const int n = blockIdx.z, b0 = blockIdx.y * BT;
  const uint32_t crank = CL ? cluster_ctarank() : 0u;
  const int unit0 = (int)crank * U, TH = blockDim.x, W = (TH - kXIo) >> 5;
  const size_t ND = (size_t)N * D, col = (size_t)n * D + unit0;
  const bool exch = !p.grad_cut;  // with the recurrent gradient cut no dh crosses a step: no products, no exchange

  extern __shared__ __align__(128) unsigned char xsm[];
  const int plane = G::plane(U), db = G::db(U), xs = NIN * plane, rb = CS * plane;
  const uint32_t sm = smem_u32(xsm), dt = sm + 128, ring = sm + G::off_i(U), recv = sm + G::off_r(U);
  uint64_t* full = reinterpret_cast<uint64_t*>(xsm);  // [2] bytes of partial sums have arrived
  if (CL && tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    fence_mbar_init();
    if (exch) {
      mbar_arrive_expect_tx(&full[0], rb);             // partial sums of step index 0 (t = T-1)
      if (T > 1) mbar_arrive_expect_tx(&full[1], rb);  // step index 1
    }
  }
  for (int i = tid; i < 2 * db / 16; i += TH) sts128(dt + i * 16, make_uint4(0u, 0u, 0u, 0u));  // (padding quads stay zero)
  __syncthreads();
  if (CL) cluster_arrive();  // waited for before the first push

  if (warp >= W) {
    const int io = tid - 32 * W, inv = 65536 / Q + 1;
    // rows beyond B: zero activations and cotangents make their deltas zero; their states only have to be finite divisors
    for (int i = io; i < kXStages * xs / 16; i += kXIo) {
      const int pl = i * 16 % xs / plane;
      const uint32_t v = pl >= GC && pl < GC + NNEED ? 0x3f800000u : 0u;
      sts128(ring + i * 16, make_uint4(v, v, v, v));
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kXIo) : "memory");
    const float* lp[G::NL];
    uint32_t ls[G::NL], kind = 0;  // two bits per chunk: activation, state, cotangent
#pragma unroll
    for (int i = 0; i < G::NL; ++i) {
      const int idx = io + i * kXIo;
      int pl, b, q;
      x_chunk<BT>(idx, Q, inv, pl, b, q);
      const size_t bg = b0 + b;
      ls[i] = ring + (uint32_t)((pl * Q + q) * BT + b) * 16u;
      if (idx >= NIN * BT * Q || b0 + b >= B) {
        lp[i] = nullptr;
      } else if (pl < GC) {
        lp[i] = p.cache + ((bg * T + (T - 1)) * GCA + pl) * ND + col + 4 * q;
      } else if (pl < GC + NNEED) {  // states at t - 1
        lp[i] = p.states + (((size_t)C::need(pl - GC) * B + bg) * T + (T - 1)) * ND - ND + col + 4 * q;
        kind |= 1u << (2 * i);
      } else {
        lp[i] = p.dstates + (size_t)(pl - GC - NNEED) * p.ds_ss + bg * p.ds_sb + (size_t)(T - 1) * p.ds_st + (size_t)n * p.ds_sn + unit0 + 4 * q;
        kind |= 2u << (2 * i);
      }
    }
    auto load = [&](int t, int stage) {  // in step order T-1, T-2, ...
      if (t >= 0) {
#pragma unroll
        for (int i = 0; i < G::NL; ++i)
          if (lp[i] != nullptr) {
            const uint32_t k = kind >> (2 * i) & 3u;
            const float* src = lp[i];
            if (k == 1u && t == 0) {  // the initial state takes the place of states[-1]
              int pl, b, q;
              x_chunk<BT>(io + i * kXIo, Q, inv, pl, b, q);
              src = p.s0 + ((size_t)C::need(pl - GC) * B + b0 + b) * ND + col + 4 * q;
            }
            cp_async16_u32(ls[i] + stage * xs, src);
            lp[i] -= k == 0u ? GCA * ND : k == 1u ? ND : (size_t)p.ds_st;
          }
      }
      cp_async_commit();
    };
    float* sp[G::NS];
    uint32_t ss[G::NS], first = 0;  // bit i: chunk i goes to dg0
#pragma unroll
    for (int i = 0; i < G::NS; ++i) {
      const int idx = io + i * kXIo;
      int pl, b, q;
      x_chunk<BT>(idx, Q, inv, pl, b, q);
      const size_t row = (size_t)(b0 + b) * T + (T - 1);
      ss[i] = dt + xq_off<BT>(pl * Q + q, b);
      sp[i] = idx >= (Gw + GSH) * BT * Q || b0 + b >= B ? nullptr
              : GSH && pl == 0                          ? p.dg0 + row * ND + col + 4 * q
                                                        : p.dWx + (row * Gw + (pl - GSH)) * ND + col + 4 * q;
      if (GSH && pl == 0) first |= 1u << i;
    }
    auto store = [&](int j) {  // the deltas of step index j
#pragma unroll
      for (int i = 0; i < G::NS; ++i)
        if (sp[i] != nullptr) {
          *reinterpret_cast<uint4*>(sp[i]) = lds128(ss[i] + (j & 1) * db);
          sp[i] -= (first >> i & 1u) ? ND : Gw * ND;
        }
    };
#pragma unroll 1
    for (int s = 0; s < kXStages; ++s) load(T - 1 - s, s);
    cp_async_wait<kXStages - 1>();
    __syncthreads();  // the inputs of the first step
    int stage = 0;
    // barrier j of the CTA: the deltas of step j are complete, its inputs consumed, the inputs of step j + 1 have landed
    for (int j = 0; j < T; ++j) {
      cp_async_wait<kXStages - 2>();
      __syncthreads();
      load(T - 1 - j - kXStages, stage);
      store(j);
      stage = stage + 1 == kXStages ? 0 : stage + 1;
    }
    cp_async_wait<0>();
    if (CL) {
      __syncwarp();
      cluster_wait();
      cluster_arrive_relaxed();
      cluster_wait();
    }
    return;
  }

  const int kk = lane & (KS - 1), b = lane & (BT - 1), ul = warp * UW + lane / LPU, uc = ul < U ? ul : U - 1, unit = unit0 + uc;
  const bool own = (lane & (LPU - 1)) < BT && ul < U, live = b0 + b < B;
  const size_t nd = (size_t)n * D + unit;
  auto column0 = [&](int i) { return CL ? (warp + i * W) * 16 + (lane >> 3) * 4 : warp * UW + lane / KS * 4; };  // of task i
  P2 w[TB][4][KQ][2];  // column, k quad (gate, unit quad)
#pragma unroll
  for (int i = 0; i < TB; ++i) {
    const int c0 = column0(i);
#pragma unroll
    for (int k = 0; k < KQ; ++k) {
      const int q = k * KS + kk, g = q / Q, u = unit0 + 4 * (q - g * Q);
      float4 r[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        r[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q < Gr * Q && c0 < D) r[e] = __ldg(reinterpret_cast<const float4*>(p.R + (((size_t)g * N + n) * D + u + e) * D + c0));
      }
      w[i][0][k][0] = v_pair<P2>(r[0].x, r[1].x); w[i][0][k][1] = v_pair<P2>(r[2].x, r[3].x);
      w[i][1][k][0] = v_pair<P2>(r[0].y, r[1].y); w[i][1][k][1] = v_pair<P2>(r[2].y, r[3].y);
      w[i][2][k][0] = v_pair<P2>(r[0].z, r[1].z); w[i][2][k][1] = v_pair<P2>(r[2].z, r[3].z);
      w[i][3][k][0] = v_pair<P2>(r[0].w, r[1].w); w[i][3][k][1] = v_pair<P2>(r[2].w, r[3].w);
    }
  }
  float car[S], cur[NNEED], dbacc[Gt], rec = 0.f;
#pragma unroll
  for (int s = 0; s < S; ++s) car[s] = 0.f;
#pragma unroll
  for (int g = 0; g < Gt; ++g) dbacc[g] = 0.f;
#pragma unroll
  for (int k = 0; k < NNEED; ++k) cur[k] = live ? p.states[(((size_t)C::need(k) * B + b0 + b) * T + (T - 1)) * ND + nd] : 1.f;
  const uint32_t word = (uint32_t)((uc >> 2) * BT + b) * 16u + (uint32_t)(uc & 3) * 4u;
  const uint32_t dr = dt + (uint32_t)(kk * BT) * 16u, sw = (uint32_t)(kk * BT >> 3) & (BT - 1);
  const bool drop = p.test_drop && crank == 0;  // test hook: CTA 0 withholds its message of the second step
  bool poisoned = false;
  auto collect = [&](int j, int t) {  // CS > 1: the partial sums of step index j
    if constexpr (G::VOTE) {
      if (!mbar_wait_warp(&full[j & 1], (uint32_t)((j >> 1) & 1), poisoned)) {
        poisoned = true;
        if (lane == 0) report_timeout(p.status, t);
      }
      mbar_arrive_expect_tx_if(tid == 0 && j + 2 < T && !poisoned, &full[j & 1], rb);
    } else if (!poisoned) {
      if (!mbar_wait_bounded(&full[j & 1], (uint32_t)((j >> 1) & 1))) {
        poisoned = true;
        report_timeout(p.status, t);
      }
      else if (tid == 0 && j + 2 < T) mbar_arrive_expect_tx(&full[j & 1], rb);
    }
    float x = 0.f, y = 0.f;
#pragma unroll 2
    for (int c = 0; c < CS; ++c) {
      const float s = __uint_as_float(lds32(recv + (j & 1) * rb + c * plane + word));
      if (c & 1) y += s; else x += s;
    }
    rec = x + y;
  };
  __syncthreads();  // the inputs of the first step have landed
  int stage = 0;
  for (int j = 0; j < T; ++j) {  // j-th step of the reverse loop, time index t = T-1-j
    const uint32_t in = ring + stage * xs + word;
    float cv[GCA], prv[NNEED], ext[NEXT], co[BwdCoef<CELL>::N], dR_[Gr], dW_[Gw], dB_[Gt];
#pragma unroll
    for (int k = 0; k < GC; ++k) cv[k] = __uint_as_float(lds32(in + k * plane));
#pragma unroll
    for (int k = 0; k < NNEED; ++k) prv[k] = __uint_as_float(lds32(in + (GC + k) * plane));
#pragma unroll
    for (int k = 0; k < NEXT; ++k) ext[k] = __uint_as_float(lds32(in + (GC + NNEED + k) * plane));
    cell_backward_coef<CELL>(ext, car, cv, cur, prv, co);
    if (CL && exch && j > 0) collect(j - 1, T - 1 - j);
    float r = car[0] + rec;
    if (p.gclip > 0.f) r = clampf(r, p.gclip);
    cell_backward_apply<CELL>(ext[0] + r, co, car, dR_, dW_, dB_);
    if (own) {
#pragma unroll
      for (int g = 0; g < Gr; ++g) sts32(dt + (j & 1) * db + xq_off<BT>(g * Q + (uc >> 2), b) + (uc & 3) * 4u, __float_as_uint(dR_[g]));
      if constexpr (GSH) sts32(dt + (j & 1) * db + xq_off<BT>(3 * Q + (uc >> 2), b) + (uc & 3) * 4u, __float_as_uint(dW_[2]));
    }
#pragma unroll
    for (int g = 0; g < Gt; ++g) dbacc[g] += dB_[g];
#pragma unroll
    for (int k = 0; k < NNEED; ++k) cur[k] = prv[k];
    __syncthreads();
    if (CL && j == 0) cluster_wait();
    stage = stage + 1 == kXStages ? 0 : stage + 1;
    if (!exch) continue;
    // ---- dh_{t-1} of this CTA's deltas
#pragma unroll
    for (int i = 0; i < TB; ++i) {
      P2 acc[4][BT];
#pragma unroll
      for (int k = 0; k < KQ; ++k) {
        P2 lo[BT], hi[BT];
#pragma unroll
        for (int e = 0; e < BT; ++e) x_unpack(lds128(dr + (j & 1) * db + (uint32_t)(k * KS * BT) * 16u + (((uint32_t)e ^ sw) << 4)), lo[e], hi[e]);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int e = 0; e < BT; ++e) acc[c][e] = k == 0 ? v_mul(w[i][c][k][0], lo[e]) : v_fma(w[i][c][k][0], lo[e], acc[c][e]);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int e = 0; e < BT; ++e) acc[c][e] = v_fma(w[i][c][k][1], hi[e], acc[c][e]);
      }
      float v[4][BT];
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int e = 0; e < BT; ++e) { const float2 s = v_get(acc[c][e]); v[c][e] = s.x + s.y; }
      if constexpr (!CL) {
        rec = x_reduce_units<LPU, BT>(v, lane);
      } else {
        x_reduce<8, BT, 4>(v, lane);
        const int cq = column0(i) >> 2, owner = cq / Q;  // the quad of columns
        if ((lane & 7) < BT && owner < CS && !poisoned && !(drop && j == 1)) {
          const uint32_t peer = map_to_cta(sm, (uint32_t)owner);
          st_async_v4(peer + (recv - sm) + (uint32_t)((j & 1) * rb + (int)crank * plane + ((cq - owner * Q) * BT + b) * 16), v[0][0], v[1][0], v[2][0],
                      v[3][0], peer + (j & 1) * 8);
        }
      }
    }
  }
  if (CL && exch) collect(T - 1, -1);
  // ---- cotangents of the initial states (h: the carried part and the matrix part of the last step), bias gradient
  if (own && live) {
    p.ds0[(size_t)(b0 + b) * ND + nd] = car[0] + rec;
#pragma unroll
    for (int s = 1; s < S; ++s) p.ds0[((size_t)s * B + b0 + b) * ND + nd] = car[s];
  }
#pragma unroll
  for (int g = 0; g < Gt; ++g) {
#pragma unroll
    for (int m = 1; m < BT; m *= 2) dbacc[g] += __shfl_xor_sync(0xffffffffu, dbacc[g], m);
    if ((lane & (LPU - 1)) == 0 && ul < U) atomicAdd(p.dbias + (size_t)g * ND + nd, dbacc[g]);
  }
  if (CL) { __syncwarp(); cluster_arrive_relaxed(); cluster_wait(); }
}

}  // namespace FRNN_NS
