// Reverse time loop for head dims above 256: the reverse lane loop (frnn_lane_bwd.cuh) with the geometry of frnn_big_fwd.cuh.  A warp
// owns up to four 16-row tiles of p and all K = Gr * U gate rows of its CTA; KRP of its k-pairs are in registers, the next in
// tensor memory (see the forward loop), then in shared memory, the rest comes from L2 (CTAs of 64 units: with 8 rows LSTM from head dim 960, sLSTM from 704 up,
// with 16 rows LSTM from 576, sLSTM from 448 up).  Twice as many warps multiply as run the cell (U / 8); the other half moves the data
// meanwhile.  The sums of a tile, or a pair of tiles, leave as soon as they are complete, so their exchange overlaps the products of the next.
// K is padded to a multiple of 32 with zero fragments (the delta columns there are zero, or the GRU's input-only gate).
//
// Replaces FLASHRNNCellFusedBackward (reference flashrnn/flashrnn/fused/flashrnn_fused_backward.cu:129-624).
#pragma once
#include "frnn_big_fwd.cuh"
#include "frnn_lane_bwd.cuh"

namespace FRNN_NS {

template <int CELL, int U, int NT>
struct BigBwdGeom {
  using C = Cell<CELL>;
  static constexpr int BT = 8 * NT, NT8 = NT, UNITS = U, STAGES = kBigStages - 1;
  static constexpr bool CL = true;
  static constexpr int WC = U / 8, W = 2 * WC, IOT = 32 * (W - WC), TH = 32 * W;  // warps of the cell, of the products; the others move the data
  static constexpr int NB = NT;
  static constexpr int K = C::Gr * U, KP = (K + 31) / 32;
  static constexpr int MT = 4;  // p tiles per warp, at most: D / 16 <= 4 W
  static constexpr int GCM = CacheGeom<C::GC>::MAIN;
  static constexpr bool GCX = CacheGeom<C::GC>::EXTRA;
  static constexpr int NSS = C::NNEED + C::NEXT;
  static constexpr int KRP_WANT = U == 32 ? 4 : U == 48 ? 3 : 2, KRP = KRP_WANT < KP ? KRP_WANT : KP;
  static constexpr int DCOLS = C::Gr == 3 ? 4 * U : KP * 32, DT = opnd_bytes(DCOLS), DB = NT * DT;
  static constexpr bool DR = false;
  static __host__ __device__ constexpr uint32_t doff(uint32_t row, uint32_t k) { return opnd_off(row, k); }
  static constexpr int CP = io_pitch(U * 2 * GCM), EP = io_pitch(U * 2), SP = io_pitch(U * 4);
  static constexpr int IN_E = GCM ? BT * CP : 0, IN_S = IN_E + (GCX ? BT * EP : 0), IN_B = IN_S + NSS * BT * SP;
  // shared memory: barriers | delta tiles | input ring | 2 x partial sums received | fragments of R^T
  static constexpr int OFF_D = 128, OFF_I = OFF_D + 2 * DB, OFF_V = (OFF_I + STAGES * IN_B + 127) / 128 * 128;
  static __host__ __device__ constexpr int recv_bytes(int D) { return D / 16 * 512 * NT; }  // of one step
  static __host__ __device__ constexpr int off_r(int D) { return OFF_V + 2 * recv_bytes(D); }
  static __host__ __device__ constexpr int tiles(int D) { return (D / 16 + W - 1) / W; }  // p tiles per warp
  // tiles are multiplied MG at a time, one read of the deltas for both (U = 48, D = 768 LSTM step 5240 -> 4610 clk; with all of R^T in registers
  // one by one, in two accumulator sets: D = 512 2235 -> 2030); units of one k-pair of them per warp in shared memory, in the order of use
  static constexpr int MG = U == 32 ? 1 : 2;
  static constexpr int KL = KP - KRP;  // k-pairs beyond those in registers
  // of them, those in tensor memory, for each group of MG tiles: a lane's 16 words of a k-pair of a group lie in 16 columns of its own lane
  static constexpr bool TM = MG == 2 && KL > 0;
  static constexpr int TCOLS = TM ? 512 / (W / 4) / 16 * 16 : 0, TFIT = TCOLS / 16 / (MT / MG), KT = KL < TFIT ? KL : TFIT;
  static __host__ __device__ constexpr int fsm(int D) {
    const int want = (tiles(D) + MG - 1) / MG * (KL - KT), fit = ((int)kSmemBudget - off_r(D)) / (W * MG * 1024);
    return want < fit ? want : (fit < 0 ? 0 : fit);
  }
  static __host__ __device__ constexpr size_t smem(int D) { return tmem_alone(TM, (size_t)off_r(D) + (size_t)fsm(D) * W * MG * 1024); }
};

// One compute lane: two adjacent units of NB batch rows.  (lane_bwd_kernel has the same in local variables.  With this struct in its place
// the compiler gives its loops other registers: LSTM D = 96 B1024 502 -> 646 us, D = 64 582 -> 621, GRU D = 128 536 -> 563, geometric mean of 182 problems 1.00.)
template <int CELL, class G, class F2>
struct BwdLane {
  using C = Cell<CELL>;
  static constexpr int Gr = C::Gr, Gw = C::Gw, Gt = C::Gt, S = C::S, GC = C::GC, GCA = GC > 0 ? GC : 1, NNEED = C::NNEED, NEXT = C::NEXT;
  static constexpr int NB = G::NB, BT = G::BT, U = G::UNITS, GCM = G::GCM, NSS = G::NSS;
  F2 car[NB][S], cur[NB][NNEED], dbacc[Gt];
  F2 co[NB][BwdCoef<CELL>::N], dext0[NB];     // what the step's deltas need beside the recurrent part of dh
  uint32_t cw[NB], ew[NB], sw[NB], dloc[NB];  // activation and state words of row nb in the input ring, delta words in the tile
  uint4 in_c[NB];
  uint32_t in_x[NB];
  uint2 in_s[NB][NSS];
  size_t nd;
  int a, tig, bt0, f32, ul, dt;
  uint32_t d0;

  __device__ __forceinline__ int row_of(int nb) const { return nb * 8 + 2 * tig + a; }
  // d0: delta tiles (dt bytes per 8 rows), in: input ring; ul: first unit within the CTA, unit: within the head
  __device__ __forceinline__ void init(const LoopParams& p, uint32_t d0_, int dt_, uint32_t in, int lane, int ul_, int unit, int n, int bt0_) {
    const size_t ND = (size_t)p.N * p.D;
    a = (lane >> 2) & 1; tig = lane & 3; bt0 = bt0_; f32 = p.state_f32; ul = ul_; dt = dt_; d0 = d0_;
    nd = (size_t)n * p.D + unit;
#pragma unroll
    for (int g = 0; g < Gt; ++g) dbacc[g] = v_pair<F2>(0.f, 0.f);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const int r = row_of(nb), b = bt0 + r;
      cw[nb] = in + r * G::CP + ul * 2 * GCM;
      ew[nb] = in + G::IN_E + r * G::EP + ul * 2;
      sw[nb] = in + G::IN_S + r * G::SP + ul * (f32 ? 4 : 2);
      dloc[nb] = d0 + (r >> 3) * dt + opnd_off(r & 7, ul);
#pragma unroll
      for (int s = 0; s < S; ++s) car[nb][s] = v_pair<F2>(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < NNEED; ++k) {
        float2 v = make_float2(1.f, 1.f);
        if (b < p.B) v = load_state2(p.states, (((size_t)C::need(k) * p.B + b) * p.T + (p.T - 1)) * ND + nd, f32);
        cur[nb][k] = v_pair<F2>(v.x, v.y);
      }
    }
  }
  __device__ __forceinline__ void load_inputs(int stage) {
    const uint32_t so = stage * G::IN_B;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      if constexpr (GCM == 4) in_c[nb] = lds128(cw[nb] + so);
      else if constexpr (GCM == 1) in_c[nb].x = lds32(cw[nb] + so);
      if constexpr (GC > 4) in_x[nb] = lds32(ew[nb] + so);
#pragma unroll
      for (int k = 0; k < NSS; ++k) {
        if (f32) in_s[nb][k] = lds64(sw[nb] + so + k * (BT * G::SP));
        else in_s[nb][k].x = lds32(sw[nb] + so + k * (BT * G::SP));
      }
    }
  }
  __device__ __forceinline__ void form_coefs() {
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      F2 chv[GCA], ss[NSS];
      if constexpr (GCM > 0) {
        const uint32_t ww[4] = {in_c[nb].x, in_c[nb].y, in_c[nb].z, in_c[nb].w};
#pragma unroll
        for (int k = 0; k < GCM; ++k) chv[k] = v_unpack<F2>(ww[k]);
        if constexpr (GC > 4) chv[GC - 1] = v_unpack<F2>(in_x[nb]);
      }
#pragma unroll
      for (int k = 0; k < NSS; ++k)
        ss[k] = f32 ? v_pair<F2>(__uint_as_float(in_s[nb][k].x), __uint_as_float(in_s[nb][k].y)) : v_unpack<F2>(in_s[nb][k].x);
      cell_backward_coef<CELL>(ss + NNEED, car[nb], chv, cur[nb], ss, co[nb]);
      dext0[nb] = ss[NNEED];
#pragma unroll
      for (int k = 0; k < NNEED; ++k) cur[nb][k] = ss[k];
    }
  }
  // gate g's word of a lane lies g * U columns on: a constant distance when U / 8 blocks leave the permutation unchanged
  __device__ __forceinline__ uint32_t dgate(int nb, int g) const {
    if constexpr (U % 32 == 0) return dloc[nb] + g * (U * 16);
    else return d0 + (row_of(nb) >> 3) * dt + opnd_off(row_of(nb) & 7, g * U + ul);
  }
  // the step's gate deltas into the tile at `off`; rec: recurrent part of dh
  __device__ __forceinline__ void deltas(const LoopParams& p, const F2 (&rec)[NB], uint32_t off) {
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      F2 dR_[Gr], dW_[Gw], dB_[Gt];
      F2 r = car[nb][0];
      if (!p.grad_cut) r = v_add(r, rec[nb]);
      if (p.gclip > 0.f) r = v_clamp(r, p.gclip);
      cell_backward_apply<CELL>(v_add(dext0[nb], r), co[nb], car[nb], dR_, dW_, dB_);
#pragma unroll
      for (int g = 0; g < Gr; ++g) sts32(dgate(nb, g) + off, v_pack(dR_[g]));
      if constexpr (Gr == 3) sts32(dgate(nb, 3) + off, v_pack(dW_[2]));
#pragma unroll
      for (int g = 0; g < Gt; ++g) dbacc[g] = v_add(dbacc[g], dB_[g]);
    }
  }
  // cotangent of the initial states, bias gradient
  __device__ __forceinline__ void store_grads(const LoopParams& p, const F2 (&rec)[NB]) {
    const size_t ND = (size_t)p.N * p.D;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      if (bt0 + row_of(nb) >= p.B) continue;
      const size_t off = (size_t)(bt0 + row_of(nb)) * ND + nd;
      if (!p.grad_cut) car[nb][0] = v_add(car[nb][0], rec[nb]);
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const float2 v = v_get(car[nb][s]);
        store_state2(p.ds0, off + (size_t)s * p.B * ND, f32, v.x, v.y);
      }
    }
#pragma unroll
    for (int g = 0; g < Gt; ++g) {
      const float2 v = v_get(dbacc[g]);
      atomicAdd(p.dbias + (size_t)g * ND + nd, v.x);
      atomicAdd(p.dbias + (size_t)g * ND + nd + 1, v.y);
    }
  }
};

template <int CELL, int U, int NT>
__global__ void __launch_bounds__(BigBwdGeom<CELL, U, NT>::TH, 1) big_bwd_kernel(const __grid_constant__ LoopParams p) {
  using G = BigBwdGeom<CELL, U, NT>;
  constexpr int MT = G::MT, NB = G::NB, W = G::W, DB = G::DB, DT = G::DT, KP = G::KP, KRP = G::KRP, TH = G::TH;
  const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
  const int gid = lane >> 2, tig = lane & 3, a = gid & 1;
  const int T = p.T, N = p.N, D = p.D, CS = p.CS;
  const int n = blockIdx.z, bt0 = blockIdx.y * G::BT;
  const uint32_t crank = cluster_ctarank();
  const int ptiles = D / 16, fsm = G::fsm(D), RB = G::recv_bytes(D);

  extern __shared__ __align__(128) unsigned char smem_raw[];
  const uint32_t sm = smem_u32(smem_raw), dtile = sm + G::OFF_D, recv = sm + G::OFF_V;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw);  // [2] bytes of partial sums have arrived
  // a wait of the cell's warps expired: the others, which wait for nothing but the CTA's barrier, must stop sending too
  volatile int* gave_up = reinterpret_cast<volatile int*>(smem_raw + 64);

  if (tid == 0) {
    *gave_up = 0;
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    fence_mbar_init();
    mbar_arrive_expect_tx(&full[0], RB);             // partial sums of step index 0 (t = T-1)
    if (T > 1) mbar_arrive_expect_tx(&full[1], RB);  // step index 1
  }
  constexpr bool TM = G::TM;
  if constexpr (TM) {  // (see tmem_alone)
    __syncwarp();
    if (warp == 0) tmem_alloc(reinterpret_cast<uint32_t*>(smem_raw + 96), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
  for (int i = tid; i < 2 * DB / 16; i += TH) sts128(dtile + i * 16, make_uint4(0u, 0u, 0u, 0u));  // (padding columns stay zero)
  __syncthreads();
  cluster_arrive();  // waited for before the first push

  // ---- this warp's tiles of p: warp, warp + W, ...  Fragments [n][CTA][tile][k-pair][lo, hi][lane]
  AFrag A[MT][KRP];
  const uint4* src = p.Rpack + rt_frag(n, CS, (int)crank, ptiles, warp < ptiles ? warp : 0, KP, 0) + lane;
  const int mtn = warp < ptiles ? (ptiles - 1 - warp) / W + 1 : 0;
  auto frag = [&](int m, int kp) {
    const uint4* q = src + (m * W * KP + kp) * 64;
    AFrag f;
    f.lo = __ldg(q); f.hi = __ldg(q + 32);
    return f;
  };
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int kp = 0; kp < KRP; ++kp)
      if (m < mtn) A[m][kp] = frag(m, kp);
  // the other k-pairs, KL per MG tiles: KT of them in tensor memory; of the others the first fsm in shared memory, the rest read from L2
  constexpr int MG = G::MG, KT = G::KT, KL = G::KL - KT, KR = KRP + KT;
  uint32_t tcol = 0;
  if constexpr (TM) {
    tcol = *reinterpret_cast<volatile uint32_t*>(smem_raw + 96) + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * G::TCOLS);
    __syncwarp();  // tensor memory is accessed by whole warps
#pragma unroll 1
    for (int i = 0; i < MT / MG * KT; ++i) {
      uint32_t r[16];
#pragma unroll
      for (int m = 0; m < MG; ++m) {
        AFrag f;
        f.lo = f.hi = make_uint4(0u, 0u, 0u, 0u);
        if (i / KT * MG + m < mtn) f = frag(i / KT * MG + m, KRP + i % KT);
        r[8 * m] = f.lo.x; r[8 * m + 1] = f.lo.y; r[8 * m + 2] = f.lo.z; r[8 * m + 3] = f.lo.w;
        r[8 * m + 4] = f.hi.x; r[8 * m + 5] = f.hi.y; r[8 * m + 6] = f.hi.z; r[8 * m + 7] = f.hi.w;
      }
      tmem_st16(tcol + i * 16, r);
    }
    tmem_wait_st();
  }
  const uint32_t rs = sm + G::off_r(D) + (uint32_t)(warp * fsm) * (MG * 1024) + lane * 16;
  for (int i = 0; i < fsm; ++i)
    for (int m = 0; m < MG; ++m)
      if (i / (KL > 0 ? KL : 1) * MG + m < mtn) {
        const AFrag f = frag(i / (KL > 0 ? KL : 1) * MG + m, KR + i % (KL > 0 ? KL : 1));
        sts128(rs + (i * MG + m) * 1024, f.lo);
        sts128(rs + (i * MG + m) * 1024 + 512, f.hi);
      }
  const uint32_t drd = dtile + (uint32_t)tig * 128u + ((uint32_t)(gid ^ (int)opnd_swz((uint32_t)tig)) << 4);
  const bool drop = p.test_drop && crank == 0;  // test hook: CTA 0 withholds its first message
  bool poisoned = false;
  auto products = [&](int j) {  // partial dh_{t-1} of the deltas of step index j, tile by tile, each to the CTA that owns its p
    const int buf = j & 1;
    const uint32_t db = drd + buf * DB;
#pragma unroll
    for (int m0 = 0; m0 < MT; m0 += MG) {
      if (m0 >= mtn) continue;
      constexpr int NS = 3 - MG;  // accumulator sets
      float part[NS][MG][NT][4];
#pragma unroll
      for (int i = 0; i < NS * MG * NT; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) part[i / (MG * NT)][i / NT % MG][i % NT][c] = 0.f;
      auto pair = [&](int kp, const AFrag& f0, const AFrag& f1) {
        uint4 b[NT];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) b[nt] = lds128(db + (uint32_t)(kp * 512 + nt * DT));
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int m = 0; m < MG; ++m)
            if (m == 0 || m0 + m < mtn) {
              const AFrag& f = m ? f1 : f0;
              const uint4 a = h ? make_uint4(f.lo.z, f.hi.z, f.lo.w, f.hi.w) : make_uint4(f.lo.x, f.hi.x, f.lo.y, f.hi.y);
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) mma_16816(part[h % NS][m][nt], a, h ? b[nt].z : b[nt].x, h ? b[nt].w : b[nt].y);
            }
      };
#pragma unroll
      for (int kp = 0; kp < KRP; ++kp) pair(kp, A[m0][kp], A[m0 + MG - 1][kp]);
      if constexpr (TM) {
        auto words = [&](int kp, const uint32_t* r) {
          AFrag f[MG];
#pragma unroll
          for (int m = 0; m < MG; ++m) {
            f[m].lo = make_uint4(r[8 * m], r[8 * m + 1], r[8 * m + 2], r[8 * m + 3]);
            f[m].hi = make_uint4(r[8 * m + 4], r[8 * m + 5], r[8 * m + 6], r[8 * m + 7]);
          }
          pair(kp, f[0], f[MG - 1]);
        };
        constexpr int TP = U == 48 ? 2 : 1;  // k-pairs per load
        __syncwarp();  // (the lanes may have left the barrier, or the branch around the sends before, one by one)
#pragma unroll
        for (int i = 0; i + TP <= KT; i += TP) {
          if constexpr (TP == 2) {
            uint32_t r[32];
            tmem_ld32(tcol + (m0 / MG * KT + i) * 16, r);
            words(KRP + i, r);
            words(KRP + i + 1, r + 16);
          } else {
            uint32_t r[16];
            tmem_ld16(tcol + (m0 / MG * KT + i) * 16, r);
            words(KRP + i, r);
          }
        }
        if constexpr (KT % TP != 0) {
          uint32_t r[16];
          tmem_ld16(tcol + (m0 / MG * KT + KT - 1) * 16, r);
          words(KRP + KT - 1, r);
        }
      }
      if constexpr (KL > 0) {
        const int first = m0 / MG * KL, stay = fsm - first < KL ? fsm - first : KL;
#pragma unroll 1
        for (int i = 0; i < stay; ++i) {
          AFrag f[MG];
#pragma unroll
          for (int m = 0; m < MG; ++m) { f[m].lo = lds128(rs + ((first + i) * MG + m) * 1024); f[m].hi = lds128(rs + ((first + i) * MG + m) * 1024 + 512); }
          pair(KR + i, f[0], f[MG - 1]);
        }
#pragma unroll 1
        for (int i = stay > 0 ? stay : 0; i < KL; ++i) {
          AFrag f[MG];
#pragma unroll
          for (int m = 0; m < MG; ++m)
            if (m0 + m < mtn) f[m] = frag(m0 + m, KR + i);
          pair(KR + i, f[0], f[MG - 1]);
        }
      }
      if (!poisoned && !(drop && j == 0)) {
#pragma unroll
        for (int m = 0; m < MG; ++m)
          if (m == 0 || m0 + m < mtn) {
            const int mt = warp + (m0 + m) * W, owner = mt * 16 / U, tl = mt - owner * (U / 16);
            const uint32_t dst = map_to_cta(recv + (uint32_t)(buf * RB + (((int)crank * (U / 16) + tl) * NT * 32 + lane) * 16), (uint32_t)owner);
            const uint32_t bar = map_to_cta(sm + buf * 8, (uint32_t)owner);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
              float v[4];
#pragma unroll
              for (int c = 0; c < 4; ++c) v[c] = NS == 2 ? part[0][m][nt][c] + part[NS - 1][m][nt][c] : part[0][m][nt][c];
              st_async_v4(dst + nt * 512, v[0], v[2], v[1], v[3], bar);
            }
          }
      }
    }
  };

  if (warp >= G::WC) {
    // barrier j of the CTA: the deltas of step j are complete, its inputs consumed, the inputs of step j + 1 have landed
    bwd_io<CELL, G, 0>(p, dtile, sm + G::OFF_I, tid - 32 * G::WC, crank, [&](auto& load, auto& store) {
      cp_async_wait<G::STAGES - 1>();
      __syncthreads();  // (in front of step 0)
      int stage = 0;
      for (int j = 0; j < T; ++j) {
        cp_async_wait<G::STAGES - 2>();
        __syncthreads();
        if (*gave_up) poisoned = true;
        if (j == 0) cluster_wait();
        products(j);
        load(T - 1 - j - G::STAGES, stage);
        store(j & 1);
        stage = stage + 1 == G::STAGES ? 0 : stage + 1;
      }
    });
  } else {
    const int ul = warp * 8 + (gid >> 1) * 2, unit = (int)crank * U + ul;
    BwdLane<CELL, G, S2> lx;
    lx.init(p, dtile, DT, sm + G::OFF_I, lane, ul, unit, n, bt0);
    // where this lane's partial sums arrive: source c at + c * (U/16) * NT * 512, batch tile nt at + nt * 512
    const uint32_t rsrc = recv + (uint32_t)((ul >> 4) * NT * 512 + (((ul & 15) >> 1) * 4 + tig) * 16 + a * 8);
    S2 rec[NB];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) rec[nb] = v_pair<S2>(0.f, 0.f);
    auto wait_partials = [&](int j, int t) {  // sums produced in step index j
      if (!mbar_wait_warp(&full[j & 1], (uint32_t)((j >> 1) & 1), poisoned)) {
        poisoned = true;
        *gave_up = 1;
        if (lane == 0) report_timeout(p.status, t);
      }
      mbar_arrive_expect_tx_if(tid == 0 && j + 2 < T && !poisoned, &full[j & 1], RB);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        S2 x = v_pair<S2>(0.f, 0.f), y = x;
        const uint32_t q = rsrc + (uint32_t)((j & 1) * RB + nb * 512);
#pragma unroll 4
        for (int c = 0; c < CS; ++c) {
          const uint2 w = lds64(q + (uint32_t)(c * (U / 16) * NT * 512));
          S2& r = (c & 1) ? y : x;
          r = v_add(r, v_pair<S2>(__uint_as_float(w.x), __uint_as_float(w.y)));
        }
        rec[nb] = v_add(x, y);
      }
    };
    __syncthreads();  // the inputs of the first step have landed
    int stage = 0;
    for (int j = 0; j < T; ++j) {  // j-th step of the reverse loop, time index t = T-1-j
      lx.load_inputs(stage);
      lx.form_coefs();
      if (j > 0) wait_partials(j - 1, T - 1 - j);
      lx.deltas(p, rec, (j & 1) * DB);
      __syncthreads();
      if (*gave_up) poisoned = true;
      if (j == 0) cluster_wait();
      products(j);
      stage = stage + 1 == G::STAGES ? 0 : stage + 1;
    }
    // (only these warps wait for the last sums; the barrier below keeps the CTA until they have arrived)
    wait_partials(T - 1, -1);
    lx.store_grads(p, rec);
  }
  __syncwarp();
  if constexpr (TM) tc_fence_before();
  cluster_arrive_relaxed();
  cluster_wait();
  if constexpr (TM) {
    tc_fence_after();
    __syncwarp();
    if (warp == 0) tmem_dealloc(*reinterpret_cast<volatile uint32_t*>(smem_raw + 96), 512);
  }
}

}  // namespace FRNN_NS
