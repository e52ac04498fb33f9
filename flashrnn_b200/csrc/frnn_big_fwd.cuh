// Forward time loop for head dims above 256 (multiples of 64 up to kBigMaxD), where R does not fit the registers of a cluster:
// the lane loop of frnn_lane_fwd.cuh with
//   * up to 16 CTAs of U = 32, 48 or 64 units per head (big_tile in frnn_api.cu): with few heads and rows as many SMs as a cluster can have, so that R -- 4.7 MB at
//     head dim 768 -- lies in their registers (KRP k-pairs per warp), tensor memory (tsp pairs: a lane keeps its own words of a pair in its own lane, 16 columns,
//     and loads them back into registers for the warp's MMAs) and shared memory (the rest of it) for all T steps; only what fits none of them is
//     re-read from L2 in every step (CTAs of 64 units, three or four gates: with 8 rows head dims 960 and 1024, with 16 rows LSTM and sLSTM 768, GRU 832 and up);
//   * two warps per 8-unit group that split k; the second hands its sums to the first through shared memory (one named
//     barrier of 64 threads), which runs the cell, and moves the data meanwhile (no IO warps: a 13th warp would cost the other
//     12 a quarter of their registers).
// D = 768 LSTM, 16 CTAs x 48 units: 12 x 24 MMAs per quadrant (1152 clk), 576 shared-memory wavefronts for h and the exchange of 12 KB per CTA bound a
// step.  With the pairs that are now in tensor memory in shared memory it was 1700 wavefronts, and what did not fit came from L2.  us per 48 steps of 16 rows, that
// form and this one, forward, reverse: LSTM D = 576 78, 113 -> 74, 86; 640 136, 216 -> 105, 129; 768 107, 127 -> 94, 100; 832 180, 234 -> 136, 148; 1024 216, 246 -> 168, 163; GRU D = 640 131,
// 178 -> 105, 96; 1024 213, 205 -> 170, 117; sLSTM D = 640 142, 237 -> 112, 144; 768 119, 146 -> 96, 101; 1024 232, 273 -> 176, 192.  Two pairs per load with 48 units (94 us,
// one by one 98), one with 64 (LSTM D = 640 16 rows B200 236, in pairs 266: registers).
//
// Replaces FLASHRNNCellFusedForward (reference flashrnn/flashrnn/fused/flashrnn_fused_forward.cu:146-659).
#pragma once
#include "frnn_lane_fwd.cuh"
#include "frnn_tc.cuh"

namespace FRNN_NS {

template <int CELL, int U, int NT, bool DENSE>
struct BigFwdGeom {
  using C = Cell<CELL>;
  static constexpr int BT = 8 * NT, NT8 = NT, UNITS = U, STAGES = kBigStages;
  static constexpr bool QUAD = C::Gr > 1, CL = true;
  static constexpr int ES = 0;
  static constexpr int MT = QUAD ? 2 : 1, UW = QUAD ? 8 : 16;
  static constexpr int GROUPS = U / UW, W = 2 * GROUPS, IOT = 32 * GROUPS, TH = 32 * W;
  static constexpr int NB = QUAD ? NT : 2 * NT;
  static constexpr int GCM = CacheGeom<C::GC>::MAIN;
  static constexpr bool GCX = CacheGeom<C::GC>::EXTRA;
  // k-pairs of R per warp in registers: what the register file leaves beside the ~60 of everything else, and the words on their way from tensor memory (U = 32: all
  // there are).  DENSE (Elman, 64
  // units): half of it, so that two CTAs fit an SM, 226 -> 128 registers (see big_tile in frnn_api.cu)
  static_assert(!DENSE || (!QUAD && U == 64), "the dense form is Elman's of 64 units");
  static constexpr int KRP = QUAD ? (U == 32 ? 8 : U == 48 ? 4 : NT == 2 ? 1 : 2) : (U == 32 || DENSE ? 8 : U == 48 ? 12 : 16);
  // ... and in tensor memory, of which a warp has TCOLS columns of 32 lanes: a lane's 16 words of a k-pair lie in 16 columns of its own lane
  static constexpr bool TM = QUAD && U > 32;
  static constexpr int TCOLS = TM ? 512 / (W / 4) / 16 * 16 : 0, TMAX = TCOLS / 16, TPAIRS = U == 48 ? 2 : 1;  // TPAIRS: k-pairs per load
  static __host__ __device__ constexpr int tsp(int D) { return D / 64 - KRP < 0 ? 0 : (D / 64 - KRP < TMAX ? D / 64 - KRP : TMAX); }
  // Buffers for the k-pairs that fit neither registers nor shared memory: reloaded from L2 as soon as they are used, so two pairs per warp
  // are in flight all the time, the wait for h included (one at a time, loaded where it was used: D = 1024 LSTM step 10310 clk).  Not with 16 rows, where their registers spill (B200 T32 D = 1024 451 -> 378 us)
  static constexpr int PB = QUAD && U == 64 && NT == 1 ? 2 : 0;
  static constexpr int XSH = C::Gw == 3 ? 1 : 0, XPL = C::Gw + XSH;
  static constexpr int XP = io_pitch(U * 2), XS = XPL * BT * XP;
  static constexpr int SP = io_pitch(U * 4), CP = io_pitch(U * 2 * GCM), EP = io_pitch(U * 2);
  static constexpr int OUT_C = C::S * BT * SP, OUT_E = OUT_C + (GCM ? BT * CP : 0), OUT_B = OUT_E + (GCX ? BT * EP : 0);
  // shared memory: barriers | Wx ring | results | sums of the second warps | 2 h tiles | fragments of R
  static constexpr int OFF_X = 128, OFF_O = OFF_X + kBigStages * XS, OFF_S = OFF_O + 2 * OUT_B, OFF_H = (OFF_S + GROUPS * MT * NT * 512 + 127) / 128 * 128;
  static __host__ __device__ constexpr int off_r(int D) { return OFF_H + 2 * NT * opnd_bytes(D); }
  // k-pairs of R per warp in shared memory
  static __host__ __device__ constexpr int ksp(int D) {
    const int want = D / 64 - KRP - tsp(D), fit = ((int)kSmemBudget - off_r(D)) / (W * MT * 1024);
    return want <= 0 ? 0 : (fit < 0 ? 0 : (want < fit ? want : fit));
  }
  static __host__ __device__ constexpr size_t smem(int D) { return tmem_alone(TM, (size_t)off_r(D) + (size_t)ksp(D) * W * MT * 1024); }
};

// Index (16-byte fragments) of lane 0's first fragment of unit group `grp`, k-pair kp in the packed R of head n: [n][grp][kp][m][lo, hi][lane]
template <int MT>
__device__ __forceinline__ size_t big_frag(int n, int groups, int grp, int kpairs, int kp) { return (((size_t)n * groups + grp) * kpairs + kp) * (MT * 64); }

// R[Gr,N,D,D] -> fragments; one thread per (fragment pair lo / hi, lane)
template <int CELL>
__global__ void big_pack_kernel(const elem_t* __restrict__ R, uint4* __restrict__ out, int N, int D) {
  using C = Cell<CELL>;
  constexpr bool QUAD = C::Gr > 1;
  constexpr int MT = QUAD ? 2 : 1, UW = QUAD ? 8 : 16;
  const int groups = D / UW, kpairs = D / 32;
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)N * groups * kpairs * MT * 64) return;
  const int lane = (int)(idx & 31), hi = (int)((idx >> 5) & 1), gid = lane >> 2, tig = lane & 3;
  size_t r = idx >> 6;
  const int m = (int)(r % MT); r /= MT;
  const int kp = (int)(r % kpairs); r /= kpairs;
  const int grp = (int)(r % groups), n = (int)(r / groups);
  const int g = QUAD ? hi * 2 + (gid & 1) : 0, unit = grp * UW + (QUAD ? (gid >> 1) * 2 + m : 2 * gid + hi);
  out[idx] = g < C::Gr ? __ldg(reinterpret_cast<const uint4*>(R + (((size_t)g * N + n) * D + unit) * D + kp * 32 + tig * 8)) : make_uint4(0u, 0u, 0u, 0u);
}

template <int CELL, int U, int NT, bool DENSE>
__global__ void __launch_bounds__(BigFwdGeom<CELL, U, NT, DENSE>::TH, DENSE ? 2 : 1) big_fwd_kernel(const __grid_constant__ LoopParams p) {
  using G = BigFwdGeom<CELL, U, NT, DENSE>;
  constexpr int MT = G::MT, TH = G::TH, KRP = G::KRP, NS = G::QUAD ? 1 : 2;
  constexpr bool QUAD = G::QUAD;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const int T = p.T, N = p.N, B = p.B, D = p.D, CS = p.CS;
  const int n = blockIdx.z, bt0 = blockIdx.y * G::BT;
  const uint32_t crank = cluster_ctarank();
  const int f32 = p.state_f32;
  const size_t ND = (size_t)N * D;
  const int HT = opnd_bytes(D), HB = NT * HT, kph = D / 64, ksp = G::ksp(D);
  const uint32_t step_bytes = (uint32_t)(D * G::BT * 2);

  extern __shared__ __align__(128) unsigned char smem_raw[];
  const uint32_t sm = smem_u32(smem_raw), hbuf = sm + G::OFF_H;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw);  // [2] bytes of h tile x have arrived (and see lane_fwd_io)

  grid_launch_next();
  if (tid == 0) {
    for (int x = 0; x < 2; ++x) mbar_init(&full[x], 1 + G::GROUPS);
    fence_mbar_init();
    if (T > 1) mbar_arrive_expect_tx(&full[0], step_bytes);  // h_0, consumed at step 1
    if (T > 2) mbar_arrive_expect_tx(&full[1], step_bytes);  // h_1
  }
  constexpr bool TM = G::TM;
  if constexpr (TM) {  // (see tmem_alone)
    __syncwarp();
    if (warp == 0) tmem_alloc(reinterpret_cast<uint32_t*>(smem_raw + 64), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
  if (p.clear_status && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
    p.status[0] = 0u; p.status[1] = 0u; p.status[2] = 0u; p.status[3] = 0u;
  }
  // ---- warp (grp, half): units [grp * UW, +UW), k-pairs [half * kph, +kph).  Its fragments: KRP pairs in registers, the next tsp in tensor memory,
  // the next ksp in shared memory (each lane reads back what it wrote itself), the rest in global memory
  const int half = warp >= G::GROUPS, grp = warp - half * G::GROUPS;
  const uint4* src = p.Rpack + big_frag<MT>(n, D / G::UW, (int)crank * G::GROUPS + grp, D / 32, half * kph) + lane;
  AFrag A[MT][KRP];
#pragma unroll
  for (int kp = 0; kp < KRP; ++kp)
#pragma unroll
    for (int m = 0; m < MT; ++m)
      if (kp < kph) {
        A[m][kp].lo = __ldg(src + (size_t)kp * (MT * 64) + m * 64);
        A[m][kp].hi = __ldg(src + (size_t)kp * (MT * 64) + m * 64 + 32);
      }
  const int tsp = G::tsp(D), kst = KRP + tsp;  // kst: first pair in shared memory
  uint32_t tcol = 0;
  if constexpr (TM) {
    static_assert(MT == 2, "a k-pair is 16 words per lane");
    tcol = *reinterpret_cast<volatile uint32_t*>(smem_raw + 64) + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * G::TCOLS);
    __syncwarp();  // tensor memory is accessed by whole warps
    for (int i = 0; i < tsp; ++i) {
      uint32_t r[16];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint4 v = __ldg(src + (size_t)(KRP + i) * (MT * 64) + q * 32);
        r[4 * q] = v.x; r[4 * q + 1] = v.y; r[4 * q + 2] = v.z; r[4 * q + 3] = v.w;
      }
      tmem_st16(tcol + i * 16, r);
    }
    tmem_wait_st();
  }
  constexpr int PB = G::PB, PBN = PB > 0 ? PB : 1;
  const int rem = kph - kst - ksp;  // pairs in global memory
  const uint4* rsrc = src + (size_t)(kst + ksp) * (MT * 64);
  AFrag P[PBN][MT];
  auto fetch = [&](int s, int j) {  // pair j of those -> buffer s
#pragma unroll
    for (int m = 0; m < MT; ++m) { P[s][m].lo = __ldg(rsrc + (size_t)j * (MT * 64) + m * 64); P[s][m].hi = __ldg(rsrc + (size_t)j * (MT * 64) + m * 64 + 32); }
  };
  if constexpr (PB > 0) {
#pragma unroll
    for (int s = 0; s < PB; ++s)
      if (s < rem) fetch(s, s);
  }
  const uint32_t rs = sm + G::off_r(D) + (uint32_t)(warp * ksp) * (MT * 1024) + lane * 16;
  for (int i = 0; i < ksp * MT * 2; ++i) sts128(rs + i * 512, __ldg(src + (size_t)kst * (MT * 64) + i * 32));

  grid_wait_previous();  // (R may be read before it: consecutive decoding steps overlap up to here)
  for (int idx = tid; idx < G::BT * (D / 2); idx += TH) {  // h_{-1} -> tile 1
    const int bl = idx / (D / 2), k = 2 * (idx - bl * (D / 2));
    float2 v = make_float2(0.f, 0.f);
    if (bt0 + bl < B) v = load_state2(p.s0, (size_t)(bt0 + bl) * ND + (size_t)n * D + k, f32);
    sts32(hbuf + HB + (bl >> 3) * HT + opnd_off(bl & 7, k), pack_x2(v.x, v.y));
  }
  __syncthreads();
  cluster_arrive();  // barriers initialised, h_{-1} read; waited for before the first push, or before `last` may overwrite s0

  const int ul = grp * G::UW + (QUAD ? (gid >> 1) * MT : 2 * gid), unit = (int)crank * U + ul;
  const uint32_t sums = sm + G::OFF_S + (uint32_t)(grp * MT * NT * 32 + lane) * 16;
  const uint32_t hrd = hbuf + (uint32_t)(half * kph) * 512u + (uint32_t)tig * 128u + ((uint32_t)(gid ^ (int)opnd_swz((uint32_t)tig)) << 4);
  bool poisoned = false;
  auto wait_h = [&](int t) {  // h_{t-1}
    if (t > 0 && !poisoned) {
      if (!mbar_wait_bounded(&full[(t + 1) & 1], (uint32_t)(((t - 1) >> 1) & 1))) {
        poisoned = true;
        report_timeout(p.status, t);
      }
      else if (tid == 0 && t + 2 < T) mbar_arrive_expect_tx(&full[(t + 1) & 1], step_bytes);
    }
    if constexpr (TM) __syncwarp();  // (the lanes may have left the wait one by one)
  };
  float part[NS][MT][NT][4];
  auto products = [&](uint32_t hb) {  // part += this warp's rows and k range of R times the h tile
    auto pair = [&](int kp, const AFrag (&a)[MT]) {
      uint4 b[NT];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) b[nt] = lds128(hb + (uint32_t)kp * 512u + nt * HT);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
          mma_16816(part[0][m][nt], make_uint4(a[m].lo.x, a[m].hi.x, a[m].lo.y, a[m].hi.y), b[nt].x, b[nt].y);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
          mma_16816(part[NS - 1][m][nt], make_uint4(a[m].lo.z, a[m].hi.z, a[m].lo.w, a[m].hi.w), b[nt].z, b[nt].w);
    };
    auto buffered = [&](int j) {  // pairs j .. j + PB - 1 of those in global memory; each buffer moves on, behind the last pair to the next step's first
      if constexpr (PB > 0) {
#pragma unroll
        for (int s = 0; s < PB; ++s)
          if (j + s < rem) {
            pair(kst + ksp + j + s, P[s]);
            if (rem > PB) fetch(s, j + s + PB < rem ? j + s + PB : s);
          }
      }
    };
    buffered(0);
#pragma unroll
    for (int kp = 0; kp < KRP; ++kp)
      if (kp < kph) {
        AFrag a[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) a[m] = A[m][kp];
        pair(kp, a);
      }
    if constexpr (TM) {
      auto words = [&](int kp, const uint32_t* r) {
        AFrag a[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          a[m].lo = make_uint4(r[8 * m], r[8 * m + 1], r[8 * m + 2], r[8 * m + 3]);
          a[m].hi = make_uint4(r[8 * m + 4], r[8 * m + 5], r[8 * m + 6], r[8 * m + 7]);
        }
        pair(kp, a);
      };
      int i = 0;
      if constexpr (G::TPAIRS == 2) {
#pragma unroll 1
        for (; i + 1 < tsp; i += 2) {
          uint32_t r[32];
          tmem_ld32(tcol + i * 16, r);
          words(KRP + i, r);
          words(KRP + i + 1, r + 16);
        }
      }
#pragma unroll 1
      for (; i < tsp; ++i) {
        uint32_t r[16];
        tmem_ld16(tcol + i * 16, r);
        words(KRP + i, r);
      }
    }
#pragma unroll 1
    for (int i = 0; i < ksp; ++i) {
      AFrag a[MT];
#pragma unroll
      for (int m = 0; m < MT; ++m) { a[m].lo = lds128(rs + (i * MT + m) * 1024); a[m].hi = lds128(rs + (i * MT + m) * 1024 + 512); }
      pair(kst + i, a);
    }
    if constexpr (PB > 0) {
#pragma unroll 1
      for (int j = PB; j < rem; j += PB) buffered(j);
    } else {
#pragma unroll 1
      for (int kp = kst + ksp; kp < kph; ++kp) {
        AFrag a[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) { a[m].lo = __ldg(src + (size_t)kp * (MT * 64) + m * 64); a[m].hi = __ldg(src + (size_t)kp * (MT * 64) + m * 64 + 32); }
        pair(kp, a);
      }
    }
  };

  if (half) {
    // ---- second warp of a group: its sums to the first, then the data: results of the step before (named barriers 1, 2: those of an
    // even, odd step are staged and Wx of the step behind it has been read) to global memory, Wx of step t + kBigStages - 1 from it
    fwd_io<CELL, G, 0>(p, sm + G::OFF_X, sm + G::OFF_O, tid - G::IOT, crank, [&](auto& load, auto& store) {
      cp_async_wait<kBigStages - 2>();
      __syncthreads();  // (Wx of steps 0 and 1)
      bool dead = false;
      int stage = 0;
      for (int t = 0; t < T; ++t) {
        wait_h(t);
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
          for (int i = 0; i < MT * NT; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) part[s][i / NT][i % NT][c] = 0.f;
        products(hrd + ((t + 1) & 1) * HB);
#pragma unroll
        for (int i = 0; i < MT * NT; ++i) {  // (the buffer is free: the first warp has read it before it sent what this warp waited for)
          float c[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) c[q] = NS == 2 ? part[0][i / NT][i % NT][q] + part[NS - 1][i / NT][i % NT][q] : part[0][i / NT][i % NT][q];
          sts128(sums + i * 512, make_uint4(__float_as_uint(c[0]), __float_as_uint(c[1]), __float_as_uint(c[2]), __float_as_uint(c[3])));
        }
        bar_arrive<64>(3 + grp);
        if (t == 0) cluster_wait();
        else {
          bar_sync<TH>(1 + ((t - 1) & 1));
          load(t - 1 + kBigStages, stage);
          store((t - 1) & 1);
          stage = stage + 1 == kBigStages ? 0 : stage + 1;
        }
        if (t + 1 < T) {
          cp_async_wait<kBigStages - 3>();  // Wx of step t + 2
          __syncwarp();
          if (lane == 0) io_arrive(full, t, dead);
        }
      }
      bar_sync<TH>(1 + ((T - 1) & 1));
      store((T - 1) & 1);
    });
  } else {
    FwdLane<CELL, G, S2> lx;
    lx.init(p, sm + G::OFF_X, sm + G::OFF_O, HT, lane, ul, unit, n, bt0);
    if constexpr (!QUAD) lx.init_send(HT, unit);
    const int drop_t = (p.test_drop && crank == 0) ? 1 : -1;  // test hook: CTA 0 withholds its message of step 1
    const bool cache = p.cache != nullptr;
    __syncthreads();  // Wx of steps 0 and 1 has landed
    lx.start_sums(0, part[0]);
    int stage = 0;
    for (int t = 0; t < T; ++t) {
      const int nxt = t & 1;
      wait_h(t);
#pragma unroll
      for (int s = 1; s < NS; ++s)
#pragma unroll
        for (int i = 0; i < MT * NT; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) part[s][i / NT][i % NT][c] = 0.f;
      products(hrd + ((t + 1) & 1) * HB);
      float acc[MT][NT][4];
      bar_sync<64>(3 + grp);
#pragma unroll
      for (int i = 0; i < MT * NT; ++i) {
        const uint4 v = lds128(sums + i * 512);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
          acc[i / NT][i % NT][q] = (NS == 2 ? part[0][i / NT][i % NT][q] + part[NS - 1][i / NT][i % NT][q] : part[0][i / NT][i % NT][q]) + __uint_as_float(w[q]);
      }
      lx.cell(acc, p.fclip);
      if (t == 0) cluster_wait();
      lx.swap();
      if (t + 1 < T && t != drop_t && !poisoned) {
#pragma unroll 4
        for (int c = 0; c < CS; ++c) {
          const uint32_t r = crank + 1 + c, peer = map_to_cta(sm, r >= (uint32_t)CS ? r - CS : r);
          lx.send(peer + G::OFF_H + nxt * HB, peer + nxt * 8);
        }
      }
      lx.stage(nxt, cache);
      stage = stage + 1 == kBigStages ? 0 : stage + 1;
      lx.start_sums(stage, part[0]);  // (at the last step: of a stage that nobody reads)
      bar_arrive<TH>(1 + nxt);
    }
    if (p.last != nullptr) lx.store_last(p);
  }
  // Every message to this CTA has been waited for; only after an expired wait can one still be in flight, and then the barrier covers it.
  if (T > 1) { __syncwarp(); cluster_arrive_relaxed(); cluster_wait(); }
  if constexpr (TM) {
    tc_fence_before();
    __syncthreads();  // (every warp has done its last load; one that reached the cluster's barrier above has, too, but T may be 1)
    tc_fence_after();
    __syncwarp();
    if (warp == 0) tmem_dealloc(*reinterpret_cast<volatile uint32_t*>(smem_raw + 64), 512);
  }
}

}  // namespace FRNN_NS
