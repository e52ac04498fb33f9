// dR for head dims 16, 32, 64 and 96: dR[g,n,d,p] = sum_{b,t} delta_g[b,t,n,d] * h_{t-1}[b,n,p].
//
// Per byte read there is little to compute here (D products per element of delta), so what counts is how memory is read.  A CTA owns a group
// of heads whose elements lie side by side (HG * D of them: 128 to 512 bytes per gate and row), all their gates, and a contiguous range
// of rows k = (b, t): every row's run goes through shared memory once, 16 bytes per cp.async along the rows, four stages deep (eight where one CTA fills an SM), and
// every warp keeps a 64 or 96 x 32 piece of the result in registers (mma.sync m16n8k16: the accumulators of a whole head, which
// the tensor-map kernel holds in tensor memory, fit here too).
// The pieces of all CTAs meet in fp32 atomics on the gradient workspace.
// Measured (before: one 64 x 64 tile of one gate per CTA, or the tensor-map kernel), us: LSTM B1024 T128 N24 D32 617 -> 175 (5.8 TB/s),
// B1024 T256 N24 D16 1213 -> 248, B1024 T512 N16 D64 1437 -> 1232 (4.4 TB/s), B100 T500 N3 D96 135 -> 65; GRU B37 T333 N5 D96 52 -> 39;
// sLSTM B256 T512 N16 D64 with fp32 states 772 -> 369.
//
// Replaces the post-loop cublasGemmStridedBatchedEx of the reference (flashrnn/flashrnn/fused/flashrnn_fused_backward.cu:
// 1049-1058; util/blas.cu:199-219).
#include "frnn_aux.cuh"

namespace FRNN_NS {

namespace {

struct DrSmallParams {
  const elem_t* dWx;   // [B,T,Gw,N,D]
  const elem_t* dg0;   // [B,T,N,D] (GRU)
  const void* states;  // [S,B,T,N,D]; only s = 0 is read
  const void* s0;      // [S,B,1,N,D]
  float* dR;           // [Gr,N,D,D] fp32
  int T, N, Gw;
  long long K;         // B*T
  long long rows_per_split;
};

template <int D, int GR, bool F32>
struct DrSmallGeom {
  static constexpr int GPU = D == 16 ? GR : (D == 32 && GR > 1 ? 2 : 1);  // gates of a warp's piece
  static constexpr int HPU = D == 16 ? 2 : 1;                            // heads of it
  static constexpr int NT = D == 16 ? 2 : 4;                             // 8-column tiles of it
  static constexpr int UPH = (GR + GPU - 1) / GPU * (D / (8 * NT));      // pieces per head (D = 16: per two heads)
  static constexpr int HG = D == 16 ? 8 : D == 32 ? 4 : D == 64 ? (GR > 1 ? 2 : 4) : (GR > 1 ? 1 : 3);
  static constexpr int W = HG * UPH / HPU, TH = 32 * W;
  static constexpr int ROW = HG * D;             // elements of a gate's run
  static constexpr int EH = F32 ? 4 : 2;
  static constexpr int PITCH = GR * ROW * 2 + ROW * EH + 16;  // an odd multiple of 16: ldmatrix reads 8 rows without conflicts
  static constexpr int CTAS = D == 96 || (D == 64 && GR > 1) ? 1 : 2;  // per SM
  static constexpr int KC = PITCH <= 800 ? 32 : 16, STAGES = CTAS == 1 ? 8 : 4;
  static constexpr int CA = GR * ROW / 8, CH = ROW * EH / 16, CPR = CA + CH, CHUNKS = KC * CPR, PT = (CHUNKS + TH - 1) / TH;
  static constexpr size_t smem = (size_t)STAGES * KC * PITCH;
};

__device__ __forceinline__ void red_add_f32x2(float* addr, float a, float b) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(addr), "f"(a), "f"(b) : "memory");
}

template <int D, int GR, bool F32>
__global__ void __launch_bounds__(DrSmallGeom<D, GR, F32>::TH, DrSmallGeom<D, GR, F32>::CTAS) recurrent_grad_small_kernel(const DrSmallParams p) {
  using G = DrSmallGeom<D, GR, F32>;
  constexpr int GPU = G::GPU, HPU = G::HPU, NT = G::NT, MTG = D / 16, KC = G::KC, STAGES = G::STAGES, PITCH = G::PITCH, ROW = G::ROW;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const uint32_t sm = smem_u32(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = p.N, n0 = blockIdx.x * G::HG, T = p.T;
  const size_t ND = (size_t)N * D;
  const long long k0 = (long long)blockIdx.y * p.rows_per_split;
  const long long k1 = k0 + p.rows_per_split < p.K ? k0 + p.rows_per_split : p.K;
  if (k0 >= k1) return;  // uniform for the CTA
  const int nchunks = (int)((k1 - k0 + KC - 1) / KC);

  // ---- this thread's 16-byte pieces of a chunk: piece i is row r, column c of [KC][CPR]; the first CA columns are delta, the others h
  const unsigned char* src[G::PT];
  uint32_t dst[G::PT];
  int tt[G::PT];  // h: time index of the row
#pragma unroll
  for (int i = 0; i < G::PT; ++i) {
    const int idx = tid + i * G::TH, r = idx / G::CPR, c = idx - r * G::CPR;
    const long long k = k0 + r;
    src[i] = nullptr;
    tt[i] = 0;
    dst[i] = sm + r * PITCH + c * 16;
    if (c < G::CA) {
      const int g = c * 8 / ROW, e = c * 8 - g * ROW;
      if (n0 * D + e < N * D)
        src[i] = reinterpret_cast<const unsigned char*>(GR == 3 && g == 0 ? p.dg0 + (size_t)k * ND + (size_t)n0 * D + e
                                                                          : p.dWx + ((size_t)k * p.Gw + (GR == 3 ? g - 1 : g)) * ND + (size_t)n0 * D + e);
    } else {
      const int e = (c - G::CA) * 16 / G::EH;
      if (n0 * D + e < N * D) src[i] = static_cast<const unsigned char*>(p.states) + ((size_t)k * ND + (size_t)n0 * D + e) * G::EH - ND * G::EH;
      tt[i] = (int)((uint32_t)k % (uint32_t)T);  // (2^32 rows do not fit the memory)
    }
    if (idx >= G::CHUNKS) src[i] = nullptr;
    if (idx < G::CHUNKS && src[i] == nullptr)  // columns beyond the last head
      for (int s = 0; s < STAGES; ++s) sts128(dst[i] + s * (KC * PITCH), make_uint4(0u, 0u, 0u, 0u));
  }
  auto load = [&](int chunk, int stage) {
    if (chunk < nchunks) {
#pragma unroll
      for (int i = 0; i < G::PT; ++i) {
        if (src[i] == nullptr) continue;
        const int idx = tid + i * G::TH, r = idx / G::CPR, c = idx - r * G::CPR;
        const long long k = k0 + (long long)chunk * KC + r;
        const uint32_t d = dst[i] + stage * (KC * PITCH);
        if (c < G::CA) {
          if (k < k1) cp_async16_u32(d, src[i]);
          else sts128(d, make_uint4(0u, 0u, 0u, 0u));
          src[i] += (size_t)KC * (GR == 3 && c * 8 < ROW ? 1 : p.Gw) * ND * 2;
        } else {
          if (k < k1) {
            const unsigned char* s = src[i];
            if (tt[i] == 0)  // h_{t-1} of t = 0 is the initial state
              s = static_cast<const unsigned char*>(p.s0) + ((size_t)((uint32_t)k / (uint32_t)T) * ND + (size_t)n0 * D) * G::EH + (size_t)(c - G::CA) * 16;
            cp_async16_u32(d, s);
          } else {
            sts128(d, make_uint4(0u, 0u, 0u, 0u));  // (delta is zero there; this only has to be finite)
          }
          src[i] += (size_t)KC * ND * G::EH;
          tt[i] += KC;
          while (tt[i] >= T) tt[i] -= T;
        }
      }
    }
    cp_async_commit();
  };

  // ---- this warp's piece: heads hl .. hl + HPU - 1 of the group, gates g0 .. g0 + GPU - 1, columns c0 ..
  const int unit = warp / G::UPH, part = warp - unit * G::UPH;
  const int hl = unit * HPU, cb = part % (D / (8 * NT)), g0 = part / (D / (8 * NT)) * GPU, c0 = cb * 8 * NT;
  float acc[HPU][GPU][MTG][NT][4];
#pragma unroll
  for (int i = 0; i < HPU * GPU * MTG * NT; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i / (GPU * MTG * NT)][i / (MTG * NT) % GPU][i / NT % MTG][i % NT][c] = 0.f;
  const int j = lane >> 3, r8 = lane & 7, gid = lane >> 2, tig = lane & 3;
  const uint32_t a_lane = (uint32_t)((j >> 1) * 8 + r8) * PITCH + (j & 1) * 16, b_lane = (uint32_t)((j & 1) * 8 + r8) * PITCH + (j >> 1) * 16;

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) load(s, s);
  int stage = 0;
  for (int c = 0; c < nchunks; ++c) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    load(c + STAGES - 1, stage == 0 ? STAGES - 1 : stage - 1);
    const uint32_t base = sm + stage * (KC * PITCH);
#pragma unroll
    for (int ks = 0; ks < KC / 16; ++ks) {
      const uint32_t kb = base + ks * 16 * PITCH;
#pragma unroll
      for (int h = 0; h < HPU; ++h) {
        uint32_t b[NT][2];
        const uint32_t hb = kb + GR * ROW * 2;
        const int e = (hl + h) * D + c0;  // element of the run
        if constexpr (F32) {
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const uint32_t at = hb + (uint32_t)(q * 8 + 2 * tig) * PITCH + (e + nt * 8 + gid) * 4;
              b[nt][q] = pack_x2(__uint_as_float(lds32(at)), __uint_as_float(lds32(at + PITCH)));
            }
        } else {
#pragma unroll
          for (int np = 0; np < NT / 2; ++np) ldmatrix_x4_trans(hb + b_lane + (e + np * 16) * 2, b[2 * np][0], b[2 * np][1], b[2 * np + 1][0], b[2 * np + 1][1]);
        }
#pragma unroll
        for (int g = 0; g < GPU; ++g)
          if (GR % GPU == 0 || g0 + g < GR) {
#pragma unroll
            for (int mt = 0; mt < MTG; ++mt) {
              uint4 a;
              ldmatrix_x4_trans(kb + a_lane + ((g0 + g) * ROW + (hl + h) * D + mt * 16) * 2, a.x, a.y, a.z, a.w);
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) mma_16816(acc[h][g][mt][nt], a, b[nt][0], b[nt][1]);
            }
          }
      }
    }
    stage = stage + 1 == STAGES ? 0 : stage + 1;
  }
  cp_async_wait<0>();
#pragma unroll
  for (int h = 0; h < HPU; ++h) {
    if (n0 + hl + h >= N) continue;
#pragma unroll
    for (int g = 0; g < GPU; ++g)
      if (GR % GPU == 0 || g0 + g < GR) {
        float* out = p.dR + (((size_t)(g0 + g) * N + n0 + hl + h) * D + gid) * D + c0 + 2 * tig;
#pragma unroll
        for (int mt = 0; mt < MTG; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int q = 0; q < 2; ++q) red_add_f32x2(out + (mt * 16 + q * 8) * D + nt * 8, acc[h][g][mt][nt][2 * q], acc[h][g][mt][nt][2 * q + 1]);
      }
  }
}

template <int D, int GR, bool F32>
cudaError_t launch(DrSmallParams p, int sm_count, cudaStream_t stream) {
  using G = DrSmallGeom<D, GR, F32>;
  const auto kern = recurrent_grad_small_kernel<D, GR, F32>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem);
  if (e != cudaSuccess) return e;
  const long long groups = (p.N + G::HG - 1) / G::HG, chunks = (p.K + G::KC - 1) / G::KC;
  long long splits = G::CTAS * (long long)sm_count / groups;  // one turn through the GPU
  if (splits > (chunks + 2) / 3) splits = (chunks + 2) / 3;            // the atomics stay a small share
  if (splits < 1) splits = 1;
  if (splits > 65535) splits = 65535;
  p.rows_per_split = (chunks + splits - 1) / splits * G::KC;
  splits = (p.K + p.rows_per_split - 1) / p.rows_per_split;
  kern<<<dim3((unsigned)groups, (unsigned)splits), G::TH, G::smem, stream>>>(p);
  return cudaGetLastError();
}
template <int D, bool F32>
cudaError_t by_gates(const DrSmallParams& p, int Gr, int sm_count, cudaStream_t stream) {
  return Gr == 4 ? launch<D, 4, F32>(p, sm_count, stream) : Gr == 3 ? launch<D, 3, F32>(p, sm_count, stream) : launch<D, 1, F32>(p, sm_count, stream);
}
template <bool F32>
cudaError_t by_dim(const DrSmallParams& p, int D, int Gr, int sm_count, cudaStream_t stream) {
  switch (D) {
    case 16: return by_gates<16, F32>(p, Gr, sm_count, stream);
    case 32: return by_gates<32, F32>(p, Gr, sm_count, stream);
    case 64: return by_gates<64, F32>(p, Gr, sm_count, stream);
    default: return by_gates<96, F32>(p, Gr, sm_count, stream);
  }
}

}  // namespace

bool recurrent_grad_small_supported(int D) { return D == 16 || D == 32 || D == 64 || D == 96; }

cudaError_t launch_recurrent_grad_small(int B, int T, int N, int D, int Gr, int Gw, int state_f32, const void* dWx, const void* dg0,
                                        const void* states, const void* s0, float* dR, int sm_count, cudaStream_t stream) {
  DrSmallParams p;
  p.dWx = static_cast<const elem_t*>(dWx);
  p.dg0 = static_cast<const elem_t*>(dg0);
  p.states = states; p.s0 = s0; p.dR = dR;
  p.T = T; p.N = N; p.Gw = Gw;
  p.K = (long long)B * T;
  p.rows_per_split = 0;
  return state_f32 ? by_dim<true>(p, D, Gr, sm_count, stream) : by_dim<false>(p, D, Gr, sm_count, stream);
}

}  // namespace FRNN_NS
