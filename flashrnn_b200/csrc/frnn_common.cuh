// Shared device helpers of the sm_100a time-loop kernels: PTX wrappers (warp MMA, ldmatrix, cp.async,
// cluster barrier / distributed shared memory), fp32 gate math and the per-cell traits.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "frnn_elem.cuh"

namespace FRNN_NS {

// 0..3 are the public cell ids of the C ABI.  CELL_ELMAN_CLIP is internal: Elman with forward_clip, whose backward
// needs the tanh output from before the clamp and therefore caches it (plain Elman re-reads h and caches nothing).
enum { CELL_LSTM = 0, CELL_GRU = 1, CELL_ELMAN = 2, CELL_SLSTM = 3, CELL_ELMAN_CLIP = 4 };

// Gate / state counts per cell (reference registry flashrnn/flashrnn/flashrnn.py:49-71) plus what this
// implementation caches for the backward pass and which states the backward has to re-read.
//   GC    cached values per (b,t,n,d)
//   NNEED states whose value at t-1 / t the closed-form backward needs (indices given by need(i))
//   NEXT  leading states whose external cotangent enters the backward (h, c, n; never m)
template <int CELL> struct Cell;
template <> struct Cell<CELL_LSTM> {
  static constexpr int Gr = 4, Gw = 4, Gt = 4, S = 2, GC = 4, NNEED = 1, NEXT = 2;
  __host__ __device__ static constexpr int need(int) { return 1; }
};
template <> struct Cell<CELL_GRU> {
  static constexpr int Gr = 3, Gw = 3, Gt = 4, S = 1, GC = 4, NNEED = 1, NEXT = 1;
  __host__ __device__ static constexpr int need(int) { return 0; }
};
template <> struct Cell<CELL_ELMAN> {
  static constexpr int Gr = 1, Gw = 1, Gt = 1, S = 1, GC = 0, NNEED = 1, NEXT = 1;
  __host__ __device__ static constexpr int need(int) { return 0; }
};
template <> struct Cell<CELL_ELMAN_CLIP> {
  static constexpr int Gr = 1, Gw = 1, Gt = 1, S = 1, GC = 1, NNEED = 1, NEXT = 1;
  __host__ __device__ static constexpr int need(int) { return 0; }
};
template <> struct Cell<CELL_SLSTM> {
  static constexpr int Gr = 4, Gw = 4, Gt = 4, S = 4, GC = 5, NNEED = 2, NEXT = 3;
  __host__ __device__ static constexpr int need(int i) { return i == 0 ? 1 : 2; }
};

// CELL | kNoopCell selects the measurement variant of a cell: same gate / state counts, same data movement, exchange and
// barriers, but the gate arithmetic is replaced by a pass-through.  Its step time is the floor the serial chain of the
// time loops sets without any cell math (results are meaningless).  Instantiated for the benchmark tiles only.
constexpr int kNoopCell = 8;
template <> struct Cell<CELL_LSTM | kNoopCell> : Cell<CELL_LSTM> {};
template <> struct Cell<CELL_GRU | kNoopCell> : Cell<CELL_GRU> {};
template <> struct Cell<CELL_SLSTM | kNoopCell> : Cell<CELL_SLSTM> {};

// Arguments of both time-loop kernels (forward uses the first block, backward all of it).
struct LoopParams {
  const elem_t* Wx;   // [B,T,Gw,N,D]
  const elem_t* R;           // [Gr,N,D,D] (lane loops, forward)
  const uint4* Rpack;        // recurrent matrix repacked into warp-MMA A fragments
  const elem_t* bias; // [Gt,N,D]
  const void* s0;            // [S,B,1,N,D]
  void* states;              // [S,B,T,N,D]  (forward: out, backward: in)
  elem_t* cache;      // activations, see CacheGeom in frnn_lane.cuh (forward: out or null, backward: in)
  const void* dstates;       // [S,B,T,N,D]
  elem_t* dWx;        // [B,T,Gw,N,D]
  elem_t* dg0;        // [B,T,N,D]   GRU only: delta of the recurrent-only gate
  void* ds0;                 // [S,B,1,N,D]
  float* dbias;              // fp32 [Gt,N,D] accumulated with atomics
  union {
    void* last;              // [S,B,1,N,D] forward: the states after the last step, or null
    float* dR;               // backward: fp32 [Gr,N,D,D] accumulated with atomics (reverse lane loops that form dR themselves)
  };
  unsigned* status;
  int clear_status;          // forward: CTA 0 zeroes the status block first
  int B, T, N, D;
  int test_drop;             // test hook: CTA 0 of each cluster withholds one exchange message (see frnn_plan)
  int CS;                    // CTAs per cluster
  int state_f32;             // states / dstates / s0 / ds0 are fp32 (else bf16)
  float fclip, gclip;        // <= 0: off
  int grad_cut;              // backward: ignore the matrix part of the recurrent cotangent (truncated BPTT)
  // element strides of the caller-produced tensors (D contiguous): Wx[b][t][g][n][.], dstates[s][b][t][n][.]
  long long wx_sb, wx_st, wx_sg, wx_sn;
  long long ds_ss, ds_sb, ds_st, ds_sn;
};
// Launches with 232 bytes of arguments take the host 0.2 us longer than with 224: a decoding step of GRU B1 N12 D64, where host and GPU take about the same, 2.84 us against 2.68
// (five processes each, in turn: 2.83 to 2.93 and 2.66 to 2.69).
static_assert(sizeof(LoopParams) <= 224, "launch cost");

// ------------------------------------------------------------------------------------------------ PTX
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}
// D(16x8, fp32) += A(16x16, elem_t, row) * B(16x8, elem_t, col)
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32." FRNN_MMA_TYPE "." FRNN_MMA_TYPE ".f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// the same with C = 0
__device__ __forceinline__ void mma_16816_zero(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32." FRNN_MMA_TYPE "." FRNN_MMA_TYPE ".f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void cp_async16_u32(uint32_t smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t addr, uint2 v) {
  asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// stores into another CTA's shared memory (shared::cluster addresses) that count their bytes on that CTA's mbarrier
__device__ __forceinline__ void st_async_b32(uint32_t dst, uint32_t v, uint32_t mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(v), "r"(mbar) : "memory");
}
__device__ __forceinline__ void st_async_v2(uint32_t dst, uint2 v, uint32_t mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ void st_async_v4(uint32_t dst, float a, float b, float c, float d, uint32_t mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst), "f"(a), "f"(b),
               "f"(c), "f"(d), "r"(mbar) : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// shared::cluster address of `local_addr` (a shared::cta address of this CTA) inside CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}

// threadIdx.x / 32, known to the compiler to be the same in all lanes of a warp
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// ---- programmatic dependent launch (decoding steps, launched with the attribute): the next launch may start now / every launch in front of
// this one has completed and its writes are visible
__device__ __forceinline__ void grid_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- mbarrier + bulk async copy between the shared memories of a cluster
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// named CTA barriers: `bar_arrive` does not wait.  `threads` counts those of both sides.
template <int THREADS> __device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(THREADS) : "memory"); }
template <int THREADS> __device__ __forceinline__ void bar_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(THREADS) : "memory"); }
__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits for a phase of `bar`, but never longer than ~1 s: on expiry the caller records the failure in
// the status block and stops waiting for the rest of the kernel (results are then invalid, the kernel ends).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (global_timer_ns() - t0 > 1000000000ull) return false;
  }
}
// The same for a converged warp of which every lane waits.  The branch depends on a vote, which the compiler knows to be the same in all lanes: a
// phase that is complete costs 50 clk, with a branch on each lane's own result (mbar_wait_bounded) 125 -- in the time loops that is behind the
// last arrival, in every step.  `skip`: an earlier wait of this warp expired, do not wait.  The result is the same in all lanes.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, bool skip = false) {
  auto done = [&]() {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %3, 0;\n\tsetp.eq.u32 p, 0, 0;\n\t"
        "@!q mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"((uint32_t)skip) : "memory");
    return __all_sync(0xffffffffu, ok != 0) != 0;
  };
  if (done()) return true;
  const uint64_t t0 = global_timer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
      if (done()) return true;
    if (__any_sync(0xffffffffu, global_timer_ns() - t0 > 1000000000ull)) return false;
  }
}
// mbar_arrive_expect_tx where `on`, without a branch
__device__ __forceinline__ void mbar_arrive_expect_tx_if(bool on, uint64_t* bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}"
               ::"r"(smem_u32(bar)), "r"(bytes), "r"((uint32_t)on) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// copies `bytes` (multiple of 16) from this CTA's shared memory to the same offset space of another CTA of the
// cluster; completion is signalled as transaction bytes on the destination CTA's mbarrier
__device__ __forceinline__ void bulk_copy_to_cta(uint32_t dst_cluster_addr, uint32_t src_cta_addr, uint32_t bytes,
                                                 uint32_t mbar_cluster_addr) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst_cluster_addr), "r"(src_cta_addr), "r"(bytes), "r"(mbar_cluster_addr) : "memory");
}
// true in exactly one lane of a fully converged warp
__device__ __forceinline__ bool elect_one_sync() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(pred)::"memory");
  return pred != 0;
}
// Warp-collective: one elected lane of the calling (converged) warp starts the bulk copies of this CTA's slice
// [src_cta_addr, +bytes) to the same address in every other CTA of the cluster; each copy completes on the
// destination CTA's mbarrier at `bar_cta_addr`.
// Called by EVERY warp of the CTA (`warp`, `nwarps`): warp w serves the peers w, w + nwarps, ... so that the
// copies are issued in parallel.
__device__ __forceinline__ void push_slice_to_peers(uint32_t src_cta_addr, uint32_t bytes, uint32_t bar_cta_addr,
                                                    uint32_t my_rank, uint32_t cluster_size, uint32_t warp,
                                                    uint32_t nwarps) {
  __syncwarp();
#pragma unroll 1
  for (uint32_t c = warp; c < cluster_size; c += nwarps) {
    if (c == my_rank) continue;
    const uint32_t dst = map_to_cta(src_cta_addr, c), bar = map_to_cta(bar_cta_addr, c);
    if (elect_one_sync()) bulk_copy_to_cta(dst, src_cta_addr, bytes, bar);
  }
}
__device__ __forceinline__ void report_timeout(unsigned* status, int where) {
  if (atomicCAS(status, 0u, 1u) == 0u) {
    status[1] = (unsigned)where;
    status[2] = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  }
}

// four consecutive fp32 values added to global memory in one reduction (16-byte aligned address)
__device__ __forceinline__ void red_add_f32x4(float* addr, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// ------------------------------------------------------------------------------------------------ math
// Gate nonlinearities.  Default: the hardware tanh (one MUFU op, max error ~5e-4, an order of magnitude
// below the bf16 rounding of the stored results); sigmoid(x) = 0.5 * tanh(0.5 x) + 0.5.
// -DFRNN_EXACT_ACT switches to exp-based forms accurate to ~1e-6.
__device__ __forceinline__ float fast_tanh(float x) {
#ifndef FRNN_EXACT_ACT
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return __fdividef(2.f, 1.f + __expf(-2.f * x)) - 1.f;
#endif
}
__device__ __forceinline__ float fast_sigmoid(float x) {
#ifndef FRNN_EXACT_ACT
  return fmaf(0.5f, fast_tanh(0.5f * x), 0.5f);
#else
  return __fdividef(1.f, 1.f + __expf(-x));
#endif
}
__device__ __forceinline__ float log_sigmoid(float x) { return fminf(x, 0.f) - __logf(1.f + __expf(-fabsf(x))); }
__device__ __forceinline__ float clampf(float x, float v) { return fminf(fmaxf(x, -v), v); }

__device__ __forceinline__ uint32_t pack_x2(float lo, float hi) {
  elem2_t v = floats_to_elem2(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_x2(uint32_t w) {
  elem2_t v = *reinterpret_cast<elem2_t*>(&w);
  return elem2_to_floats(v);
}

// Two fp32 values, for the loops whose lanes own two units: S2 with scalar instructions, P2 in a register pair with the packed ones
// (two multiplications or additions per issue slot, each rounded as the scalar ones are; but values that are not produced in
// pairs have to be moved together, so which is faster depends on the loop).  The v_* functions exist for float, S2 and P2: the
// cells are written once.
struct S2 { float x, y; };
struct P2 { unsigned long long v; };
template <class V> __device__ __forceinline__ V v_pair(float lo, float hi) {
  V r;
  if constexpr (sizeof(r) == sizeof(S2) && alignof(V) == alignof(S2)) { r.x = lo; r.y = hi; }
  else asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 v_get(S2 a) { return make_float2(a.x, a.y); }
__device__ __forceinline__ float2 v_get(P2 a) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v)); return r; }
__device__ __forceinline__ P2 v_fma(P2 a, P2 b, P2 c) { P2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v)); return r; }
__device__ __forceinline__ P2 v_mul(P2 a, P2 b) { P2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ P2 v_add(P2 a, P2 b) { P2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ S2 v_fma(S2 a, S2 b, S2 c) { return S2{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
__device__ __forceinline__ S2 v_mul(S2 a, S2 b) { return S2{a.x * b.x, a.y * b.y}; }
__device__ __forceinline__ S2 v_add(S2 a, S2 b) { return S2{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ float v_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float v_mul(float a, float b) { return a * b; }
__device__ __forceinline__ float v_add(float a, float b) { return a + b; }
template <class V> __device__ __forceinline__ V v_const(float c) {
  if constexpr (sizeof(V) == 8) return v_pair<V>(c, c);
  else return c;
}
template <class F> __device__ __forceinline__ float v_map(float a, F f) { return f(a); }
template <class F> __device__ __forceinline__ float v_map(float a, float b, F f) { return f(a, b); }
template <class F> __device__ __forceinline__ float v_map(float a, float b, float c, F f) { return f(a, b, c); }
template <class V, class F> __device__ __forceinline__ V v_map(V a, F f) { const float2 x = v_get(a); return v_pair<V>(f(x.x), f(x.y)); }
template <class V, class F> __device__ __forceinline__ V v_map(V a, V b, F f) {
  const float2 x = v_get(a), y = v_get(b);
  return v_pair<V>(f(x.x, y.x), f(x.y, y.y));
}
template <class V, class F> __device__ __forceinline__ V v_map(V a, V b, V c, F f) {
  const float2 x = v_get(a), y = v_get(b), z = v_get(c);
  return v_pair<V>(f(x.x, y.x, z.x), f(x.y, y.y, z.y));
}
// the value is computed in front of what follows in the program, not behind it
__device__ __forceinline__ void v_pin(float& a) { asm volatile("" : "+f"(a)); }
__device__ __forceinline__ void v_pin(S2& a) { asm volatile("" : "+f"(a.x), "+f"(a.y)); }
__device__ __forceinline__ void v_pin(P2& a) { asm volatile("" : "+l"(a.v)); }
template <class V> __device__ __forceinline__ V v_neg(V a) { return v_mul(a, v_const<V>(-1.f)); }
template <class V> __device__ __forceinline__ V v_sub(V a, V b) { return v_fma(b, v_const<V>(-1.f), a); }
template <class V> __device__ __forceinline__ V v_one_minus(V a) { return v_fma(a, v_const<V>(-1.f), v_const<V>(1.f)); }
template <class V> __device__ __forceinline__ V v_tanh(V a) { return v_map(a, [](float x) { return fast_tanh(x); }); }
template <class V> __device__ __forceinline__ V v_sigmoid(V a) {
#ifndef FRNN_EXACT_ACT
  return v_fma(v_tanh(v_mul(a, v_const<V>(0.5f))), v_const<V>(0.5f), v_const<V>(0.5f));
#else
  return v_map(a, [](float x) { return fast_sigmoid(x); });
#endif
}
template <class V> __device__ __forceinline__ V v_clamp(V a, float lim) { return v_map(a, [lim](float x) { return clampf(x, lim); }); }
template <class V> __device__ __forceinline__ uint32_t v_pack(V a) { const float2 x = v_get(a); return pack_x2(x.x, x.y); }
template <class V> __device__ __forceinline__ V v_unpack(uint32_t w) { const float2 x = unpack_x2(w); return v_pair<V>(x.x, x.y); }

// Loads / stores of a pair of adjacent state values in the run-time state dtype.
__device__ __forceinline__ float2 load_state2(const void* base, size_t elem_off, int f32) {
  if (f32) return *reinterpret_cast<const float2*>(static_cast<const float*>(base) + elem_off);
  return unpack_x2(*reinterpret_cast<const uint32_t*>(static_cast<const elem_t*>(base) + elem_off));
}
__device__ __forceinline__ void store_state2(void* base, size_t elem_off, int f32, float lo, float hi) {
  if (f32) *reinterpret_cast<float2*>(static_cast<float*>(base) + elem_off) = make_float2(lo, hi);
  else *reinterpret_cast<uint32_t*>(static_cast<elem_t*>(base) + elem_off) = pack_x2(lo, hi);
}

// ------------------------------------------------------------------------------------------------ geometry
constexpr size_t kSmemBudget = 227 * 1024;
// Head dims above 256: multiples of 64 up to this
constexpr int kBigMaxD = 1024;
// time steps of inputs in the shared-memory rings: lane loops, forward loop above head dim 256 (its reverse loop: one less)
constexpr int kLaneStages = 6, kBigStages = 4;

}  // namespace FRNN_NS
