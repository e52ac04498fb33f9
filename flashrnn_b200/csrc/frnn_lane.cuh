// What the forward and the reverse lane loop share (frnn_lane_fwd.cuh, frnn_lane_bwd.cuh): operand tiles in shared memory,
// the register-resident product, and the exchange between the CTAs of a cluster.
#pragma once
#include "frnn_cell.cuh"

namespace FRNN_NS {

// Operand tile of 8 batch rows x K 16-bit values: blocks of 8 k, each [8 rows][16 bytes] = 128 contiguous bytes, the rows of
// block i permuted by opnd_swz(i).  The 8 units (or gate rows) a warp produces for the 8 rows are ONE 128-byte block: what it
// sends to another CTA, or stores, is one line instead of eight pieces (the exchange is charged per piece: with rows of a
// plain [row][k] tile the C2 forward step took 1592 clk).  The permutation keeps the reads -- 16 bytes per lane, two rows of
// four blocks per wavefront -- and the stores of pairs of blocks free of bank conflicts.
__host__ __device__ constexpr uint32_t opnd_swz(uint32_t blk) { return (blk & 1) * 3 | ((blk & 2) << 1); }
__host__ __device__ constexpr uint32_t opnd_off(uint32_t row, uint32_t k) { return (k >> 3) * 128 + ((row ^ opnd_swz(k >> 3)) << 4) + (k & 7) * 2; }
__host__ __device__ constexpr int opnd_bytes(int k) { return k * 16; }

// A fragments (16 rows x 32 k) of one lane: its rows gid and gid + 8, eight consecutive k each (k = 8 tig .. 8 tig + 7).
// Which k an MMA calls its k-th is free as long as both operands agree, so a pair of k-steps takes contiguous 16 bytes
// per lane from either operand -- R in its own layout in global memory, h or the deltas in shared memory -- and neither a
// repacking pass nor ldmatrix is needed.  An odd last k-step uses four k per lane (.x, .y).
struct AFrag { uint4 lo, hi; };

// acc[m][nt][.] (+)= sum over k of A[m][.] (rows of this lane's MT tiles) times the operand tile: KS k-steps of 16, NT tiles of 8
// batch rows (`nt_bytes` apart).  INIT: acc holds the start value, else it starts from zero.  NS independent accumulator sets (see
// acc_sets).  The loads run PF k-pairs ahead of the products: without it every pair waited for its own 36 clk load.
// BP: bytes between the tile's blocks; other than 128, the rows of a block are not permuted.
template <int BP>
__device__ __forceinline__ uint32_t lane_opnd(int gid, int tig) {
  return (uint32_t)tig * BP + ((uint32_t)(BP == 128 ? gid ^ (int)opnd_swz((uint32_t)tig) : gid) << 4);
}
template <int MT, int KS, int NT, int NS, bool INIT, int BP = 128, class L>
__device__ __forceinline__ void lane_mma(const AFrag (&A)[MT][(KS + 1) / 2], uint32_t tile, int nt_bytes, int gid, int tig, float (&acc)[MT][NT][4],
                                         L late) {
  constexpr int KP = KS / 2, PF = KP < 4 ? (KP < 1 ? 1 : KP) : (NT > 1 ? 3 : 4);
  static_assert(NS <= KS, "every set gets a product");
  static_assert(BP == 128 || KS % 2 == 0, "whole k-pairs");
  float part[NS][MT][NT][4];
  const uint32_t base = tile + lane_opnd<BP>(gid, tig);
  uint4 b[PF][NT];
#pragma unroll
  for (int i = 0; i < PF && i < KP; ++i)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) b[i][nt] = lds128(base + (uint32_t)(i * 4 * BP + nt * nt_bytes));
  uint2 bo[NT];
  if constexpr ((KS & 1) != 0) {  // odd last k-step: four k per lane, in blocks 4 KP + (tig >> 1)
    const uint32_t blk = (uint32_t)(tig >> 1);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      bo[nt] = lds64(tile + (uint32_t)(KP * 512 + nt * nt_bytes) + blk * 128u + (((uint32_t)gid ^ opnd_swz(blk)) << 4) + (uint32_t)(tig & 1) * 8u);
  }
  if constexpr (INIT) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int c = 0; c < 4; ++c) part[0][m][nt][c] = acc[m][nt][c];
  }
  auto step = [&](int k, const uint4& a, int m, int nt, uint32_t b0, uint32_t b1) {
    if (k < NS && !(INIT && k == 0)) mma_16816_zero(part[k % NS][m][nt], a, b0, b1);
    else mma_16816(part[k % NS][m][nt], a, b0, b1);
  };
#pragma unroll
  for (int kp = 0; kp < KP; ++kp) {
    uint4 cur[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      cur[nt] = b[kp % PF][nt];
      if (kp + PF < KP) b[kp % PF][nt] = lds128(base + (uint32_t)((kp + PF) * 4 * BP + nt * nt_bytes));
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        step(2 * kp, make_uint4(A[m][kp].lo.x, A[m][kp].hi.x, A[m][kp].lo.y, A[m][kp].hi.y), m, nt, cur[nt].x, cur[nt].y);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        step(2 * kp + 1, make_uint4(A[m][kp].lo.z, A[m][kp].hi.z, A[m][kp].lo.w, A[m][kp].hi.w), m, nt, cur[nt].z, cur[nt].w);
  }
  if constexpr ((KS & 1) != 0) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int m = 0; m < MT; ++m)
        step(2 * KP, make_uint4(A[m][KP].lo.x, A[m][KP].hi.x, A[m][KP].lo.y, A[m][KP].hi.y), m, nt, bo[nt].x, bo[nt].y);
  }
  late();  // (work the products do not depend on, while the last of them complete)
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if constexpr (NS == 4) acc[m][nt][c] = (part[0][m][nt][c] + part[1][m][nt][c]) + (part[2][m][nt][c] + part[3][m][nt][c]);
        else if constexpr (NS == 2) acc[m][nt][c] = part[0][m][nt][c] + part[1][m][nt][c];
        else acc[m][nt][c] = part[0][m][nt][c];
      }
}
// Accumulator sets for `tiles` 16x8 tiles per warp, `warps` warps per CTA and `ks` k-steps, at least `want` independent chains per
// quadrant (see the uses).  An m16n8k16 occupies the tensor pipe of its quadrant for 8 clk and its result takes about 30.
__host__ __device__ constexpr int acc_sets(int tiles, int warps, int ks, int want) {
  const int chains = tiles * (warps > 4 ? warps / 4 : 1);
  const int sets = chains >= want ? 1 : (2 * chains >= want ? 2 : 4);
  return sets <= ks ? sets : (ks >= 2 ? 2 : 1);
}
template <bool PACKED> struct PairOf { using type = S2; };
template <> struct PairOf<true> { using type = P2; };

// Words of two 16-bit values in the activation cache: [t][n][b][D/2 unit pairs][slots]; four slots of a pair side by side (one
// 16-byte access), a fifth (sLSTM) in a plane of its own behind all of them.  The layout knows nothing of tiles, so the
// forward and the reverse loop choose theirs independently.
template <int GC> struct CacheGeom {
  static constexpr int MAIN = GC >= 4 ? 4 : GC;  // words per pair in the main plane (0: nothing cached)
  static constexpr bool EXTRA = GC > 4;
};

// Lane loops with the type of the states fixed at compile time (es = 2 or 4 bytes): the other type's side of every state access costs registers and issue
// slots, and where the compiler makes more of its absence such a form is used.  It does not everywhere (16 bits: GRU D = 128 forward 228 -> 246 us, LSTM D = 192
// reverse of 16 rows 392 -> 465; fp32: LSTM D = 16 forward 99 -> 134), so each was measured; those listed are ahead by 1 to 26 % (us; T512 and few CTAs, or the GPU
// filled; * 16 rows, + with warps that only multiply).
//   16 bits, forward  LSTM D = 16 101 -> 97, * 129 -> 121, 32 168 -> 140, 64 210 -> 200, 96 85 -> 83, 128 231 -> 224, 256 * 610 -> 592; GRU 16 91 -> 89, 32 154 -> 150, * 178 -> 163, 64 * 240 ->
//            226, 96 157 -> 155; sLSTM 32 176 -> 148, 64 251 -> 243, 96 259 -> 249, * 461 -> 406, 256 149 -> 145, * 654 -> 629; Elman 16 56 -> 52, * 35.5 -> 33.6, 32 63 -> 58, 64 79 ->
//            73, 128 179 -> 171, in one CTA 21.1 -> 19.1, 256 228 -> 222
//   16 bits, reverse  LSTM 16 142 -> 132, 32 159 -> 140, 96 * 410 -> 403, 128 263 -> 249 and 106 -> 82, 192 + 292 -> 286, 256 + 337 -> 330, * 703 -> 694; GRU 96 + 155 -> 141, 128 + 235 ->
//            228, 192 + 280 -> 264, * 257 -> 249, 256 97 -> 95; sLSTM 16 153 -> 126, 32 165 -> 162, 96 + 265 -> 228, 128 + 279 -> 265, 256 * 716 -> 695; Elman 16 66 -> 65, * 48 ->
//            44.5, 32 78 -> 62, 128 + 208 -> 201, in one CTA 29.0 -> 27.3, 192 + 239 -> 230, 256 in CTAs of 64 190 -> 185
//   fp32, forward     LSTM 32 217 -> 204, 64 278 -> 241, 96 255 -> 248, 128 243 -> 234, 192 263 -> 254, 256 298 -> 295, * 607 -> 589; GRU 16 91 -> 89, 64 183 -> 179, 96 156 -> 154, 192 247 -> 245,
//            256 * 573 -> 563; sLSTM 32 230 -> 214, 96 264 -> 253, * 447 -> 435, 128 275 -> 266, 192 281 -> 278 and 327 -> 302, 256 318 -> 312, * 636 -> 630; Elman 16 56 -> 50, 32 62 -> 58, 64 87 ->
//            81, 96 159 -> 155, 128 179 -> 168, in one CTA 21.4 -> 21.0, 192 206 -> 200, 256 234 -> 224
//   fp32, reverse     LSTM 32 156 -> 136, 64 245 -> 208, 96 * 436 -> 408, 128 278 -> 272, 192 + 304 -> 299, * 397 -> 293; GRU 32 193 -> 158, 64 218 -> 207, 96 + 164 -> 153, 128 + 246 -> 234, 192 + 283 ->
//            267, * 259 -> 256; sLSTM 16 144 -> 125, 32 163 -> 146, 64 251 -> 234, 96 + 276 -> 242, 128 + 288 -> 278, 256 * 723 -> 708; Elman 16 64 -> 60, * 67.4 -> 66.2, 32 74 -> 72, 64 130 -> 125, 128 +
//            208 -> 202, in one CTA 56 -> 52
__host__ __device__ constexpr bool states_form(int cell, bool bwd, int kt, int u, int nt, bool help, int es) {
  const int d = kt * 16;
  const bool one = nt == 1, dflt = u == (d <= 64 ? d : 32), h = es == 2;  // (CTAs the tile table makes)
  if (cell == CELL_ELMAN && one && !help && ((d == 128 && u == 128) || (h && bwd && d == 256 && u == 64))) return true;
  if (!dflt) return false;
  if (!bwd) {
    if (cell == CELL_LSTM) return one ? (h ? d <= 128 : d >= 32) : (h && d == 16) || d == 256;
    if (cell == CELL_GRU) return one ? d == 16 || (h && d == 32) || (!h && (d == 64 || d == 192)) || d == 96 : h ? d == 32 || d == 64 : d == 256;
    if (cell == CELL_SLSTM) return one ? d == 32 || (h && d == 64) || d == 96 || (!h && (d == 128 || d == 192)) || d == 256 : d == 96 || d == 256;
    if (cell == CELL_ELMAN) return one ? !h || d <= 64 || d == 128 || d == 256 : h && d == 16;
    return false;
  }
  if (cell == CELL_LSTM) return one ? (h && d == 16) || d == 32 || (!h && d == 64) || (d == 128 && !help) || (d == 192 && help) || (h && d == 256 && help) : d == 96 || d == (h ? 256 : 192);
  if (cell == CELL_GRU) return one ? (!h && (d == 32 || d == 64)) || ((d == 96 || d == 128) && help) || (d == 192 && (h || help)) || (h && d == 256 && !help) : d == 192;
  if (cell == CELL_SLSTM) return one ? d == 16 || d == 32 || (!h && d == 64) || ((d == 96 || d == 128) && help) : d == 256;
  if (cell == CELL_ELMAN) return one ? d == 16 || d == 32 || (!h && d == 64) || (d == 128 && help) || (h && d == 192 && help) : d == 16;
  return false;
}
// Some of these forms need registers that cost a CTA per SM, or most of the gain, once CTAs queue up; the general form runs then.  LSTM, us, D = 64 forward, 16 bits: B150 N12
// T64 50 -> 44, B400 N12 T128 204 -> 208, B1024 N16 T64 285 -> 296, fp32: B16 N12 T512 278 -> 241, B400 233 -> 241, B1024 325 -> 336; D = 32 reverse, 16 bits: B16 N8 T512 159 -> 140, B1024 N24 T64 239 -> 244.
// D = 32 forward, fp32: LSTM B64 N24 T256 130 -> 124, B1024 N24 T32 132 -> 138, sLSTM 146 -> 134, 138 -> 146 (without gradients), B200 N24 T64 87 -> 93.
__host__ __device__ constexpr bool states_form_for_few(int cell, bool bwd, int kt, int es) {
  if (cell == CELL_LSTM) return bwd ? kt == 2 && es == 2 : kt == 4 || (kt == 2 && es == 4);
  return cell == CELL_SLSTM && !bwd && kt == 2 && es == 4;
}
// Whether the reverse loops of 32-unit clusters and 8 rows are always those with warps that only multiply (lane_help in frnn_api.cu): there is no other form then.
__host__ __device__ constexpr bool help_always(int cell, int kt) {
  return cell == CELL_LSTM ? kt == 6 || kt == 12 || kt == 16 : cell == CELL_SLSTM ? kt == 6 || kt == 8 || kt == 12 || kt == 16 : cell == CELL_GRU && kt == 6;
}
// whether the form that reads the type of the states at run time is needed
__host__ __device__ constexpr bool states_general(int cell, bool bwd, int kt, int u, int nt, bool help) {
  return !states_form(cell, bwd, kt, u, nt, help, 2) || !states_form(cell, bwd, kt, u, nt, help, 4) || states_form_for_few(cell, bwd, kt, 2) || states_form_for_few(cell, bwd, kt, 4);
}

// ---- IO warps.  A lane's values belong to 8 batch rows per warp instruction (the MMA's accumulator layout), and the L1 charges
// a global access per row touched: with the compute lanes loading Wx and storing states and cache themselves the LSTM D = 64 forward
// step spent ~700 of 1380 clk on it.  So one or two extra warps move everything between global memory and padded tiles in shared
// memory, 16 bytes per lane along the rows, and the compute lanes touch shared memory only.
__host__ __device__ constexpr int io_warps(int bytes_per_step) { return bytes_per_step > 6144 ? 2 : 1; }
// row pitch of such a tile: 16 bytes of padding make the compute lanes' accesses (4 to 16 bytes, 8 rows) conflict-free
__host__ __device__ constexpr int io_pitch(int row_bytes) { return row_bytes + 16; }

// One lane's share of a tile of ROWS rows x CPR 16-byte chunks, moved by IOT lanes: chunk i of the lane is row row(i), column col(i).
// `cpr`: the actual number of chunks per row where CPR is only the most there can be.
template <int ROWS, int CPR, int IOT>
struct IoTile {
  static constexpr int N = (ROWS * CPR + IOT - 1) / IOT;  // chunks per lane
  // where chunks per row and lanes divide one another, a chunk's place is its lane's plus a constant (one address register for all i)
  static constexpr bool COLS_FIT = IOT % CPR == 0, ROWS_FIT = CPR % IOT == 0;
  static __device__ __forceinline__ int row(int lane, int i, int cpr = CPR) {
    if (COLS_FIT && cpr == CPR) return lane / CPR + i * (IOT / CPR);
    if (ROWS_FIT && cpr == CPR) return i / (ROWS_FIT ? CPR / IOT : 1);
    return (int)((unsigned)(lane + i * IOT) / (unsigned)cpr);
  }
  static __device__ __forceinline__ int col(int lane, int i, int cpr = CPR) {
    if (COLS_FIT && cpr == CPR) return lane % CPR;
    if (ROWS_FIT && cpr == CPR) return lane + (i % (ROWS_FIT ? CPR / IOT : 1)) * IOT;
    return (int)((unsigned)(lane + i * IOT) % (unsigned)cpr);
  }
  static __device__ __forceinline__ bool in(int lane, int i, int cpr = CPR) { return (ROWS * CPR % IOT == 0 && cpr == CPR) || lane + i * IOT < ROWS * cpr; }
};

}  // namespace FRNN_NS
