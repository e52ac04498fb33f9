// C ABI of libfrnn_b200.so (declared in include/frnn.h): validation, tile selection, launches.
// No device memory is allocated or freed here and the host is never synchronised with the device,
// except in frnn_read_device_status.
#include "../../include/frnn.h"

#include <mutex>

#include "frnn_aux.cuh"
#include "frnn_lane.cuh"

namespace FRNN_NS {

struct CellDims { int Gr, Gw, Gt, S, GC; };
static bool cell_dims(int cell, CellDims* d) {
  switch (cell) {
    case CELL_LSTM:  *d = {4, 4, 4, 2, 4}; return true;
    case CELL_GRU:   *d = {3, 3, 4, 1, 4}; return true;
    case CELL_ELMAN: *d = {1, 1, 1, 1, 1}; return true;
    case CELL_SLSTM: *d = {4, 4, 4, 4, 5}; return true;
  }
  return false;
}

// The lane loops (head dims up to 256) of a kernel family (kernel_cell), direction and tile, null: none; those with warps that only multiply, null: none
constexpr LaneTiles kLaneTileAt;
static const LaneForms* lane_forms(int cell, bool bwd, int kt, int u, int nt) {
  static const LaneForms (*const tables[5][2])[2] = {{lane_fwd_lstm, lane_bwd_lstm}, {lane_fwd_gru, lane_bwd_gru}, {lane_fwd_elman, lane_bwd_elman},
                                                     {lane_fwd_slstm, lane_bwd_slstm}, {lane_fwd_elmanc, lane_bwd_elmanc}};  // by CELL_*
  const int at = u % 16 == 0 && u <= 128 ? kLaneTileAt.at[kt][u / 16] : -1;
  return at < 0 ? nullptr : &tables[cell][bwd][at][nt - 1];
}
static const LaneForms* lane_help_forms(int cell, int kt) {
  static const LaneForms* const tables[5] = {lane_bwd_help_lstm, lane_bwd_help_gru, lane_bwd_help_elman, lane_bwd_help_slstm, lane_bwd_help_elmanc};
  for (int i = 0; i < 4; ++i)
    if (kHelpKTs[i] == kt) return &tables[cell][i];
  return nullptr;
}
static LaneKernel lane_dr_kernel(int cell) {
  switch (cell) {
    case CELL_LSTM: return lane_bwd_dr_lstm;
    case CELL_GRU: return lane_bwd_dr_gru;
    case CELL_SLSTM: return lane_bwd_dr_slstm;
  }
  return LaneKernel{nullptr, 0, 0};
}
// The head dims above 256
static BigKernel big_kernel(int cell, bool bwd, int u, int nt, bool dense) {
  switch (cell) {
    case CELL_LSTM: return bwd ? big_bwd_lstm(u, nt) : big_fwd_lstm(u, nt, dense);
    case CELL_GRU: return bwd ? big_bwd_gru(u, nt) : big_fwd_gru(u, nt, dense);
    case CELL_ELMAN: return bwd ? big_bwd_elman(u, nt) : big_fwd_elman(u, nt, dense);
    case CELL_ELMAN_CLIP: return bwd ? big_bwd_elmanc(u, nt) : big_fwd_elmanc(u, nt, dense);
    case CELL_SLSTM: return bwd ? big_bwd_slstm(u, nt) : big_fwd_slstm(u, nt, dense);
  }
  return BigKernel{nullptr, 0, nullptr};
}
static cudaError_t big_pack(int cell, const void* R, void* out, int N, int D, cudaStream_t stream) {
  switch (cell) {
    case CELL_LSTM: return big_pack_lstm(R, out, N, D, stream);
    case CELL_GRU: return big_pack_gru(R, out, N, D, stream);
    case CELL_SLSTM: return big_pack_slstm(R, out, N, D, stream);
    default: return big_pack_elman(R, out, N, D, stream);
  }
}

// kernel family of a problem: the public cell id, except Elman with a forward clamp (caches its tanh output)
static int kernel_cell(const frnn_problem& pr) {
  return (pr.cell == CELL_ELMAN && pr.forward_clip > 0.f) ? (int)CELL_ELMAN_CLIP : pr.cell;
}

// Activation values cached per (b,t,n,d) in training.  Elman needs its one slot (the tanh output) only when h is
// clamped afterwards; otherwise h itself serves and no cache buffer is needed at all.
static int cache_slots_of(const frnn_problem& pr, const CellDims& cd) {
  return (pr.cell == CELL_ELMAN && !(pr.forward_clip > 0.f)) ? 0 : cd.GC;
}

static int sm_count_cached();

constexpr int kMaxTiles = 65535;  // blocks in y of a launch

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
constexpr size_t kMaxDynSmem = 227 * 1024, kSmemPerSm = 228 * 1024;
constexpr size_t kStatusBytes = 256;

// Head dims above 256 have kernels of their own (frnn_big_*.cuh).  Their plan names 64 units per CTA and clusters of D / 64; unless the
// caller asked for that, the loops split the head as big_tile says.
static bool is_big(const frnn_problem& pr) { return pr.D > 256; }
constexpr int kBigPlanUnits = 64;

// Clusters of one CTA per SM that a B200 keeps resident, by their size (12: as if; the occupancy calculator says 8)
constexpr int kResident[17] = {0, 148, 74, 45, 33, 26, 22, 17, 15, 14, 11, 8, 7, 8, 8, 7, 7};

// Units per CTA and rows / 8 of one of those loops: the fewest turns of all clusters through the GPU, weighed with what a step takes.
// `dense`: the form of Elman's 64-unit forward CTAs of which two fit an SM (frnn_big_fwd.cuh).
struct BigTile { int u, nt; bool dense; };
// A step alone, 8 / 16 rows, relative to the others of its head dim: 32, 48 and 64 units up to head dim 576 (forward) and 512 (reverse), where a 32-unit one
// of 8 rows is 100, then 48 and 64 above.  Measured, us per step: D = 384, 32, 48, 64 units: LSTM forward 0.94 / 1.41, 1.05 / 1.81, 1.41 / 2.21, reverse 0.86 / 1.49, 1.26 /
// 2.36, 1.77 / 3.57; GRU forward 0.90 / 1.38, 1.05 / 1.72, 1.39 / 2.20, reverse 0.83 / 1.40, 1.20 / 2.10, 1.42 / 2.57; sLSTM forward 0.99 / 1.51, 1.13 / 1.98, 1.60 / 2.37,
// reverse 0.87 / 1.54, 1.28 / 2.79, 1.88 / 4.76; Elman 0.80 / 1.25, 0.86 / 1.28, 0.82 / 1.28, reverse 0.96 / 1.44, 0.96 / 1.57, 1.03 / 1.76.  D = 768, 48, 64 units: LSTM
// forward 1.74 / 3.17, 2.38 / 3.95, reverse 1.82 / 3.68, 2.71 / 6.19; GRU 1.79 / 3.10, 2.40 / 3.79, reverse 1.71 / 3.25, 1.94 / 3.87; sLSTM 1.81 / 3.38, 2.53 / 4.12, reverse 1.83 / 4.96,
// 3.35 / 7.92.
constexpr int kBigWeight[4][2][5][2] = {
    {{{100, 150}, {112, 193}, {150, 235}, {87, 158}, {119, 198}}, {{100, 173}, {147, 274}, {206, 415}, {91, 184}, {136, 310}}},     // LSTM: forward, reverse
    {{{100, 153}, {117, 191}, {154, 244}, {90, 155}, {120, 190}}, {{100, 169}, {145, 253}, {171, 310}, {86, 163}, {97, 194}}},      // GRU
    {{{100, 156}, {106, 160}, {102, 175}, {100, 172}, {102, 172}}, {{100, 155}, {104, 162}, {107, 178}, {104, 170}, {106, 182}}},   // Elman
    {{{100, 153}, {114, 200}, {162, 239}, {91, 169}, {127, 206}}, {{100, 177}, {147, 321}, {216, 547}, {92, 248}, {168, 396}}}};    // sLSTM
static BigTile big_tile(const frnn_problem& pr, bool bwd) {
  const bool elman = pr.cell == CELL_ELMAN;
  BigTile best = {64, 1, false};
  long long best_cost = -1;
  auto offer = [&](int i, int nt, bool dense, int weight, int per_sm, int shared) {  // shared: a step beside another CTA's, in percent of one alone
    const long long tiles = (long long)((pr.B + 8 * nt - 1) / (8 * nt)) * pr.N, alone = kResident[pr.D / (32 + 16 * i)];
    if (nt == 1 && (pr.B + 7) / 8 > kMaxTiles) return;
    const long long turns = (tiles + alone * per_sm - 1) / (alone * per_sm), cost = tiles <= alone ? weight * 100LL : turns * weight * shared;
    if (best_cost < 0 || cost < best_cost) { best = {32 + 16 * i, nt, dense}; best_cost = cost; }
  };
  for (int i = 0; i < 3; ++i) {
    const int u = 32 + 16 * i, cs = pr.D / u;
    if (pr.D % u || cs > 16 || pr.D / 16 > u) continue;
    for (int nt = 1; nt <= (pr.B > 8 ? 2 : 1); ++nt) {
      const int weight = kBigWeight[pr.cell][bwd][pr.D > (bwd ? 512 : 576) ? 2 + i : i][nt - 1];
      // Elman's CTAs are small: two of 32 units fit an SM (of clusters of 16 little more run at once than with one), and two of 64 units in the
      // forward loop's dense form, beside each other 1.3 times slower.  That form has all of R in registers up to D = 512 and nearly all at 640, where it
      // takes the place of the other; above, its step is longer, D = 1024 1.35 / 2.44 -> 1.64 / 2.89 us, and it pays where clusters queue up.  All clusters
      // of B600, us per step, one per SM and two: N5 D320 11.1 -> 6.3, N5 D384 13.9 -> 8.5, N3 D640 22.3 -> 12.9, N2 D1024 32.4 -> 25.3.
      const bool small = elman && u == 32 && cs <= 12;
      if (!(elman && !bwd && u == 64 && pr.D <= 640)) offer(i, nt, false, weight, small ? 2 : 1, small ? 115 : 100);
      if (elman && !bwd && u == 64) {
        const bool two = big_kernel(CELL_ELMAN, false, u, nt, true).smem(pr.D) <= kSmemPerSm / 2 - 1024;
        offer(i, nt, true, nt == 1 ? 106 + (pr.D > 640 ? (pr.D - 640) / 32 : 0) : 165 + (pr.D > 640 ? (pr.D - 640) / 8 : 0), two ? 2 : 1, two ? 130 : 100);
      }
    }
  }
  return best;
}
static BigTile big_tile(const frnn_plan& pl, bool bwd) {
  if (pl.forced_tile) return {kBigPlanUnits, pl.batch_tile / 8, pl.prob.cell == CELL_ELMAN && !bwd && pl.prob.D <= 640};
  return big_tile(pl.prob, bwd);
}
// units per CTA of the reverse loop, by which R^T is packed
static int reverse_units(const frnn_plan& pl) { return is_big(pl.prob) ? big_tile(pl, true).u : pl.units_per_cta; }

// Scratch of a plan: status block, then what the plan's kernels need.  Only head dims above 256 repack R for the forward pass.
struct WsLayout { size_t rpack_fwd, rpack_bwd, grads, dg0, total; };
// units: per CTA of the reverse loop
static WsLayout workspace_layout(const frnn_problem& pr, const CellDims& cd, int units) {
  WsLayout w;
  size_t off = kStatusBytes;
  w.rpack_fwd = off; if (is_big(pr)) off = align_up(off + (size_t)(cd.Gr > 1 ? 4 : 1) * pr.N * pr.D * pr.D * 2, 256);
  w.rpack_bwd = off; if (pr.training) off = align_up(off + rt_pack_bytes(cd.Gr, pr.N, pr.D, units), 256);
  w.grads = off; if (pr.training) off = align_up(off + ((size_t)cd.Gr * pr.N * pr.D * pr.D + (size_t)cd.Gt * pr.N * pr.D) * 4, 256);
  w.dg0 = off;
  if (pr.training && pr.cell == CELL_GRU) off = align_up(off + (size_t)pr.B * pr.T * pr.N * pr.D * 2, 256);
  w.total = off;
  return w;
}

// A tile (cluster size, batch tile) is usable when both loop kernels exist for it, the CTA fits the
// instantiation's thread bound and the shared-memory budget.
static bool wide_problem(const frnn_problem& pr) {
  return wide_supported(pr.cell, pr.D, pr.dtype_state == FRNN_DTYPE_F32, pr.forward_clip, pr.grad_clip, pr.grad_cut);
}
static bool is_wide(const frnn_plan& pl) { return pl.batch_tile == kWideBatchTile; }
// LSTM and GRU at head dim 64: the forward loop alone has a 128-row form (the reverse loop stays on 16-row tiles)
static bool wide_gates_problem(const frnn_problem& pr) {
  return wide_gates_forward_supported(pr.cell, pr.D, pr.dtype_state == FRNN_DTYPE_F32);
}
// (a training pass stores activations, where the lane loop is ahead: see frnn_wide.cu)
static bool runs_wide_gates(const frnn_plan& pl) { return pl.wide_forward && !pl.prob.training; }
static int plan_threads(const CellDims& cd, int units, int bt) { return bt == kWideBatchTile ? kWideThreads : 2 * cd.Gr * units; }

// Rows / 8 the lane loops run a plan's batch tile with (the activation cache and every result are the same whatever it is): 16 where the caller
// asked for as many, or where 8-row tiles would be more than a grid holds in y; else what is faster.
// 16-row tiles reuse a fragment of R for two products but hold twice the items per lane.  Measured at batches that fill the GPU, B1024 and N * D = 1024, T = 48,
// us of 8 / 16 rows; forward: GRU D = 64 205 / 185, D = 32 162 / 181 (B256 N24 T128 96 / 92), D = 16 166 / 175 (B1024 N24 T128 192 / 169); LSTM D = 64 217 / 305, D = 96 356 / 324 (B200 118 / 137), D = 128 463 / 390, D = 192
// 545 / 667, D = 256 1222 / 921; GRU D = 96 333 / 297 (B200 113 / 127), D = 128 361 / 378, D = 192 500 / 634, D = 256 1184 / 865; sLSTM D = 64 301 / 471, D = 96 493 / 419 (B256 N8
// T128, three turns of 16-row clusters, 256 / 288),
// D = 128 568 / 477, D = 192 624 / 754, D = 256 1280 / 1020.  Reverse: one CTA per head, D = 64, LSTM 248 / 287, GRU 218 / 299, sLSTM 304 / 369; clusters, LSTM D = 96 to
// 256 493 / 395, 513 / 456, 1063 / 884, 1394 / 1082, GRU 381 / 386 (B200 130 / 158), 421 / 421 (B200 134 / 160), 558 / 499, 738 / 1002, sLSTM 565 / 662, 612 / 703, 1020 / 800,
// 1442 / 1128.  D = 16, B1024, N = 24, 40 (T = 96), 64, 96: forward sLSTM 332 / 292, 585 / 533, 369 / 328, 523 / 484, LSTM 210 / 189, 392 / 326, 248 / 229, 358 / 337 (without
// gradients 134 / 139, 237 / 207, 149 / 166, 235 / 245), Elman 49 / 49, 138 / 81, 68 / 57, 142 / 89, reverse 131 / 82, 210 / 113, 151 / 92, 233 / 137, sLSTM 371 / 394, 648 / 586,
// 347 / 491, 536 / 731; with a quarter of the tiles 8 rows are ahead everywhere, by 5 to 20 %.
constexpr long long kManyTiles = 1500;
static int lane_nt(const frnn_problem& pr, bool bwd, int bt, bool forced) {
  if (bt < 16) return 1;
  if (forced || (pr.B + 7) / 8 > kMaxTiles) return 2;
  const int D = pr.D;
  const long long tiles = (long long)((pr.B + 15) / 16) * pr.N;
  if (D == 16 && pr.cell != CELL_GRU) return tiles >= kManyTiles && (pr.cell == CELL_ELMAN || (!bwd && (pr.cell == CELL_SLSTM || pr.training))) ? 2 : 1;
  const bool two = bwd ? D >= 96 && (pr.cell == CELL_LSTM || D == 192 || (pr.cell == CELL_SLSTM && D == 256))
                       : D == 256 || (D <= 64 && pr.cell == CELL_GRU) || (D == 128 && pr.cell != CELL_GRU) || (D == 96 && pr.cell == CELL_SLSTM && tiles >= 180);
  return two ? 2 : 1;
}

// The reverse lane loop with warps that only multiply (8-row clusters of 32-unit CTAs).  Where every CTA has an SM to itself, always: us per 256 steps of one tile
// without / with, beside the geometry.  With more CTAs only where it is ahead there too; us of B200 T48 and N * D = 768, without / with: LSTM D = 96 111 / 99, 192 176 / 167, 256
// 215 / 195; sLSTM D = 96 122 / 110, 128 124 / 115, 192 183 / 171, 256 218 / 190; GRU D = 96 80 / 72 (B1024 T32 233 / 212), but 128 83 / 97, 192 118 / 157, 256 136 / 172; Elman D = 96 41 / 38,
// but B1024 T32 124 / 130.
static bool lane_help(const frnn_problem& pr, int cs, int u, int nt) {
  if (cs < 2 || cs > 16 || u != 32 || nt != 1) return false;
  const bool alone = (long long)((pr.B + 7) / 8) * pr.N <= kResident[cs];
  return alone || help_always(kernel_cell(pr), pr.D / 16);
}

// Whether the reverse lane loop forms dR as well (lane_bwd_dr): head dim 64 with one CTA per head, 8 rows and 16-bit states.  Not for the shortest
// sequences: a CTA adds its 48 or 64 KB of sums to the gradient once.  Backward pass, us, dR in its own kernel / in the loop, B1024 N16: LSTM T16 162 / 172, T20 192 / 190, T24 229 /
// 222, T32 281 / 262, GRU T24 212 / 179, sLSTM T24 260 / 241.  A step of the LSTM's and the sLSTM's loop takes 20 to 60 ns longer with it, which on long sequences
// only pays once their own kernel takes that.  LSTM, tiles: T256 2 132 / 134, 8 136 / 133, 24 144 / 134, T512 2 240 / 246, 8 245 / 247, 16 251 / 253, 24 261 / 251, T2048 16 918 /
// 943, 24 959 / 949, 32 980 / 951.  sLSTM: T64 24 58 / 51, T256 8 138 / 144, 24 150 / 146, T512 24 267 / 273, 48 284 / 275, T2048 24 986 / 1036, 48 1043 / 1043, 64 1070 /
// 1043.  GRU, any: T512 1 232 / 193, 24 249 / 196, T2048 24 917 / 727.
constexpr int kDrMinSteps = 24, kDrShort = 256, kDrThreads = 32;
static bool lane_dr(const frnn_plan& pl, int nt) {
  const frnn_problem& pr = pl.prob;
  if (pr.D != 64 || pl.cluster_size != 1 || nt != 1 || pr.cell == CELL_ELMAN || pr.dtype_state == FRNN_DTYPE_F32 || pl.forced_tile) return false;
  const long long tiles = (long long)((pr.B + 7) / 8) * pr.N;
  const int enough = pr.cell == CELL_GRU ? 0 : pr.cell == CELL_LSTM ? (pr.T <= kDrShort ? 0 : 24) : pr.T <= kDrShort ? 24 : 48;
  return pr.T >= kDrMinSteps && tiles >= enough;
}

// The lane loop of a plan's tile: with the type of its states fixed where there is such a form and it pays, else the general one.
static LaneKernel lane_loop(const frnn_problem& pr, bool bwd, int u, int nt, bool help) {
  const int cell = kernel_cell(pr), kt = pr.D / 16, f32 = pr.dtype_state == FRNN_DTYPE_F32;
  const LaneForms* f = help ? lane_help_forms(cell, kt) : lane_forms(cell, bwd, kt, u, nt);
  if (!f) return LaneKernel{nullptr, 0, 0};
  if (f->few[f32].fn == f->many[f32].fn) return f->few[f32];
  return (long long)((pr.B + 8 * nt - 1) / (8 * nt)) * pr.N * (pr.D / u) <= 2LL * sm_count_cached() ? f->few[f32] : f->many[f32];
}
static bool lane_exists(const frnn_problem& pr, bool bwd, int u, int nt) {
  if (bwd && u == 32 && nt == 1 && help_always(kernel_cell(pr), pr.D / 16)) return true;
  const LaneForms* f = lane_forms(kernel_cell(pr), bwd, pr.D / 16, u, nt);
  return f && f->few[pr.dtype_state == FRNN_DTYPE_F32].fn;
}

static bool tile_ok(const frnn_problem& pr, const CellDims& cd, int cs, int bt) {
  const int D = pr.D;
  if (bt == kWideBatchTile) return cs == 1 && wide_problem(pr);  // 128-row tensor-core loops: one CTA per head and tile
  if (cs < 1 || D % cs) return false;
  if (is_big(pr)) return D / cs == kBigPlanUnits && (bt == 8 || bt == 16);
  // clusters above 8 CTAs (a non-portable size): 16 CTAs of 16 units for head dim 256
  if (cs > 8 && !(cs == 16 && D == 256)) return false;
  const int U = D / cs;
  if (U % 16 || ((U / 16) & (U / 16 - 1))) return false;  // 16 * power of two
  if (bt != 8 && bt != 16 && bt != 32) return false;
  // a CTA owns at most 512 gate-row halves (256 from head dim 256, 384 from 192 up: the registers that hold R), and with
  // 32-row tiles at most 192 gate rows
  const int threads = 2 * cd.Gr * U;
  if (threads > (D < 192 ? 512 : D < 256 ? 384 : 256)) return false;
  if (bt == 32 && cd.Gr * U > 192) return false;
  for (int nt = 1; nt <= (bt < 16 ? 1 : 2); ++nt)
    if (!lane_exists(pr, false, U, nt) || !lane_exists(pr, true, U, nt)) return false;
  return true;
}

// Default tile per problem.  Small-batch problems are bound by the per-step latency of the serial chain, so
// the head is spread over as many SMs as a portable cluster allows; large-batch problems already fill the
// GPU with (head, batch tile) pairs and take the smallest cluster (no cross-CTA exchange when it is 1).
static bool choose_tile(const frnn_problem& pr, const CellDims& cd, int want_cs, int want_bt, int* cs_out, int* bt_out) {
  // Large batches of a cell / head dim the 128-row tensor-core loops cover: those stream at the HBM rate once their
  // (head, 128-row tile) pairs occupy most of the SMs
  if (want_bt == kWideBatchTile && wide_gates_problem(pr)) want_bt = 16;  // 128-row forward loop over 16-row reverse tiles
  if ((want_bt == kWideBatchTile || (!want_bt && !want_cs && (long long)(pr.B / kWideBatchTile) * pr.N >= 64)) &&
      tile_ok(pr, cd, 1, kWideBatchTile) && (want_cs == 0 || want_cs == 1)) {
    *cs_out = 1;
    *bt_out = kWideBatchTile;
    return true;
  }
  // Large batches of the cells with three or four gates (128 or more (head, 16-row tile) pairs): plans of 16 rows, of which lane_nt and big_tile
  // say what each loop takes at a time.  Small batches: 8 rows, more CTAs and shorter steps (one tile alone, 8 / 16 rows, T = 128, us of both loops:
  // LSTM D = 64 119 / 211, D = 128 137 / 195, GRU D = 256 178 / 259), and Elman above head dim 16 (B1024 N6 D = 128, T = 32: 129 / 113, but B1024 N12 D = 64 84 / 88).
  const long long tiles16 = (long long)((pr.B + 15) / 16) * pr.N;
  const bool rows16 = cd.Gr >= 3 ? tiles16 >= 128 : pr.D == 16 && tiles16 >= kManyTiles && (pr.B + 7) / 8 <= kMaxTiles;
  const int bt_pref[3] = {rows16 ? 16 : 8, rows16 ? 8 : 16, 32};
  for (int bi = 0; bi < 3; ++bi) {
    const int bt = want_bt ? want_bt : bt_pref[bi];
    const long long pairs = (long long)((pr.B + bt - 1) / bt) * pr.N;
    const bool fill = pairs >= 128;
    // power-of-two cluster sizes first, then the others
    const int order_small[8] = {8, 4, 2, 1, 6, 3, 7, 5};
    const int order_large[8] = {1, 2, 4, 8, 3, 6, 5, 7};
    const int sms = sm_count_cached();
    // The preferred cluster, small batch or large: 32 units per CTA from head dim 96 (clusters of D / 32), the whole head in one CTA up to head
    // dim 64, without any exchange.  us of both loops, one 8-row tile and T = 128 | B1024, N * D = 768 and T = 32 with the better of 8 and 16 rows:
    // D = 64, 1, 2, 4 CTAs: LSTM 119, 129, 123 | 274, 354, 443; GRU 107, 119, 114 | 244, 301, 386; sLSTM 129, 125, 121 | 352, 468, 536; Elman 54, 92, 90 | 84,
    // 153, 252.  D = 96, 3, 6 CTAs: LSTM 142, 125 | 436, 524.  D = 128, 2, 4, 8 CTAs: LSTM 205, 137, 135 | 534, 465, 593; GRU 175, 138, 135 | 425, 430, 543; sLSTM
    // 206, 158, 156 | 610, 599, 762.  D = 192, 3, 6 CTAs: GRU 189, 148 | 543, 569.  D = 256, 8, 16 CTAs: LSTM 181, 190 | 1068, 1490.
    // Small batches fall back to smaller clusters when the preferred one would not give every CTA an SM of its own; the second pass takes
    // whatever exists.
    const int cs32 = pr.D <= 64 ? 1 : ((pr.D % 32 == 0 && pr.D / 32 <= 8) ? pr.D / 32 : 0);
    for (int pass = 0; pass < 2; ++pass)
      for (int ci = -1; ci < 8; ++ci) {
        // Elman, where its CTAs fill the GPU or would not all get an SM: the whole head in one CTA up to head dim 128, 64 units per CTA above.  us of
        // both loops, T = 48: B150 N10 D = 128, 1, 2, 4 CTAs 62, 74, 100; D = 192, 3, 6 CTAs, B150 N5 84, 125, N10 145, 196; D = 256, 2, 4, 8 CTAs, B150 N5
        // 169, 119, 183, B300 N4 244, 190, 265.  (Forward alone, B1024 N4 D = 256 T64, 2, 4 CTAs 274, 307: without gradients the smallest cluster.)
        const int first = cd.Gr > 1 || (!fill && (pass == 0 || pr.D < 192)) ? cs32 : pr.D >= 192 && (pr.training || !fill) ? pr.D / 64 : 0;
        if (ci < 0 && (want_cs || is_big(pr) || !first)) continue;
        int cs = ci < 0 ? first : (want_cs ? want_cs : (fill ? order_large[ci] : order_small[ci]));
        if (ci >= 0 && !fill && !want_cs && cs32 && cs > cs32) continue;  // fewer than 32 units per CTA
        if (is_big(pr) && !want_cs) cs = pr.D / kBigPlanUnits;
        const bool crowded = !fill && !want_cs && !is_big(pr) && pairs * cs > sms;
        if (!(pass == 0 && crowded) && tile_ok(pr, cd, cs, bt)) { *cs_out = cs; *bt_out = bt; return true; }
        if (want_cs || is_big(pr)) break;
      }
    if (want_bt) break;
  }
  return false;
}

static int validate_problem(const frnn_problem* pr, CellDims* cd) {
  if (!pr) return FRNN_ERR_NULL;
  if (!cell_dims(pr->cell, cd)) return FRNN_ERR_CELL;
  constexpr int io = kF16 ? FRNN_DTYPE_F16 : FRNN_DTYPE_BF16;  // the element type this build of the kernels computes in
  if (pr->dtype_io != io) return FRNN_ERR_DTYPE;
  if (pr->dtype_state != io && pr->dtype_state != FRNN_DTYPE_F32) return FRNN_ERR_DTYPE;
  if (pr->B < 1 || pr->T < 1 || pr->N < 1 || pr->D < 1) return FRNN_ERR_SHAPE;
  if (pr->N > 65535) return FRNN_ERR_SHAPE;
  if (pr->D % 16) return FRNN_ERR_SHAPE;
  bool kt_ok = pr->D > 256 && pr->D <= kBigMaxD && pr->D % kBigPlanUnits == 0;
  for (int i = 0; i < kNumKT; ++i) kt_ok = kt_ok || (kKTs[i] * 16 == pr->D);
  if (!kt_ok) return FRNN_ERR_SHAPE;
  return FRNN_OK;
}

// The kernel a time loop of a plan runs, with its CTAs.  fn null: there is none (a measurement variant of another tile).
struct LoopLaunch {
  const void* fn;
  int threads, stages;
  size_t smem;
  int cs, u, rows;
  bool dr;  // the reverse loop forms dR, too
};
static LoopLaunch loop_of(const frnn_plan& pl, bool bwd) {
  const frnn_problem& pr = pl.prob;
  const int cell = kernel_cell(pr);
  if (is_big(pr)) {
    const BigTile t = big_tile(pl, bwd);
    int nt = t.nt;
    BigKernel k = big_kernel(cell, bwd, t.u, nt, t.dense);
    if (k.fn && k.smem(pr.D) > kSmemBudget) k = big_kernel(cell, bwd, t.u, nt = 1, t.dense);  // (sLSTM reverse from head dim 960 up)
    if (!k.fn || pl.probe_noop_cell) return LoopLaunch{};
    return LoopLaunch{k.fn, k.threads, bwd ? kBigStages - 1 : kBigStages, k.smem(pr.D), pr.D / t.u, t.u, 8 * nt};
  }
  const int kt = pr.D / 16, u = pl.units_per_cta, nt = lane_nt(pr, bwd, pl.batch_tile, pl.forced_tile);
  const bool dr = bwd && !pl.probe_noop_cell && lane_dr(pl, nt);
  LaneKernel k = {nullptr, 0, 0};
  if (pl.probe_noop_cell) k = lane_floor(pr.cell, bwd, kt, u, nt, pr.dtype_state == FRNN_DTYPE_F32 ? 4 : 2);
  else if (dr) k = lane_dr_kernel(cell);
  else if (bwd && lane_help(pr, pl.cluster_size, u, nt)) k = lane_loop(pr, true, u, nt, true);
  if (!k.fn && !pl.probe_noop_cell) k = lane_loop(pr, bwd, u, nt, false);
  return LoopLaunch{reinterpret_cast<const void*>(k.fn), k.threads, kLaneStages, k.smem, pl.cluster_size, u, 8 * nt, dr};
}
// x: the CTAs of a cluster, y: tiles of the batch, z: heads
static int loop_tiles(const LoopLaunch& k, const frnn_problem& pr) { return (pr.B + k.rows - 1) / k.rows; }
static dim3 loop_grid(const LoopLaunch& k, const frnn_problem& pr) { return dim3((unsigned)k.cs, (unsigned)loop_tiles(k, pr), (unsigned)pr.N); }

static int fill_plan(const frnn_problem* pr, int cs, int bt, int stages, frnn_plan* out) {
  CellDims cd;
  const int rc = validate_problem(pr, &cd);
  if (rc) return rc;
  if (!out) return FRNN_ERR_NULL;
  if (stages != 0 && stages != 4) return FRNN_ERR_PLAN;  // (the one depth there was before the loops had rings of their own)
  int ccs = 0, cbt = 0;
  if (!choose_tile(*pr, cd, cs, bt, &ccs, &cbt)) return (cs || bt) ? FRNN_ERR_PLAN : FRNN_ERR_SHAPE;
  if ((long long)((pr->B + cbt - 1) / cbt) > 65535) return FRNN_ERR_SHAPE;
  frnn_plan pl = {};
  pl.abi_version = FRNN_ABI_VERSION;
  pl.prob = *pr;
  pl.cluster_size = ccs;
  pl.units_per_cta = pr->D / ccs;
  pl.batch_tile = cbt;
  pl.threads = plan_threads(cd, pl.units_per_cta, cbt);
  // A step of the 128-row forward loop takes about 2.5 us however few CTAs run, so it pays once they occupy most of the SMs.  Inference, N16 T128, B = 512,
  // 640, 768, 1024, 2048 (64, 80, 96, 128, 256 CTAs), us against the better of the lane loops: LSTM 299 / 255, 313 / 323, 325 / 392, 345 / 459, 696 / 901; GRU 245 /
  // 213, 250 / 269, 255 / 326, 273 / 388, 536 / 762.
  pl.wide_forward = wide_gates_problem(*pr) && ccs == 1 && cbt == 16 &&
                    (bt == kWideBatchTile || (!cs && !bt && (long long)(pr->B / kWideBatchTile) * pr->N >= 96));
  pl.wx_stages = is_wide(pl) ? kWideFwdStages : runs_wide_gates(pl) ? kWideGatesStages : is_big(*pr) ? kBigStages : kLaneStages;
  pl.cache_slots = cache_slots_of(*pr, cd);
  // one bf16 pair per (item, slot, step) in the time loops' own order; batch rows padded to whole tiles
  const uint64_t rows = (uint64_t)((pr->B + cbt - 1) / cbt) * cbt;
  pl.cache_bytes = rows * pr->T * pl.cache_slots * pr->N * pr->D * 2;
  pl.forced_tile = (cs || bt) && bt != kWideBatchTile;  // (128 rows: a loop of its own, the other loops as if nothing was asked for)
  if (is_big(*pr))
    for (int bwd = 0; bwd <= (pr->training ? 1 : 0); ++bwd)
      if (loop_tiles(loop_of(pl, bwd), *pr) > kMaxTiles) return FRNN_ERR_SHAPE;  // (sLSTM from head dim 960 up has no 16-row reverse loop)
  const WsLayout w = workspace_layout(*pr, cd, reverse_units(pl));
  pl.workspace_bytes = w.total;
  pl.grads_offset = w.grads;
  pl.grads_count = (uint64_t)cd.Gr * pr->N * pr->D * pr->D + (uint64_t)cd.Gt * pr->N * pr->D;
  *out = pl;
  return FRNN_OK;
}

static int check_plan(const frnn_plan* pl, CellDims* cd) {
  if (!pl) return FRNN_ERR_NULL;
  if (pl->abi_version != FRNN_ABI_VERSION) return FRNN_ERR_PLAN;
  const int rc = validate_problem(&pl->prob, cd);
  if (rc) return rc;
  if (!tile_ok(pl->prob, *cd, pl->cluster_size, pl->batch_tile)) return FRNN_ERR_PLAN;
  if (pl->units_per_cta * pl->cluster_size != pl->prob.D) return FRNN_ERR_PLAN;
  if (pl->threads != plan_threads(*cd, pl->units_per_cta, pl->batch_tile)) return FRNN_ERR_PLAN;
  if (pl->forced_tile != 0 && pl->forced_tile != 1) return FRNN_ERR_PLAN;
  if (pl->workspace_bytes != workspace_layout(pl->prob, *cd, reverse_units(*pl)).total) return FRNN_ERR_PLAN;
  if (pl->wide_forward && !(pl->wide_forward == 1 && wide_gates_problem(pl->prob) && pl->cluster_size == 1 && pl->batch_tile == 16))
    return FRNN_ERR_PLAN;
  return FRNN_OK;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Strides of a caller-produced tensor: all zero = dense (the defaults are filled in), else each a non-negative
// multiple of 8 elements (16 bytes: what the 4/8-byte cp.async reads and the tensor maps need).
static bool resolve_strides(const int64_t (&in)[4], const long long (&dense)[4], long long (&out)[4]) {
  if (!in[0] && !in[1] && !in[2] && !in[3]) {
    for (int i = 0; i < 4; ++i) out[i] = dense[i];
    return true;
  }
  for (int i = 0; i < 4; ++i) {
    if (in[i] < 0 || in[i] % 8) return false;
    out[i] = in[i];
  }
  return true;
}

// `overlap`: a decoding step behind another may start, and read R, while that one still runs (everything else waits for it on the device):
// launch and prologue, about half of a one-token step, disappear behind the step before
static int launch_loop(const frnn_plan& pl, bool bwd, LoopParams lp, cudaStream_t stream) {
  const LoopLaunch k = loop_of(pl, bwd);
  if (!k.fn) return FRNN_ERR_PLAN;
  const bool overlap = !bwd && pl.keep_packed_r;
  lp.CS = k.cs;
  // always the fixed maximum, never this plan's own size: the attribute belongs to the kernel, not to the launch, and a
  // second host thread launching the same instantiation with a larger tile must not find it lowered in between
  cudaError_t e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDynSmem);
  if (e != cudaSuccess) return (int)e;
  if (k.cs > 8) {  // clusters of more than 8 CTAs are a non-portable size: opt in
    e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return (int)e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = loop_grid(k, pl.prob);
  cfg.blockDim = dim3((unsigned)k.threads, 1, 1);
  cfg.dynamicSmemBytes = k.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned na = 0;
  if (k.cs > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = (unsigned)k.cs;
    attr[na].val.clusterDim.y = 1;
    attr[na++].val.clusterDim.z = 1;
  }
  if (overlap) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  void* args[1] = {&lp};
  return (int)cudaLaunchKernelExC(&cfg, k.fn, args);
}

static int sm_count_cached() {
  static std::mutex mu;
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev] == 0) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    cached[dev] = v;
  }
  return cached[dev];
}

}  // namespace FRNN_NS

using namespace FRNN_NS;

// This file is compiled twice (see frnn_elem.cuh).  The bfloat16 build owns the public names and forwards float16
// problems to the float16 build, whose entry points carry the suffix _f16 and stay private to the library.
#ifdef FRNN_F16
#define FRNN_ENTRY(name) __attribute__((visibility("hidden"))) name##_f16
#define FRNN_FORWARD_F16(is_f16, call)
#else
#define FRNN_ENTRY(name) name
#define FRNN_FORWARD_F16(is_f16, call) \
  if (is_f16) return call
extern "C" {
int frnn_query_f16(const frnn_problem*, frnn_plan*);
int frnn_query_tile_f16(const frnn_problem*, int, int, int, frnn_plan*);
int frnn_query_loop_f16(const frnn_plan*, int, frnn_loop_shape*);
int frnn_query_dr_f16(const frnn_plan*, int32_t*, int32_t*);
int frnn_forward_f16(const frnn_plan*, const frnn_fwd_args*, void*);
int frnn_backward_parts_f16(const frnn_plan*, const frnn_bwd_args*, void*, int);
int frnn_finalize_grads_f16(const frnn_plan*, const void*, void*, void*, void*);
}
#endif
// float32 problems (Wx, R, b, states and gradients all fp32) go to the float32 loops of frnn_f32.cu
#ifdef FRNN_F16
#define FRNN_FORWARD_F32(is_f32, call)
#else
#define FRNN_FORWARD_F32(is_f32, call) \
  if (is_f32) return call
extern "C" {
int frnn_query_f32(const frnn_problem*, int, int, int, frnn_plan*);
int frnn_query_loop_f32(const frnn_plan*, int, frnn_loop_shape*);
int frnn_forward_f32(const frnn_plan*, const frnn_fwd_args*, void*);
int frnn_backward_parts_f32(const frnn_plan*, const frnn_bwd_args*, void*, int);
int frnn_finalize_grads_f32(const frnn_plan*, const void*, void*, void*, void*);
}
#endif
static inline bool wants_f32(const frnn_problem* pr) { return pr && pr->dtype_io == FRNN_DTYPE_F32; }
static inline bool wants_f32(const frnn_plan* pl) { return pl && pl->prob.dtype_io == FRNN_DTYPE_F32; }
static inline bool wants_f16(const frnn_problem* pr) { return pr && pr->dtype_io == FRNN_DTYPE_F16; }
static inline bool wants_f16(const frnn_plan* pl) { return pl && pl->prob.dtype_io == FRNN_DTYPE_F16; }

extern "C" {

#ifndef FRNN_F16
int frnn_abi_version(void) { return FRNN_ABI_VERSION; }
#endif

int FRNN_ENTRY(frnn_query)(const frnn_problem* problem, frnn_plan* out) {
  FRNN_FORWARD_F32(wants_f32(problem), frnn_query_f32(problem, 0, 0, 0, out));
  FRNN_FORWARD_F16(wants_f16(problem), frnn_query_f16(problem, out));
  return fill_plan(problem, 0, 0, 0, out);
}

int FRNN_ENTRY(frnn_query_tile)(const frnn_problem* problem, int cluster_size, int batch_tile, int wx_stages, frnn_plan* out) {
  FRNN_FORWARD_F32(wants_f32(problem), frnn_query_f32(problem, cluster_size, batch_tile, wx_stages, out));
  FRNN_FORWARD_F16(wants_f16(problem), frnn_query_tile_f16(problem, cluster_size, batch_tile, wx_stages, out));
  return fill_plan(problem, cluster_size, batch_tile, wx_stages, out);
}

int FRNN_ENTRY(frnn_query_loop)(const frnn_plan* plan, int backward, frnn_loop_shape* out) {
  FRNN_FORWARD_F32(wants_f32(plan), frnn_query_loop_f32(plan, backward, out));
  FRNN_FORWARD_F16(wants_f16(plan), frnn_query_loop_f16(plan, backward, out));
  CellDims cd;
  const int rc = check_plan(plan, &cd);
  if (rc) return rc;
  if (!out) return FRNN_ERR_NULL;
  const frnn_problem& pr = plan->prob;
  if (backward && !pr.training) return FRNN_ERR_TRAINING;
  if (is_wide(*plan) || (!backward && runs_wide_gates(*plan))) {
    const uint32_t tiles = (uint32_t)((pr.B + kWideBatchTile - 1) / kWideBatchTile);
    *out = {FRNN_LOOP_WIDE, 1, pr.D, kWideBatchTile, is_wide(*plan) ? kWideThreads : kWideGatesThreads,
            !is_wide(*plan) ? kWideGatesStages : backward ? kWideBwdStages : kWideFwdStages, {tiles, (uint32_t)pr.N, 1}};
    return FRNN_OK;
  }
  const LoopLaunch k = loop_of(*plan, backward != 0);
  if (!k.fn) return FRNN_ERR_PLAN;
  const dim3 g = loop_grid(k, pr);
  *out = {is_big(pr) ? FRNN_LOOP_BIG : FRNN_LOOP_LANE, k.cs, k.u, k.rows, k.threads - (k.dr ? kDrThreads : 0), k.stages, {g.x, g.y, g.z}};
  return FRNN_OK;
}

int FRNN_ENTRY(frnn_query_dr)(const frnn_plan* plan, int32_t* in_loop, int32_t* threads_on_top) {
  FRNN_FORWARD_F16(wants_f16(plan), frnn_query_dr_f16(plan, in_loop, threads_on_top));
  frnn_loop_shape s;
  const int rc = frnn_query_loop(plan, 1, &s);
  if (rc) return rc;
  if (!in_loop || !threads_on_top) return FRNN_ERR_NULL;
  const bool lane = s.loop == FRNN_LOOP_LANE && loop_of(*plan, true).dr;
  *in_loop = lane || s.loop == FRNN_LOOP_WIDE;
  *threads_on_top = lane ? kDrThreads : 0;
  return FRNN_OK;
}

int FRNN_ENTRY(frnn_forward)(const frnn_plan* plan, const frnn_fwd_args* a, void* stream_) {
  FRNN_FORWARD_F32(wants_f32(plan), frnn_forward_f32(plan, a, stream_));
  FRNN_FORWARD_F16(wants_f16(plan), frnn_forward_f16(plan, a, stream_));
  CellDims cd;
  int rc = check_plan(plan, &cd);
  if (rc) return rc;
  if (!a || !a->Wx || !a->R || !a->b || !a->s0 || !a->states || !a->workspace) return FRNN_ERR_NULL;
  const frnn_problem& pr = plan->prob;
  if (pr.training && cache_slots_of(pr, cd) > 0 && !a->cache) return FRNN_ERR_NULL;
  if (!aligned16(a->Wx) || !aligned16(a->R) || !aligned16(a->b) || !aligned16(a->s0) || !aligned16(a->states) ||
      !aligned16(a->workspace) || (a->cache && !aligned16(a->cache)))
    return FRNN_ERR_ALIGN;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const WsLayout w = workspace_layout(pr, cd, reverse_units(*plan));
  unsigned char* ws = static_cast<unsigned char*>(a->workspace);
  const long long nd = (long long)pr.N * pr.D;
  const long long wx_dense[4] = {(long long)pr.T * cd.Gw * nd, cd.Gw * nd, nd, pr.D};
  long long wxs[4];
  if (!resolve_strides(a->wx_stride, wx_dense, wxs)) return FRNN_ERR_ALIGN;

  const bool wide_gates = runs_wide_gates(*plan), wide = is_wide(*plan) || wide_gates;
  // keep_packed_r: the workspace is left as the previous call left it (R fragments kept, status block not cleared, so
  // an expired wait of an earlier step stays on record until the caller reads it).  The other loops clear the block themselves.
  cudaError_t e = plan->keep_packed_r || !wide ? cudaSuccess : cudaMemsetAsync(ws, 0, kStatusBytes, stream);
  if (e != cudaSuccess) return (int)e;
  if (a->last && !aligned16(a->last)) return FRNN_ERR_ALIGN;
  // `last`: one strided device copy of states[:, :, T-1] behind the 128-row loops; the others store it
  auto copy_last = [&]() -> cudaError_t {
    if (!a->last) return cudaSuccess;
    const size_t row = (size_t)pr.N * pr.D * (pr.dtype_state == FRNN_DTYPE_F32 ? 4 : 2);
    return cudaMemcpy2DAsync(a->last, row, static_cast<const unsigned char*>(a->states) + (size_t)(pr.T - 1) * row,
                             (size_t)pr.T * row, row, (size_t)cd.S * pr.B, cudaMemcpyDeviceToDevice, stream);
  };
  if (is_wide(*plan)) {
    if (plan->probe_noop_cell) return FRNN_ERR_PLAN;
    e = launch_wide_forward(a->Wx, wxs[0], wxs[1], wxs[3], a->R, a->b, a->s0, a->states, reinterpret_cast<unsigned*>(ws), pr.B,
                            pr.T, pr.N, plan->test_drop_exchange, stream);
    return (int)(e == cudaSuccess ? copy_last() : e);
  }
  if (wide_gates) {  // LSTM / GRU, head dim 64: 128-row forward loop
    if (plan->probe_noop_cell) return FRNN_ERR_PLAN;
    e = launch_wide_gates_forward(pr.cell, a->Wx, wxs[0], wxs[1], wxs[2], wxs[3], a->R, a->b, a->s0, a->states,
                                 reinterpret_cast<unsigned*>(ws), pr.B, pr.T, pr.N, pr.forward_clip, plan->test_drop_exchange, stream);
    return (int)(e == cudaSuccess ? copy_last() : e);
  }
  if (is_big(pr) && !plan->keep_packed_r) e = big_pack(kernel_cell(pr), a->R, ws + w.rpack_fwd, pr.N, pr.D, stream);
  if (e != cudaSuccess) return (int)e;

  LoopParams lp = {};
  lp.Wx = static_cast<const elem_t*>(a->Wx);
  lp.R = static_cast<const elem_t*>(a->R);
  lp.last = a->last;
  lp.clear_status = !plan->keep_packed_r;
  lp.Rpack = reinterpret_cast<const uint4*>(ws + w.rpack_fwd);
  lp.bias = static_cast<const elem_t*>(a->b);
  lp.s0 = a->s0;
  lp.states = a->states;
  lp.cache = pr.training ? static_cast<elem_t*>(a->cache) : nullptr;
  lp.status = reinterpret_cast<unsigned*>(ws);
  lp.B = pr.B; lp.T = pr.T; lp.N = pr.N; lp.D = pr.D;
  lp.state_f32 = pr.dtype_state == FRNN_DTYPE_F32;
  lp.fclip = pr.forward_clip; lp.gclip = pr.grad_clip; lp.grad_cut = pr.grad_cut;
  lp.test_drop = plan->test_drop_exchange;
  lp.wx_sb = wxs[0]; lp.wx_st = wxs[1]; lp.wx_sg = wxs[2]; lp.wx_sn = wxs[3];
  return launch_loop(*plan, false, lp, stream);
}

#ifndef FRNN_F16
int frnn_backward(const frnn_plan* plan, const frnn_bwd_args* a, void* stream_) {
  return frnn_backward_parts(plan, a, stream_, FRNN_PART_LOOP | FRNN_PART_DR);
}
#endif

int FRNN_ENTRY(frnn_backward_parts)(const frnn_plan* plan, const frnn_bwd_args* a, void* stream_, int parts) {
  FRNN_FORWARD_F32(wants_f32(plan), frnn_backward_parts_f32(plan, a, stream_, parts));
  FRNN_FORWARD_F16(wants_f16(plan), frnn_backward_parts_f16(plan, a, stream_, parts));
  CellDims cd;
  int rc = check_plan(plan, &cd);
  if (rc) return rc;
  const frnn_problem& pr = plan->prob;
  if (!pr.training) return FRNN_ERR_TRAINING;
  if (!a || !a->R || !a->s0 || !a->states || !a->dstates || !a->dWx || !a->ds0 || !a->workspace) return FRNN_ERR_NULL;
  if (cache_slots_of(pr, cd) > 0 && !a->cache) return FRNN_ERR_NULL;
  if (!aligned16(a->R) || !aligned16(a->s0) || !aligned16(a->states) || !aligned16(a->dstates) || !aligned16(a->dWx) ||
      !aligned16(a->ds0) || !aligned16(a->workspace) || (a->cache && !aligned16(a->cache)))
    return FRNN_ERR_ALIGN;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const WsLayout w = workspace_layout(pr, cd, reverse_units(*plan));
  unsigned char* ws = static_cast<unsigned char*>(a->workspace);
  float* grads = reinterpret_cast<float*>(ws + w.grads);
  const size_t nR = (size_t)cd.Gr * pr.N * pr.D * pr.D, nb = (size_t)cd.Gt * pr.N * pr.D;
  const long long nd = (long long)pr.N * pr.D;
  const long long ds_dense[4] = {(long long)pr.B * pr.T * nd, (long long)pr.T * nd, nd, pr.D};
  long long dss[4];
  if (!resolve_strides(a->dstates_stride, ds_dense, dss)) return FRNN_ERR_ALIGN;

  cudaError_t e = cudaSuccess;
  if ((parts & FRNN_PART_LOOP) && !is_wide(*plan)) {
    const bool big = is_big(pr);
    e = launch_bwd_prepare(a->R, ws + w.rpack_bwd, cd.Gr, pr.N, pr.D, reverse_units(*plan), big, grads, nR + nb,
                           reinterpret_cast<unsigned*>(ws), stream);
    if (e != cudaSuccess) return (int)e;
  } else if (parts & FRNN_PART_LOOP) {
    e = cudaMemsetAsync(ws, 0, kStatusBytes, stream);
    if (e != cudaSuccess) return (int)e;
    e = cudaMemsetAsync(grads, 0, (nR + nb) * sizeof(float), stream);
    if (e != cudaSuccess) return (int)e;
  }
  if (is_wide(*plan)) {  // one kernel: reverse loop with dR and db accumulated inside; the dR part has nothing left to do
    if (plan->probe_noop_cell) return FRNN_ERR_PLAN;
    if (parts & FRNN_PART_LOOP)
      e = launch_wide_backward(a->R, a->s0, a->states, a->dstates, dss[1], dss[2], dss[3], a->dWx, a->ds0, grads, grads + nR,
                               reinterpret_cast<unsigned*>(ws), pr.B, pr.T, pr.N, plan->test_drop_exchange, stream);
    return (int)e;
  }

  LoopParams lp = {};
  lp.Rpack = reinterpret_cast<const uint4*>(ws + w.rpack_bwd);
  lp.s0 = a->s0;
  lp.states = const_cast<void*>(a->states);
  lp.cache = static_cast<elem_t*>(const_cast<void*>(a->cache));
  lp.dstates = a->dstates;
  lp.dWx = static_cast<elem_t*>(a->dWx);
  lp.dg0 = reinterpret_cast<elem_t*>(ws + w.dg0);
  lp.ds0 = a->ds0;
  lp.dbias = grads + nR;
  lp.dR = grads;
  lp.status = reinterpret_cast<unsigned*>(ws);
  lp.B = pr.B; lp.T = pr.T; lp.N = pr.N; lp.D = pr.D;
  lp.state_f32 = pr.dtype_state == FRNN_DTYPE_F32;
  lp.fclip = pr.forward_clip; lp.gclip = pr.grad_clip; lp.grad_cut = pr.grad_cut;
  lp.test_drop = plan->test_drop_exchange;
  lp.ds_ss = dss[0]; lp.ds_sb = dss[1]; lp.ds_st = dss[2]; lp.ds_sn = dss[3];
  if (parts & FRNN_PART_LOOP) {
    rc = launch_loop(*plan, true, lp, stream);
    if (rc) return rc;
  }
  if (loop_of(*plan, true).dr) return FRNN_OK;  // nothing left to do for the dR part
  // dR.  Small heads: what counts is reading whole runs of neighbouring heads (frnn_dr_small.cu).  From head dim 128 up, 16-bit states: both
  // operands are [64 steps][64] tiles a tensor-map copy delivers ready for the MMA (LSTM B16 T1024 N4 D256 0.087 ms against 0.167 ms for the cp.async-fed
  // kernel; above 256, in column tiles, LSTM B16 T1024 N1 D768 0.445 -> 0.138 ms, against the warp-MMA kernel).  Above 256 the warp-MMA kernel is ahead
  //  * where less than half of a tile's 64 steps of one batch row would be used (Elman B342 T26 N5 D384 0.082 against 0.179 ms);
  //  * on few products: the tensor-map kernel takes 18 to 31 us however few they are, the other 6 us and 16 more per 1e9 products (LSTM N1 D320, 512, 2048,
  //    4096 rows 10, 16, 27 against 25, 21, 23 us; Elman N1 D512, 2048, 4096, 8000 rows 12, 19, 31 against 25, 23, 23; GRU N1 D768, 512, 1000 rows 16, 25 against 31, 23).
  // fp32 states: the cp.async-fed tcgen05 kernel while a row tile of dR, D columns, fits one TMEM allocation, the warp-MMA kernel above.
  const bool tma_pays = pr.D <= 256 || (2 * pr.T >= (pr.T + 63) / 64 * 64 && (double)nR * pr.B * pr.T >= 1.2e9);
  if ((parts & FRNN_PART_DR) && recurrent_grad_small_supported(pr.D))
    e = launch_recurrent_grad_small(pr.B, pr.T, pr.N, pr.D, cd.Gr, cd.Gw, lp.state_f32, a->dWx, ws + w.dg0, a->states, a->s0, grads,
                                    sm_count_cached(), stream);
  else if ((parts & FRNN_PART_DR) && recurrent_grad_tma_supported(pr.D, lp.state_f32) && tma_pays)
    e = launch_recurrent_grad_tma(pr.cell, pr.B, pr.T, pr.N, pr.D, cd.Gr, cd.Gw, a->dWx, ws + w.dg0, a->states, a->s0, grads,
                                  reinterpret_cast<unsigned*>(ws), plan->test_drop_exchange, sm_count_cached(), stream);
  else if ((parts & FRNN_PART_DR) && pr.D <= 256)
    e = launch_recurrent_grad_tc(pr.cell, pr.B, pr.T, pr.N, pr.D, cd.Gr, cd.Gw, lp.state_f32, a->dWx, ws + w.dg0, a->states,
                                 a->s0, grads, reinterpret_cast<unsigned*>(ws), sm_count_cached(), stream);
  else if (parts & FRNN_PART_DR)
    e = launch_recurrent_grad(pr.cell, pr.B, pr.T, pr.N, pr.D, cd.Gr, cd.Gw, lp.state_f32, a->dWx, ws + w.dg0, a->states,
                            a->s0, grads, sm_count_cached(), stream);
  return (int)e;
}

int FRNN_ENTRY(frnn_finalize_grads)(const frnn_plan* plan, const void* grads_f32, void* dR, void* db, void* stream_) {
  FRNN_FORWARD_F32(wants_f32(plan), frnn_finalize_grads_f32(plan, grads_f32, dR, db, stream_));
  FRNN_FORWARD_F16(wants_f16(plan), frnn_finalize_grads_f16(plan, grads_f32, dR, db, stream_));
  CellDims cd;
  int rc = check_plan(plan, &cd);
  if (rc) return rc;
  if (!grads_f32 || !dR || !db) return FRNN_ERR_NULL;
  const frnn_problem& pr = plan->prob;
  const size_t nR = (size_t)cd.Gr * pr.N * pr.D * pr.D, nb = (size_t)cd.Gt * pr.N * pr.D;
  return (int)launch_cast_grads(static_cast<const float*>(grads_f32), dR, db, nR, nb, static_cast<cudaStream_t>(stream_));
}

#ifndef FRNN_F16
int frnn_read_device_status(const void* workspace, void* stream_, frnn_dev_status* out) {
  if (!workspace || !out) return FRNN_ERR_NULL;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  cudaError_t e = cudaMemcpyAsync(out, workspace, sizeof(frnn_dev_status), cudaMemcpyDeviceToHost, stream);
  if (e != cudaSuccess) return (int)e;
  return (int)cudaStreamSynchronize(stream);
}

const char* frnn_status_string(int code) {
  switch (code) {
    case FRNN_OK: return "ok";
    case FRNN_ERR_NULL: return "frnn: a required pointer is NULL";
    case FRNN_ERR_CELL: return "frnn: unknown cell (expected lstm, gru, elman or slstm)";
    case FRNN_ERR_SHAPE: return "frnn: unsupported shape (B,T,N >= 1; head_dim in {16,32,64,96,128,192,256} or a multiple of 64 up to 1024; float32: a multiple of 4 up to 1024)";
    case FRNN_ERR_DTYPE: return "frnn: unsupported dtype (Wx/R/b bfloat16 or float16 with states of the same type or float32; or everything float32)";
    case FRNN_ERR_ALIGN: return "frnn: tensor pointers must be 16-byte aligned";
    case FRNN_ERR_PLAN: return "frnn: invalid plan or tile for this problem";
    case FRNN_ERR_TRAINING: return "frnn: backward needs a plan made with training = 1";
    case FRNN_ERR_DEVICE: return "frnn: no sm_100 device / kernel image";
    case FRNN_ERR_TOO_LARGE: return "frnn: size beyond the fixed limit of this entry point";
    default: break;
  }
  if (code > 0) return cudaGetErrorString(static_cast<cudaError_t>(code));
  return "frnn: unknown status";
}
#endif

}  // extern "C"
