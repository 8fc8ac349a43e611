// The few-rows kernel's plan and entry points (the kernel itself: qmm_rows.cuh; its instantiations: qmm_rows_*.cu).
#include "qmm_rows.cuh"

#include <algorithm>

namespace qmm {

using namespace rows;

namespace rows {
#define QMM_ROWS_EXTERN(QK, XT) \
  extern template int launch_rows_kernel<QK, XT>(const CUtensorMap&, const CUtensorMap&, RowsParams&, RowsPlan&, const RowsShape&, bool, cudaStream_t);
QMM_ROWS_EXTERN(kAff4, __nv_bfloat16)
QMM_ROWS_EXTERN(kAff4, __half)
QMM_ROWS_EXTERN(kAff4, float)
QMM_ROWS_EXTERN(kAff8, __nv_bfloat16)
QMM_ROWS_EXTERN(kAff8, __half)
QMM_ROWS_EXTERN(kAff8, float)
QMM_ROWS_EXTERN(kMx4, __nv_bfloat16)
QMM_ROWS_EXTERN(kMx4, __half)
QMM_ROWS_EXTERN(kMx4, float)
}  // namespace rows

namespace {

size_t smem_of(const RowsPlan& pl, const RowsShape& sh, int segs) {
  const int qk = sh.tt == kTabE8 ? kMx4 : sh.stage == kBlockRows * kSliceK ? kAff8 : kAff4;
  const bool quads = table_quads(sh.groups, sh.tt), twice = sums_twice(qk, sh.groups, sh.tt, sh.exact || sh.tokens == 4);
  auto own = [&](bool q, bool t) { return pl.ring * (pl.blocks * sh.stage + table_stage_bytes(pl.blocks, sh.groups, sh.tt, q)) + sums_bytes(sh.groups, t); };
  // (at least what the plainest layout takes: a few hundred bytes decide between plans whose costs are close, and the costs were fitted with these)
  const size_t shares = static_cast<size_t>(pl.blocks) * 512, warp = std::max(own(quads, twice), own(false, false));
  return 1024 + kHeadBytes + static_cast<size_t>(pl.warps) * (warp + pl.red_bufs * shares + more_x_bytes(sh.tokens)) +
         (pl.cluster > 1 ? kExchangeSlots * pl.cluster * shares : 0) + (segs ? (2 * static_cast<size_t>(segs) + 1) * 4 : 0);
}

// How K and the tiles are shared out: the plan of the least load. The load stands for the time of the busiest SM, in slices of 32
// rows that one warp works through: tiles per cluster x warps resident on the SM (at least 6: fewer leave it waiting for memory) x
// what a tile costs a warp -- its slices (half as much where a tile is one block of 16 rows), plus what it costs besides its codes,
// half a slice for 32 rows and 0.35 for 16 (barriers and addresses are per tile, not per row), 0.05 more in a cluster -- and 4 for the
// cluster's meeting at the start and the end. More CTAs per tile (a larger cluster) is what keeps K within 8 warps x 512 codes of
// registers when K is long, and what fills the machine when a weight has few tiles; more than one slice per warp reloads the
// activations with every tile and is left for where nothing else fits. Tiles of one block cost more per row, but an SM that has one tile
// or two waits less for them (8 rows, mxfp4 5760 x 2880: 2.4 tiles of 16 rows per SM instead of 1.2 -> 2 of 32).
//
// Clusters of CTAs of one or two warps, three or four CTAs on an SM, cost more than the load says, and whether one of them came out ahead hung on the tables' bytes: 8 rows,
// float32 against MXFP4 28480 x 2048 49.9 us as 222 clusters of two, 31.4 as tiles of whole K; 2 rows 24512 x 4096 in groups of 32 26.0 / 17.2; 22464 x 7680 mxfp4 53.4 / 35.4.
// Of 56 shapes where such a plan had the least load none was the faster for it. (The order of float32 sums goes with the plan: 756 products of float32 activations are 1.003 times as far from float64
// as with such clusters, the farthest as far, 2.4e-7; those whose plan changed 1.01, of 0.91 to 1.14, at 5e-8.)
//
// The constants were fitted to measured times of an earlier form of the kernel; what they pick against the best of all plans, us back to back in a graph: 8 rows 28672 x 4096 17.2 / 17.2 (the
// next best 21.2), 128256 x 4096 58.2 / 58.2 (68.8), 4096 x 14336 14.1 / 14.1 (17.2), 4096 x 4096 5.9 / 5.8, 1024 x 1024 3.3 / 3.3,
// 16 rows 4096 x 4096 7.7 / 7.7 (8.5), 128256 x 4096 109 / 109 (138), 4 rows 5632 x 2048 4.7 / 4.7 (4.9), 2048 x 5632 7.0 / 7.0, 8-bit 8 rows 14336 x 4096 in groups of 64 13.5 / 13.5, of 128 13.5 / 13.1,
// 4096 x 14336 17.8 / 15.8, mxfp4 8 rows 5760 x 2880 8.4 / 8.4, float32 4 rows 4096 x 4096 9.2 / 9.2.
RowsPlan plan_rows(int64_t chunks, int64_t rows, int slices, const RowsShape& sh, int segs, bool pair = false) {
  const int sms = device_sm_count();
  RowsPlan best = {};
  for (int blocks = kMaxBlocks; blocks >= (sh.exact || pair ? kMaxBlocks : 1); --blocks) {
    const int tile_rows = pair ? kBlockRows : kBlockRows * blocks;
    const int64_t items = chunks * ((rows + tile_rows - 1) / tile_rows);
    for (int c = 1; c <= kMaxCluster; c *= 2) {
      if (c > slices && c > 1) break;
      RowsPlan pl = {};
      pl.blocks = blocks;
      pl.cluster = c;
      pl.slices_per_cta = (slices + c - 1) / c;
      pl.slices_per_warp = (pl.slices_per_cta + kMaxWarps - 1) / kMaxWarps;
      if (pl.slices_per_warp > 1 && c < kMaxCluster) continue;        // (reloading activations per tile: only where nothing else is left)
      pl.warps = (pl.slices_per_cta + pl.slices_per_warp - 1) / pl.slices_per_warp;
      pl.slices_per_cta = pl.warps * pl.slices_per_warp;
      if (c > 1 && pl.warps < 3) continue;                            // (see above)
      int per_sm = kMaxWarps / pl.warps;
      if (per_sm > 4) per_sm = 4;
      pl.ring = kMaxRing;
      pl.red_bufs = 4;
      const size_t budget = static_cast<size_t>(kSmemLimit) / per_sm - 1024;
      while (pl.red_bufs > 3 && smem_of(pl, sh, segs) > budget) --pl.red_bufs;
      while (pl.ring > 2 && smem_of(pl, sh, segs) > budget) --pl.ring;
      while (pl.ring > 1 && smem_of(pl, sh, segs) > static_cast<size_t>(kSmemLimit)) --pl.ring;
      pl.smem = smem_of(pl, sh, segs);
      if (pl.smem > static_cast<size_t>(kSmemLimit)) continue;
      while (per_sm > 1 && pl.smem > static_cast<size_t>(kSmemLimit) / per_sm - 1024) --per_sm;
      int64_t clusters = static_cast<int64_t>(sms) * per_sm / c;
      if (clusters > items) clusters = items;
      if (clusters < 1) clusters = 1;
      pl.grid = static_cast<int>(clusters * c);
      const int64_t tiles = (items + clusters - 1) / clusters;
      const int64_t resident = (clusters * c + sms - 1) / sms;
      const int64_t busy = resident * pl.warps > 6 ? resident * pl.warps : 6;      // (fewer warps leave an SM waiting)
      const double tile = blocks == 2 ? pl.slices_per_warp + (c > 1 ? 0.55 : 0.5) : 0.5 * pl.slices_per_warp + (c > 1 ? 0.4 : 0.35);
      double load = static_cast<double>(tiles) * busy * tile + (c > 1 ? 4.0 : 0.0);
      if (pl.ring == 1) load *= 100.0;               // (nothing is loaded while a box is worked on: where nothing else fits)
      pl.load = load;
      if (!best.warps || load < best.load) best = pl;
    }
  }
  return best;
}

// Rows of a chunk are what the registers take. Nine to sixteen rows are two chunks: the CTAs that work on either half pass over
// the weight side by side, so that the second reads it from L2 (16 rows of 4096 x 4096: 7.7 us; as one chunk of 16, half of whose activations
// live in shared memory, 14.2 when this was 9.2).
RowsShape shape_of(const qmm_problem& p, bool exact) {
  const bool mx = p.mode == QMM_MODE_MXFP4;
  const int bits = (!mx && p.bits == 8) ? 8 : 4, group = mx ? 32 : p.group_size;
  return {p.x_dtype == QMM_F32 ? 4 : 8, kSliceK / group, mx ? kTabE8 : (p.table_dtype == QMM_BF16 ? kTabBf16 : (p.table_dtype == QMM_F16 ? kTabF16 : kTabF32)),
          kBlockRows * kSliceK * bits / 8, exact && !mx && p.x_dtype != QMM_F32};
}

}  // namespace

double rows_estimate(const qmm_problem& p) {
  const RowsShape sh = shape_of(p, true);
  const double load = plan_rows((p.M + sh.tokens - 1) / sh.tokens, p.N, static_cast<int>((p.K + kSliceK - 1) / kSliceK), sh, 0).load;
  return 5.3 + load * (sh.groups == 16 ? 0.41 : sh.groups == 8 ? 0.38 : 0.34);
}

bool rows_supports(const qmm_problem& p) {
  if (p.mode == QMM_MODE_FLOAT || p.K < 32 || p.K % 32 || p.K >= (1LL << 30) || p.N < 1 || p.M < 1 || p.batch < 1) return false;
  if (p.M >= (1LL << 31) || p.batch >= (1LL << 31)) return false;
  if (p.group_sizes && p.batch > kMaxSegments) return false;
  const int64_t nw = p.num_weights > 0 ? p.num_weights : (p.w_batch_stride ? p.batch : 1);
  if (p.batch * ((p.M + 3) / 4) * ((p.N + 15) / 16) >= (1LL << 31)) return false;       // items are counted in 32 bits
  return nw * p.N < (1LL << 31);                    // TMA row coordinates are 32-bit
}

// A grouped product of at most 8 rows per expert on average streams its experts' weights here: an even share is one pass of a weight, and what
// routing makes uneven still costs less than the tensor-core kernel's 64-row tiles. Above it those win, even shares or not. Experts' shares are
// only known on the device, and a share of n rows passes its weight ceil(n / 8) times: the worst, all rows on one expert, is dearer here from 3 rows an
// expert on. us here / tensor cores (back to back in a graph, weights from HBM), even, random and all on one:
//   rows an expert            4                                    8                                     12
//   4-bit  8 x 14336 x 4096   56/88    56/88    30/17              56/88     68/88   54/17               103/89   103/89    78/30
//   4-bit  8 x 4096 x 14336   71/82    71/82    39/42              72/81     87/82   69/42               133/82   132/82   101/42
//   4-bit 32 x 2048 x 2048    22/37    22/37    13/14              22/37     27/37   20/14                36/37    34/37    28/15
//   mxfp4 32 x 2880 x 2880    69/64    74/64    35/18              69/64     90/64   67/19               127/64   121/64    95/19
//   8-bit  8 x 4096 x 4096    29/37    29/37    17/19              30/37     32/37   26/19                45/37    46/37    34/19
// (MXFP4 would be as fast or faster there from few rows on, since that kernel looks its values up; it rounds each weight to 16 bits, this one none.)
bool rows_grouped_pays(const qmm_problem& p) { return rows_supports(p) && p.M <= 8 * p.batch; }

// The decode family as callers may force it: dense or gathered products of up to 16 rows of 16-bit activations.
bool gemv_supports(const qmm_problem& p) {
  return (p.x_dtype == QMM_BF16 || p.x_dtype == QMM_F16) && !p.group_sizes && p.M <= 16 && p.batch <= 65535 && rows_supports(p);
}

namespace {

// The plan of a problem (grouped: of an even share of its rows for every expert).
RowsPlan plan_of(const qmm_problem& p, const RowsShape& sh, bool pair) {
  const int64_t per_seg = p.group_sizes ? (p.M + p.batch - 1) / p.batch : p.M, live = p.group_sizes ? (p.batch < p.M ? p.batch : p.M) : p.batch;
  return plan_rows(live * ((per_seg + sh.tokens - 1) / sh.tokens), p.N, static_cast<int>((p.K + kSliceK - 1) / kSliceK), sh, p.group_sizes ? static_cast<int>(p.batch) : 0, pair);
}

}  // namespace

bool rows_plan(const qmm_problem& p, bool exact, bool pair, int32_t plan[5]) {
  const RowsPlan pl = plan_of(p, shape_of(p, exact), pair);
  const int32_t of[5] = {pl.blocks, pl.cluster, pl.warps, pl.ring, pl.grid};
  for (int i = 0; i < 5; ++i) plan[i] = of[i];
  return pl.warps != 0;
}

int launch_rows(const qmm_problem& p, cudaStream_t stream, const RowsGather* gather, bool exact, const RowsPair* pair) {
  RowsParams rp = {};
  rp.x = p.x; rp.scales = p.scales; rp.biases = p.biases; rp.y = p.y;
  rp.lhs_idx = p.lhs_idx; rp.rhs_idx = p.rhs_idx; rp.group_sizes = p.group_sizes;
  if (pair) {
    rp.scales2 = pair->scales;
    rp.biases2 = pair->biases;
  }
  if (gather) {
    rp.x_rows = gather->x_rows;
    rp.total_x_rows = gather->total_x_rows;
  }
  rp.status = device_status_word();
  if (!rp.status) return fail(QMM_ERR_CUDA, "could not allocate the device status word");
  const bool mx = p.mode == QMM_MODE_MXFP4;
  const int bits = (!mx && p.bits == 8) ? 8 : 4;
  const int group = mx ? 32 : p.group_size;
  rp.x_batch_stride = p.x_batch_stride; rp.y_batch_stride = p.y_batch_stride;
  rp.num_weights = p.num_weights > 0 ? p.num_weights : 1;
  rp.x_batches = p.x_batches;
  rp.M = p.M; rp.K = static_cast<int>(p.K); rp.N = static_cast<int>(p.N); rp.segs = static_cast<int>(p.batch);
  rp.groups = rp.K / group;
  rp.weight_rows = (p.rhs_idx || p.group_sizes || p.w_batch_stride) ? rp.N : 0;
  rp.table_dtype = p.table_dtype; rp.y_dtype = p.y_dtype;
  const RowsShape sh = shape_of(p, exact);
  const int chunk = sh.tokens;
  const int entry = mx ? 1 : (p.table_dtype == QMM_F32 ? 4 : 2);
  const int64_t nweights = p.num_weights > 0 ? p.num_weights : (p.w_batch_stride ? p.batch : 1);
  rp.table_bytes = nweights * p.N * rp.groups * entry;
  // (a slice's entries start on the units that its own row of entries and a row of the table are multiples of)
  const int slice_bytes = sh.groups * entry, row_bytes_t = rp.groups * entry;
  rp.table_unit = (row_bytes_t | slice_bytes) % 8 == 0 && row_bytes_t % slice_bytes == 0 ? (slice_bytes % 16 == 0 ? 16 : 8) : (row_bytes_t | slice_bytes) % 4 == 0 ? 4 : 1;
  RowsPlan pl = plan_of(p, sh, pair != nullptr);
  if (!pl.warps) return fail(QMM_ERR_UNSUPPORTED, "few-rows kernel: no plan fits shared memory");
  const int tile_rows = pair ? kBlockRows : kBlockRows * pl.blocks;
  rp.tiles = (rp.N + tile_rows - 1) / tile_rows;
  pl.items = p.batch * ((p.M + chunk - 1) / chunk) * rp.tiles;
  rp.cluster = pl.cluster; rp.slices_per_cta = pl.slices_per_cta; rp.slices_per_warp = pl.slices_per_warp;
  rp.ring = pl.ring; rp.red_bufs = pl.red_bufs;

  // The packed weight as a 2-D byte tensor [rows, K*bits/8] over every weight matrix behind `w`; what a box
  // reaches past the last row or the end of a row is zero-filled by the TMA unit.
  const uint64_t row_bytes = static_cast<uint64_t>(p.K) * bits / 8;
  CUtensorMap wm;
  const int rc = tensor_map_2d(&wm, QMM_U8, p.w, row_bytes, static_cast<uint64_t>(p.N) * nweights, row_bytes, kBoxBytes, tile_rows, 1);
  if (rc) return rc;
  CUtensorMap wm2 = wm;
  if (pair) {
    const int rc2 = tensor_map_2d(&wm2, QMM_U8, pair->w, row_bytes, static_cast<uint64_t>(p.N) * nweights, row_bytes, kBoxBytes, tile_rows, 1);
    if (rc2) return rc2;
  }
  // A gather's indices decide which weight the first boxes come from: it is serialized in the ordinary way.
  const bool early = !p.lhs_idx;
  auto launch = [&](auto kind) {
    constexpr int QK = decltype(kind)::value;
    if (p.x_dtype == QMM_BF16) return launch_rows_kernel<QK, __nv_bfloat16>(wm, wm2, rp, pl, sh, early, stream);
    if (p.x_dtype == QMM_F16) return launch_rows_kernel<QK, __half>(wm, wm2, rp, pl, sh, early, stream);
    return launch_rows_kernel<QK, float>(wm, wm2, rp, pl, sh, early, stream);
  };
  if (mx) return launch(std::integral_constant<int, kMx4>());
  if (bits == 8) return launch(std::integral_constant<int, kAff8>());
  return launch(std::integral_constant<int, kAff4>());
}

namespace {

bool pair_takes(const qmm_problem& p) { return (p.x_dtype == QMM_BF16 || p.x_dtype == QMM_F16) && p.y_dtype == p.x_dtype && !p.lhs_idx && rows_supports(p); }

}  // namespace

// (tiles of two blocks alone: 8-bit codes with the widest tables, the longest K and a thousand experts leave no room for them)
bool rows_pair_supports(const qmm_problem& p) { return pair_takes(p) && plan_of(p, shape_of(p, false), true).warps != 0; }

// 4-bit codes have the same tiles either way: one launch took 0.64 of the time of two products and the gate on average of 39 shapes (MXFP4 0.70 of 44, but 14016 x 7296 101 us against
// 92); dense ones always have a plan, and are not asked for it. Of 8-bit codes tiles of two blocks, 16 rows of each weight, leave two slots of a ring or half the warps, and then two products
// in plans of their own are the faster. By the plans' loads (one is some 0.35 us): expert blocks, us as one launch / two, by what one has more than twice the other: 16 of 8 experts 2816 -> 8576
// 1.00 93 / 101, 14 of 32 3328 -> 4736 1.57 189 / 153, 2 of 16 2688 -> 6528 1.89 78 / 58, 6 of 8 896 -> 5888 1.32 59 / 48. Dense ones save two launches, 18 of these units or less: 2 rows
// 1280 -> 11080 +14 11.8 / 14.3, 9 rows 3200 -> 3944 +22 30.3 / 25.4, 16 rows 2048 -> 13192 +26 26.4 / 28.8, 4 rows 3968 -> 14720 +30 37.4 / 32.7.
bool rows_pair_pays(const qmm_problem& p) {
  if (!pair_takes(p)) return false;
  const bool eight = p.mode != QMM_MODE_MXFP4 && p.bits == 8;
  if (!eight && !p.group_sizes) return true;
  const RowsShape sh = shape_of(p, false);
  const RowsPlan one = plan_of(p, sh, true);
  return one.warps && (!eight || one.load <= 2.0 * plan_of(p, sh, false).load + (p.group_sizes ? 0.0 : 18.0));
}

int launch_gemv(const qmm_problem& p, cudaStream_t stream) {
  if (route_override() != QMM_ROUTE_GEMV_FMMA && gemv_imma_supports(p)) return launch_gemv_imma(p, stream);
  return launch_rows(p, stream);
}

}  // namespace qmm
