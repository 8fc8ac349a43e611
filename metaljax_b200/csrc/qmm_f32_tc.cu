// Float32 activations of more than a few rows on the 5th-generation tensor cores (`y = x . deq(w)^T`, src/metaljax/qmm.py:2491,
// in the precision that keras keeps by default).
//
// Arithmetic, that of the few-rows kernel (qmm_rows.cuh) in another place: the codes are never dequantized. A code minus its centre (q - 8,
// q - 128, an E2M1 value) is exact in 16 bits, the MMA's A operand in tensor memory; a float32 activation is three pieces, the B operand: against 4-bit codes
// bf16 ones (8 + 8 + 8 bits), against 8-bit and MXFP4 ones f16 (11 + 11 + 11), for which each 512 codes of a row are brought to [2^14, 2^15) by
// their largest finite magnitude, and their sums back. Every group (of 8-bit codes, every 64) has accumulators of its own, two columns of tensor memory per row, one for the first piece and one for the
// others: a tensor core truncates each sum that it makes, and the small pieces' sums are small. They are read back, scaled and added up in
// float32 registers: y += s * sum (q - C) x, and, for a row whose four groups have biases of their own (b + C s is not nought), (b + C s) sum x.
// Range: activations up to 2^120 give finite results where those fit (against 8-bit codes as bf16 pieces, unscaled, a group's sum was infinite from 2^118 on, and below
// 2^-110 the pieces ran out of exponents: 4.5e-3 of the result's norm at 2^-126). 4-bit codes take those below 2^-110 with fewer than 24 bits.
//
// Split. K is shared out to the CTAs of a cluster (up to 8). A CTA converts its stretch of K of a chunk of 16, 32 or 48 activation rows once, into
// swizzled tiles that stay in shared memory; tiles of 128 weight rows pass by. The CTAs' partial tiles are pushed with st.async to the CTA that owns 128 / c of the
// tile's rows, which adds them up in rank order a tile late. No scratch, no atomics, fixed order of summation.
//
// What bounds it: the few-rows kernel takes four rows a pass over the weight, and takes the codes apart for each of them (33 rows: nine times). Here a pass
// takes up to 48. 33 rows of 4096 x 4096: 34.6 -> 24.5 us (13 K clocks a tile and cluster of eight: 8 K of them the codes, the MMAs' issue and the adding up, which
// are latency at 18 warps, the rest the exchange; 14 or 15 such clusters fit the machine); 64 rows of 14336 x 4096 178 -> 85, 4096 x 14336 234 -> 108.
// Relative error against float64 (1e-8, 2-norm; N(0, 1) / one sign / outliers of 300; 33 rows), few-rows kernel -> here: 4-bit groups of 64 K 4096 8.5 / 5.4 / 9.5 -> 7.3 /
// 4.2 / 8.3, K 14336 9.4 / 4.6 / 10.1 -> 8.6 / 4.3 / 9.4, of 128 K 4096 7.8 / 5.2 / 10.2 -> 6.8 / 4.2 / 9.4; 8-bit of 128 K 12288 13.4 / 12.5 / 20.4 -> 10.2 / 9.4 / 13.4; MXFP4
// K 4096 9.3 / 9.3 / 11.1 -> 7.8 / 7.8 / 9.3, K 14336 10.1 / 10.1 / 11.5 -> 9.8 / 9.9 / 10.9. (Ranks added up one after another and two sums to a group of 128: K 14336 9.1 / 5.0
// / 9.8, of 128 9.1 / 5.0 / 9.9, MXFP4 K 4096 9.7 / 9.7 / 10.0. All pieces in one accumulator: 9.4 / 6.4 / 9.7 at K 4096, and 24 in groups of 128.)
//
// Warps: 0 = weights' producer, 1 = MMA issuer (+ tensor memory), 2..9 = two teams that turn codes into A, 10..17 = adding up, half of the rows
// to each four. All of them convert the activations. A step is two K blocks: a wait costs a warp about as much as a third of a block's codes, and
// a warp by itself issues an instruction in some four clocks, so that there are many of either kind.
// Every wait on an mbarrier is bounded. Launched with programmatic stream serialization: before griddepcontrol.wait only the weights are touched.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "qmm_internal.h"
#include "qmm_ptx.cuh"
#include "qmm_tcgen05.cuh"

namespace qmm {
namespace {

using namespace ptx;
using namespace tc;

constexpr int kTileRows = 128;         // weight rows of a tile: lanes of tensor memory
constexpr int kBK = 64;                // K of a block: 32 columns of A
constexpr int kStepK = 2 * kBK;        // K of a step: a weight box, a slot of A
constexpr int kTeams = 2;
constexpr int kAddWarps = 8;
constexpr int kWarps = 2 + 4 * kTeams + kAddWarps;
constexpr int kThreads = kWarps * 32;
constexpr int kAddWarp = 2 + 4 * kTeams;
constexpr int box_bytes(int bits) { return kTileRows * kStepK * bits / 8; }
constexpr int kMaxBoxes = 8;
constexpr int kASlots = 4;             // steps of A in tensor memory
constexpr int kASlotsAt = 0, kDAt = kASlots * 64;
constexpr int d_slots(int t) { return t == 48 ? 2 : 4; }     // accumulators in tensor memory
constexpr int kMaxDSlots = 4;
constexpr int kMaxCluster = 8;
constexpr int kSmemLimit = 227 * 1024;
static_assert(kTeams <= kASlots, "a parity cannot tell a slot's use from the one two rounds before");

enum { kAff4 = 0, kAff8 = 1, kMx4 = 2 };

struct F32Params {
  const float* x;
  const void* scales;
  const void* biases;
  void* y;
  int* status;
  int64_t M, N;
  int K, groups, group_shift, table_dtype, y_dtype;
  int tiles, steps, most_steps;        // tiles of the weight; steps of K, and the most of them that a CTA has
  int cluster, slots, boxes;           // CTAs that share K; partial tiles on their way to an owner; places of the weights' ring
  unsigned most_inverse, less_inverse; // 2^32 / (16 steps) rounded up, of a CTA with most_steps and of one with a step less
  unsigned share, share_more;          // (chunk, tile) items of every cluster, and how many clusters have one more
};

// Shared memory from the 1024-byte aligned start: barriers, the activations [block][piece][T rows x 128 bytes], the weights' ring, the activations' sums over a group
// [4 steps][T], what the slices' sums are multiplied by [slice][T], the partial tiles [slot][128 rows][T + 4].
constexpr int kWFull = 0, kWEmpty = kWFull + 8 * kMaxBoxes, kAFull = kWEmpty + 8 * kMaxBoxes, kAEmpty = kAFull + 8 * kASlots, kDFull = kAEmpty + 8 * kASlots,
              kDEmpty = kDFull + 8 * kMaxDSlots, kXFull = kDEmpty + 8 * kMaxDSlots, kXFree = kXFull + 16, kTmemSlot = kXFree + 16, kAbort = kTmemSlot + 4, kHead = 1024;
static_assert(kAbort + 4 <= kHead, "");
constexpr int partial_row(int t) { return (t + 4) * 4; }
constexpr int partial_bytes(int t) { return kTileRows * partial_row(t); }
constexpr int x_block(int t) { return 3 * t * 128; }
constexpr int kSliceSteps = 4;         // 512 codes of a row are scaled together (48 rows: all of a CTA's, which are no more)
constexpr int most_slices(int t, int steps) { return t == 48 ? 1 : (steps + kSliceSteps - 2) / kSliceSteps + 1; }      // slices start at multiples of 512 codes
constexpr size_t smem_of(int t, int steps, int slots, int boxes, int bits) {
  return 1024 + kHead + boxes * box_bytes(bits) + static_cast<size_t>(steps) * (2 * x_block(t) + 4 * t * 4) + most_slices(t, steps) * t * 4 + static_cast<size_t>(slots) * partial_bytes(t);
}

// Packed words -> pairs of codes minus their centre (exact): bf16 (4-bit) or f16.
template <int QK>
__device__ __forceinline__ void codes16(const uint32_t (&w)[4], uint32_t* out) {
  if constexpr (QK == kAff4) {         // 32 codes, as (q - 8) / 64: a code in the low bits is the subnormal q 2^-133, one FMA with 2^127 and -1 / 8 takes it there (exactly)
    using H = Half2Ops<__nv_bfloat16>;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t even = w[j] & 0x0F0F0F0Fu, odd = (w[j] >> 4) & 0x0F0F0F0Fu;
#pragma unroll
      for (int i = 0; i < 4; ++i) out[j * 4 + i] = H::fma(permute(even, odd, i | ((8 + i) << 4) | ((4 + i) << 8) | ((12 + i) << 12)), 0x7F007F00u, 0xBE00BE00u);
    }
  } else if constexpr (QK == kAff8) {  // 16 codes: 1024 + q - 1152
    using H = Half2Ops<__half>;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      out[j * 2] = H::sub(__byte_perm(w[j], 0x64646464u, 0x4140u), 0x64806480u);
      out[j * 2 + 1] = H::sub(__byte_perm(w[j], 0x64646464u, 0x4342u), 0x64806480u);
    }
  } else {                             // 32 E2M1 codes: magnitude at the exponent's boundary is the value times 2^-14
    using H = Half2Ops<__half>;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t hi = w[j] >> 4;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t t = __byte_perm(w[j], hi, i | ((4 + i) << 8)) & 0x000F000Fu;
        out[j * 4 + i] = H::mul(((t & 0x00070007u) << 9) | ((t & 0x00080008u) << 12), 0x74007400u);      // 2^14
      }
    }
  }
}

__device__ __forceinline__ void fma2(float& y0, float& y1, float s, float a0, float a1) {
  asm("{ .reg .b64 y, s, a; mov.b64 y, {%0, %1}; mov.b64 s, {%2, %2}; mov.b64 a, {%3, %4}; fma.rn.f32x2 y, s, a, y; mov.b64 {%0, %1}, y; }"
      : "+f"(y0), "+f"(y1) : "f"(s), "f"(a0), "f"(a1));
}
// y0, y1 += s * (a + b), two at a time.
__device__ __forceinline__ void add_fma2(float& y0, float& y1, float s, const uint32_t* a, const uint32_t* b) {
  asm("{ .reg .b64 y, s, a, b; mov.b64 y, {%0, %1}; mov.b64 s, {%2, %2}; mov.b64 a, {%3, %4}; mov.b64 b, {%5, %6}; add.rn.f32x2 a, a, b; fma.rn.f32x2 y, s, a, y; mov.b64 {%0, %1}, y; }"
      : "+f"(y0), "+f"(y1) : "f"(s), "r"(a[0]), "r"(a[1]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void st_async4(uint32_t addr, uint32_t bar, float a, float b, float c, float d) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}

// QK: quantization kind. T: activation rows of a chunk. WIDE: float32 tables.
template <int QK, int T, bool WIDE>
__global__ void __launch_bounds__(kThreads, 1)
qmm_f32_tc_kernel(const __grid_constant__ CUtensorMap w_map, const F32Params p) {
  constexpr int kBits = QK == kAff8 ? 8 : 4;
  constexpr int kRowBytes = kBK * kBits / 8, kBoxBytes = 2 * kRowBytes, kBox = box_bytes(kBits);      // of a weight row in a block, in a box
  constexpr float kCentre = QK == kAff8 ? 128.0f : 8.0f, kUnit = QK == kAff4 ? 64.0f : 1.0f;     // (4-bit codes go in divided by 64)
  constexpr int kXBlock = x_block(T), kPiece = T * 128, kRow = partial_row(T), kDSlots = d_slots(T);
  constexpr bool kScaled = QK != kAff4;                // f16 pieces of scaled slices
  static_assert(kDAt + kDSlots * 2 * T <= 512 && T % 16 == 0, "");

  extern __shared__ uint8_t f32_smem_raw[];
  const uint32_t smem = (smem_u32(f32_smem_raw) + 1023) & ~1023u;
  const uint32_t x_at = smem + kHead, w_at = x_at + p.most_steps * 2 * kXBlock, sums_at = w_at + p.boxes * kBox, back_at = sums_at + p.most_steps * 4 * T * 4,
                 part_at = back_at + most_slices(T, p.most_steps) * T * 4;
  const uint32_t abort_at = smem + kAbort;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // (what the issuer's operands come from is the same in all lanes, and is made known as such: see tc_mma_block)
  auto same = [](int v) -> int { return __shfl_sync(0xffffffffu, v, 0); };
  const int csize = p.cluster, rank = same(csize > 1 ? static_cast<int>(cluster_rank()) : 0);
  const int step0 = same(p.steps * rank / csize), nsteps = same(p.steps * (rank + 1) / csize - step0);
  // Accumulators of a step: one a group, or of 8-bit codes one every 64 (11 + 8 + 7 bits are more than a float32 sum holds: 1.25e-7 of the result's norm, 1.0e-7 so).
  const int group_units = QK == kAff8 && p.group_shift == 7 ? 2 : 1, step_units = (kStepK >> p.group_shift) * group_units;
  const unsigned cluster = blockIdx.x / csize;
  const unsigned first = cluster * p.share + min(cluster, p.share_more);
  const int items = same(p.share + (cluster < p.share_more ? 1u : 0u));

  auto wait = [&](uint32_t bar, uint32_t parity, int where) -> bool { return wait_phase(smem + bar, parity, abort_at, where); };
  auto init = [&](uint32_t bar, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem + bar), "r"(n)); };

  // What an adding-up lane reads of a tile's tables: four entries of its row at a time, and which of them lie in its CTA's K.
  const int trow_lane = (warp & 3) * 32 + lane;
  constexpr int kEntry = QK == kMx4 ? 1 : WIDE ? 4 : 2;
  const int g_first = step0 * kStepK >> p.group_shift, g_end = min((step0 + nsteps) * kStepK >> p.group_shift, p.groups);
  auto table_row = [&](int tile) -> int64_t {
    const int64_t n = static_cast<int64_t>(tile) * kTileRows + trow_lane;
    return (n < p.N ? n : p.N - 1) * p.groups;
  };
  auto ahead = [&](int tile) {                           // into L2
    if (tile >= p.tiles) return;
    const int64_t at = table_row(tile);
    auto lines = [&](const void* table) {
      const uint8_t* q = static_cast<const uint8_t*>(table) + at * kEntry;
      for (int o = g_first * kEntry; o < g_end * kEntry; o += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(q + o));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(q + (g_end - 1) * kEntry));
    };
    lines(p.scales);
    if constexpr (QK != kMx4) lines(p.biases);
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.boxes; ++i) { init(kWFull + 8 * i, 1); init(kWEmpty + 8 * i, 4); }
    for (int i = 0; i < kASlots; ++i) { init(kAFull + 8 * i, 4); init(kAEmpty + 8 * i, 1); }
    for (int i = 0; i < kDSlots; ++i) { init(kDFull + 8 * i, 1); init(kDEmpty + 8 * i, kAddWarps); }
    for (int i = 0; i < 2; ++i) { init(kXFull + 8 * i, 1); init(kXFree + 8 * i, kAddWarps * csize); }
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(abort_at), "r"(0) : "memory");
    mbar_init_fence();
    const int tile0 = static_cast<int>(first % p.tiles);
    for (int b = 0; b < p.boxes && b < nsteps && items; ++b) {        // the first boxes travel while the rest is set up
      mbar_expect_tx(smem + kWFull + 8 * b, kBox);
      tma_load_2d(&w_map, w_at + b * kBox, smem + kWFull + 8 * b, (step0 + b) * kBoxBytes, tile0 * kTileRows);
    }
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem + kTmemSlot), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp >= kAddWarp && items) ahead(static_cast<int>(first % p.tiles));
  tc_fence_before();
  __syncthreads();
  if (csize > 1) cluster_barrier();
  tc_fence_after();
  // Not before tensor memory is this CTA's: a CTA of the next launch that came first (two fit an SM's shared memory where K is short; today registers forbid it) would
  // hold some while it waits for this grid, and the allocation above has no limit.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(smem + kTmemSlot) : "memory");
  tmem = __shfl_sync(0xffffffffu, tmem, 0);

  bool ok = true;
  // where each role is in its rings, over all chunks
  uint32_t slot = 0, phase = 0;                          // producer: box; issuer: slot of A
  uint32_t dslot = 0, dphase = 0;                        // issuer and adding up: accumulator
  uint32_t steps_before = 0;                             // the teams: steps of earlier tiles
  int added = 0;                                         // adding up: tiles pushed
  int late_tile = -1;                                    // ... and the one that is to be added up (a tile late)
  int64_t late_row = 0;
  bool issued = false;

  // The owner's part of a tile: 128 / csize of its rows, the CTAs' partial sums in rank order.
  const int own_shift = 7 - (31 - __clz(csize)), own = 1 << own_shift;
  auto add_up = [&](int item, int tile, int64_t row0) -> bool {
    const uint32_t s = p.slots == 1 ? 0u : item & 1u, ph = (p.slots == 1 ? item : item >> 1) & 1u;
    const int thread = (warp - kAddWarp) * 32 + lane;
    if (thread == 0) mbar_expect_tx(smem + kXFull + 8 * s, kTileRows * T * 4);
    if (!wait_phase<true>(smem + kXFull + 8 * s, ph, abort_at, 35)) return false;
    __syncwarp();
    const uint32_t from = part_at + s * partial_bytes(T);
    constexpr int kAdders = 32 * kAddWarps, kMost = kTileRows * (T / 4) / kAdders;       // (all of a tile's rows are this CTA's where there is no cluster)
#pragma unroll 1                                         // (two at a time spill: 9 rows 4096 x 14336 in groups of 32 65.0 us, 57.2 so)
    for (int j = 0; j < kMost; ++j) {
      const int i = thread + j * kAdders;
      if (i >= own * (T / 4)) break;
      const int r = i & (own - 1), t4 = i >> own_shift;
      const uint32_t at = from + r * kRow + t4 * 16;
      float v[4];
      // Neighbours first, then their sums: a rounding is relative to the sum so far, and one after another the last ones were all of a whole result (K 14336, one
      // sign: 5.0e-8, the few-rows kernel 4.6e-8).
      auto sum = [&](auto count) {
        constexpr int kCount = decltype(count)::value;
        float4 f[kCount];
#pragma unroll
        for (int c = 0; c < kCount; ++c) f[c] = ldsf128<0>(at + (c << own_shift) * kRow);
#pragma unroll
        for (int d = 1; d < kCount; d *= 2)
#pragma unroll
          for (int c = 0; c < kCount; c += 2 * d) f[c] = make_float4(f[c].x + f[c + d].x, f[c].y + f[c + d].y, f[c].z + f[c + d].z, f[c].w + f[c + d].w);
        v[0] = f[0].x; v[1] = f[0].y; v[2] = f[0].z; v[3] = f[0].w;
      };
      if (csize == 8) sum(std::integral_constant<int, 8>());
      else if (csize == 4) sum(std::integral_constant<int, 4>());
      else if (csize == 2) sum(std::integral_constant<int, 2>());
      else sum(std::integral_constant<int, 1>());
      const int64_t n = static_cast<int64_t>(tile) * kTileRows + rank * own + r, m = row0 + t4 * 4;
      int64_t o = m * p.N + n;
      const int left = n < p.N ? static_cast<int>(p.M - m < 4 ? p.M - m : 4) : 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (e < left) {
          if (p.y_dtype == QMM_F32) reinterpret_cast<float*>(p.y)[o] = v[e];
          else if (p.y_dtype == QMM_BF16) reinterpret_cast<__nv_bfloat16*>(p.y)[o] = __float2bfloat16_rn(v[e]);
          else reinterpret_cast<__half*>(p.y)[o] = __float2half_rn(v[e]);
        }
        o += p.N;
      }
    }
    __syncwarp();                                        // this warp has read its part of the slot: tell those who fill it
    if (lane < csize) remote_arrive_release(in_cta(smem + kXFree + 8 * s, lane));
    return true;
  };

  for (int done = 0; done < items && ok;) {
    const unsigned chunk = (first + done) / p.tiles;
    const int tile0 = same(static_cast<int>(first + done - chunk * p.tiles)), tiles = same(items - done < p.tiles - tile0 ? items - done : p.tiles - tile0);
    const int64_t row0 = static_cast<int64_t>(chunk) * T;

    if (done == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
    // ---- this CTA's stretch of K of the chunk's rows, as three pieces ----
    // (a lane has eight elements of a row, its neighbours those beside them)
    [[maybe_unused]] auto group_sum = [&](float sum, int c, int t, bool here) {
      const int eights = 1 << (p.group_shift - 3);
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      if (eights > 4) sum += __shfl_xor_sync(0xffffffffu, sum, 4);
      if (eights > 8) sum += __shfl_xor_sync(0xffffffffu, sum, 8);
      if ((lane & (eights - 1)) == 0 && here) sts32(sums_at + ((c >> (p.group_shift - 3)) * T + t) * 4, sum);
    };
    if constexpr (kScaled) {                             // a warp has a row's slice, sixteen elements a lane
      const int eights = nsteps * 16, slice0 = T == 48 ? 0 : step0 / kSliceSteps, slices = T == 48 ? 1 : (step0 + nsteps - 1) / kSliceSteps - slice0 + 1;
      constexpr int kAtOnce = 2;
      for (int u0 = warp; u0 < T * slices; u0 += kWarps * kAtOnce) {
        float f[kAtOnce][2][8];
        auto place = [&](int u, int h) -> int { return (T == 48 ? 0 : (slice0 + u / T) * (kSliceSteps * 16) - step0 * 16) + h * 32 + lane; };      // which eight elements
#pragma unroll
        for (int j = 0; j < kAtOnce; ++j) {
          const int u = u0 + j * kWarps;
          const int64_t m = row0 + u % T;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int c = place(u, h), k = step0 * kStepK + c * 8;
            float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
            if (u < T * slices && m < p.M && c >= 0 && c < eights && k < p.K) {
              const float4* src = reinterpret_cast<const float4*>(p.x + m * p.K + k);
              a = __ldg(src);
              b = __ldg(src + 1);
            }
            f[j][h][0] = a.x; f[j][h][1] = a.y; f[j][h][2] = a.z; f[j][h][3] = a.w;
            f[j][h][4] = b.x; f[j][h][5] = b.y; f[j][h][6] = b.z; f[j][h][7] = b.w;
          }
        }
#pragma unroll
        for (int j = 0; j < kAtOnce; ++j) {
          const int u = u0 + j * kWarps, t = u % T;
          if (u >= T * slices) continue;
          uint32_t most = 0;
          bool odd = false;                              // an infinity or a NaN among them
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const uint32_t bits = __float_as_uint(f[j][i >> 3][i & 7]) & 0x7FFFFFFFu;
            odd |= bits >= 0x7F800000u;
            most = max(most, bits >= 0x7F800000u ? 0u : bits);
          }
          const uint32_t e = max(__reduce_max_sync(0xffffffffu, most) >> 23, 15u);
          const float up = __uint_as_float((268u - e) << 23);
          if (lane == 0) sts32(back_at + (u / T * T + t) * 4, __uint_as_float((e - 14u) << 23));
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int c = place(u, h);
            const bool here = c >= 0 && c < eights;
            auto& g = f[j][h];
            const uint32_t to = x_at + (c >> 3) * kXBlock + t * 128 + (((c ^ t) & 7) << 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) g[i] *= up;
            if constexpr (QK != kMx4) group_sum(((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + (g[6] + g[7])), c, t, here);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              uint32_t v[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                v[q] = Half2Ops<__half>::pack(g[2 * q], g[2 * q + 1]);
                if (i < 2) {                             // what the piece leaves over (exact); an infinity leaves nothing, a NaN stays one
                  const float2 got = __half22float2(*reinterpret_cast<const __half2*>(&v[q]));
                  const bool whole0 = odd && i == 0 && fabsf(g[2 * q]) > 3.402823466e38f, whole1 = odd && i == 0 && fabsf(g[2 * q + 1]) > 3.402823466e38f;
                  g[2 * q] = whole0 ? 0.0f : g[2 * q] - got.x;
                  g[2 * q + 1] = whole1 ? 0.0f : g[2 * q + 1] - got.y;
                }
              }
              if (here) sts128(to + i * kPiece, __uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), __uint_as_float(v[3]));
            }
          }
        }
      }
    } else {
      const int pieces = nsteps * 16, units = T * pieces;
      const unsigned inverse = nsteps == p.most_steps ? p.most_inverse : p.less_inverse;
      auto row_of = [&](int u) -> int { return static_cast<int>(__umulhi(static_cast<unsigned>(u), inverse)); };
      constexpr int kAtOnce = 4;                         // requests in flight
      for (int u0 = threadIdx.x; u0 < units; u0 += kThreads * kAtOnce) {
        float4 a[kAtOnce], b[kAtOnce];
#pragma unroll
        for (int j = 0; j < kAtOnce; ++j) {
          const int u = u0 + j * kThreads, t = row_of(u), k = step0 * kStepK + (u - t * pieces) * 8;
          const int64_t m = row0 + t;
          a[j] = b[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (u < units && m < p.M && k < p.K) {
            const float4* src = reinterpret_cast<const float4*>(p.x + m * p.K + k);
            a[j] = __ldg(src);
            b[j] = __ldg(src + 1);
          }
        }
#pragma unroll
        for (int j = 0; j < kAtOnce; ++j) {
          const int u = u0 + j * kThreads, t = row_of(u), c = u - t * pieces;
          if (u >= units) continue;                      // (whole warps: a row has eight pieces a block, and T is a multiple of 16)
          float f[8] = {a[j].x, a[j].y, a[j].z, a[j].w, b[j].x, b[j].y, b[j].z, b[j].w};
          float sum = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
          const bool odd = !(fabsf(sum) <= 3.402823466e38f);       // an infinity or a NaN among them, perhaps
          group_sum(sum, c, t, true);
          // A piece is the eight bits of a mantissa that come next, cut off: what it leaves over is exact (the last eight are; below 2^-110, where it is more than
          // bf16's exponents reach, it is rounded). An infinity leaves nothing (not a NaN), and a NaN stays one.
          const uint32_t to = x_at + (c >> 3) * kXBlock + t * 128 + (((c ^ t) & 7) << 4);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            uint32_t h[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              h[e] = i < 2 ? __byte_perm(__float_as_uint(f[2 * e]), __float_as_uint(f[2 * e + 1]), 0x7632) : Half2Ops<__nv_bfloat16>::pack(f[2 * e], f[2 * e + 1]);
            sts128(to + i * kPiece, __uint_as_float(h[0]), __uint_as_float(h[1]), __uint_as_float(h[2]), __uint_as_float(h[3]));
            if (i < 2) {
#pragma unroll
              for (int e = 0; e < 8; ++e) f[e] -= __uint_as_float(__float_as_uint(f[e]) & 0xffff0000u);
              if (i == 0 && odd) {
                const float was[8] = {a[j].x, a[j].y, a[j].z, a[j].w, b[j].x, b[j].y, b[j].z, b[j].w};
#pragma unroll
                for (int e = 0; e < 8; ++e)
                  if (fabsf(was[e]) > 3.402823466e38f && was[e] == was[e]) f[e] = 0.0f;
              }
            }
          }
        }
      }
    }
    fence_proxy_async();
    __syncthreads();

    if (warp == 0) {
      // ---------------- weights ----------------
      if (lane == 0) {
        for (int i = 0; ok && i < tiles; ++i) {
          for (int b = 0; b < nsteps; ++b) {
            if (done || i || b >= p.boxes) {             // (the first ones went out at the start)
              if (!(ok = wait(kWEmpty + 8 * slot, phase ^ 1u, 31))) break;
              mbar_expect_tx(smem + kWFull + 8 * slot, kBox);
              tma_load_2d(&w_map, w_at + slot * kBox, smem + kWFull + 8 * slot, (step0 + b) * kBoxBytes, (tile0 + i) * kTileRows);
            }
            if (++slot == static_cast<uint32_t>(p.boxes)) { slot = 0; phase ^= 1u; }
          }
        }
      }
    } else if (warp == 1) {
      // ---------------- MMA issuer ----------------
      // first piece and second side by side, 2 T columns; the third on top of the second
      constexpr int kFormat = kScaled ? 0 : 1;
      constexpr uint32_t idesc1 = instr_desc(kFormat, kTileRows) | (static_cast<uint32_t>(T >> 3) << 17), idesc2 = instr_desc(kFormat, kTileRows) | (static_cast<uint32_t>(T >> 2) << 17);
      // (variables of this branch alone, known to be the same in all lanes, and one loop that is left where all lanes have seen a wait run out)
      uint32_t as = same(slot), aph = same(phase), ds = same(dslot), dph = same(dphase);
      const int total = same(tiles * nsteps);
      int b = 0;
      for (int i = 0; i < total; ++i) {
        if (!__all_sync(0xffffffffu, wait(kAFull + 8 * as, aph, 32))) break;
        bool there = true;
#pragma unroll 1
        for (int u = 0; u < step_units; ++u) {
          there = wait(kDEmpty + 8 * ds, dph ^ 1u, 33);
          if (!__all_sync(0xffffffffu, there)) break;
          tc_fence_after();
          const uint32_t d = tmem + kDAt + ds * (2 * T);
          if (step_units == 4) {
            const uint32_t acol = tmem + kASlotsAt + as * 64 + u * 16, desc = desc_low(x_at + (2 * b + (u >> 1)) * kXBlock) + (u & 1) * 4;
            tc_mma_half(d, acol, desc, kDescHigh, idesc2, 0u);
            tc_mma_half(d + T, acol, desc + 2 * (kPiece / 16), kDescHigh, idesc1, 1u);
          } else {
            for (int h = 0; h < 3 - step_units; ++h) {   // K blocks of the accumulator
              const uint32_t acol = tmem + kASlotsAt + as * 64 + (u + h) * 32, desc = desc_low(x_at + (2 * b + u + h) * kXBlock);
              tc_mma_block<false>(d, acol, desc, kDescHigh, idesc2, h);
              tc_mma_block<false>(d + T, acol, desc + 2 * (kPiece / 16), kDescHigh, idesc1, 1u);
            }
          }
          tc_commit<false>(smem + kDFull + 8 * ds, 0);
          if (++ds == kDSlots) { ds = 0; dph ^= 1u; }
        }
        if (!__all_sync(0xffffffffu, there)) break;
        tc_commit<false>(smem + kAEmpty + 8 * as, 0);
        issued = true;
        if (++as == kASlots) { as = 0; aph ^= 1u; }
        if (++b == nsteps) b = 0;
      }
      slot = as; phase = aph; dslot = ds; dphase = dph;
      // (done with the chunk, or gave up: what was issued completes before the activations are overwritten or tensor memory is given back)
      if (issued) mbar_drain(smem + kAEmpty + 8 * (slot ? slot - 1 : kASlots - 1), slot ? phase : phase ^ 1u);
    } else if (warp < kAddWarp) {
      // ---------------- codes -> A ----------------
      const int team = (warp - 2) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
      // 16-byte chunk c of a row lies at chunk c XOR row & 7 (rows of 128 bytes) or row / 2 & 3 (of 64): the TMA unit's swizzle of that width
      const uint32_t wrow = w_at + row * kBoxBytes, chunk0 = (kBoxBytes == 128 ? row & 7 : (row >> 1) & 3) << 4, to = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + kASlotsAt;
      const uint32_t n_end = steps_before + tiles * nsteps;
      for (uint32_t n = steps_before + ((team - steps_before) & (kTeams - 1)); n < n_end; n += kTeams) {
        // (the slot first: it says that the step kASlots before is done with, and so that the box before in this step's place, of kASlots or more, is too)
        const uint32_t lap = n / p.boxes, bs = n - lap * p.boxes;
        if (!(ok = wait(kAEmpty + 8 * (n % kASlots), (n / kASlots & 1u) ^ 1u, 34) && wait(kWFull + 8 * bs, lap & 1u, 36))) break;
        __syncwarp();
        tc_fence_after();
        const uint32_t from = wrow + bs * kBox;
#pragma unroll
        for (int q = 0; q < 4; ++q) {                    // 32 codes -> 16 columns
          uint32_t out[16];
#pragma unroll
          for (int c = 0; c < kRowBytes / 32; ++c) {
            const uint4 v = lds128<0>(from + (((q * (kRowBytes / 32) + c) << 4) ^ chunk0));
            const uint32_t words[4] = {v.x, v.y, v.z, v.w};
            codes16<QK>(words, out + c * 8);
          }
          tmem_st16(to + (n % kASlots) * 64 + q * 16, out);
        }
        __syncwarp();
        if (lane == 0) arrive_n(smem + kWEmpty + 8 * bs, 1);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_n(smem + kAFull + 8 * (n % kASlots), 1);
      }
      steps_before = n_end;
    } else {
      // ---------------- adding up ----------------
      constexpr int kOwn = T / 2;                        // activation rows of four warps
      const int t_own = (warp - kAddWarp) / 4 * kOwn;
      const uint32_t from = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + kDAt + t_own;
      struct Entries { uint32_t v[WIDE ? 4 : QK == kMx4 ? 1 : 2]; };
      const bool aligned = p.groups % 4 == 0 && ((reinterpret_cast<uintptr_t>(p.scales) | (QK == kMx4 ? 0 : reinterpret_cast<uintptr_t>(p.biases))) & 15) == 0;
      auto entries = [&](const void* table, int64_t trow, int g) -> Entries {      // of groups g .. g + 3
        Entries e;
        if (aligned) {
          const uint8_t* q = static_cast<const uint8_t*>(table) + (trow + g) * kEntry;
          if constexpr (WIDE) {
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(q));
            e.v[0] = u.x; e.v[1] = u.y; e.v[2] = u.z; e.v[3] = u.w;
          } else if constexpr (QK == kMx4) {
            e.v[0] = __ldg(reinterpret_cast<const uint32_t*>(q));
          } else {
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(q));
            e.v[0] = u.x; e.v[1] = u.y;
          }
        } else {
          uint32_t one[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int64_t at = trow + min(g + i, p.groups - 1);
            if constexpr (WIDE) one[i] = __ldg(static_cast<const uint32_t*>(table) + at);
            else if constexpr (QK == kMx4) one[i] = __ldg(static_cast<const uint8_t*>(table) + at);
            else one[i] = __ldg(static_cast<const uint16_t*>(table) + at);
          }
          if constexpr (WIDE) {
#pragma unroll
            for (int i = 0; i < 4; ++i) e.v[i] = one[i];
          } else if constexpr (QK == kMx4) {
            e.v[0] = one[0] | one[1] << 8 | one[2] << 16 | one[3] << 24;
          } else {
            e.v[0] = one[0] | one[1] << 16; e.v[1] = one[2] | one[3] << 16;
          }
        }
        return e;
      };
      auto value = [&](const Entries& e, int i) -> float {
        if constexpr (WIDE) return __uint_as_float(e.v[i]);
        else if constexpr (QK == kMx4) return __uint_as_float(max((e.v[0] >> (8 * i) & 0xffu) << 23, 0x00400000u));      // 2^(e8 - 127)
        else return table_value(e.v[i >> 1] >> (16 * (i & 1)) & 0xffffu, p.table_dtype);
      };
      const int g_batch = g_first & ~3;
      Entries sc = {}, bi = {};                          // of the tile's first groups
      auto first_entries = [&](int tile) {
        sc = entries(p.scales, table_row(tile), g_batch);
        if constexpr (QK != kMx4) bi = entries(p.biases, table_row(tile), g_batch);
      };
      first_entries(tile0);
      for (int i = 0; ok && i < tiles; ++i) {
        const int tile = tile0 + i;
        const int64_t trow = table_row(tile);
        Entries sc_next = sc, bi_next = bi;
        ahead(i + 1 < tiles ? tile + 1 : p.tiles);
        float y[kOwn];
#pragma unroll
        for (int t = 0; t < kOwn; ++t) y[t] = 0.0f;
        // (the sums of four groups at a time, in their slice's units: a rounding is relative to the sum so far. 48 rows' are of 512 codes at most.)
        constexpr bool kTwoLevels = T < 48;
        float total[kTwoLevels ? kOwn : 1];
#pragma unroll
        for (int t = 0; t < (kTwoLevels ? kOwn : 1); ++t) total[t] = 0.0f;
        const int last = (step0 + nsteps) * kStepK >> p.group_shift;       // (past the last group, perhaps: the end of the last step)
#pragma unroll 1
        for (int g0 = g_batch; ok && g0 < last; g0 += 4) {
          if (g0 + 4 < g_end) {                          // (the next four are on their way while these are used)
            sc_next = entries(p.scales, trow, g0 + 4);
            if constexpr (QK != kMx4) bi_next = entries(p.biases, trow, g0 + 4);
          }
          // (b + C s) sum x, while the accumulators are made: 25.5 -> 28.3 us at 33 rows of 4096 x 4096, 27.8 where the ranges are left to the block (83 with the entries read again for each group in a pass of its own)
          if constexpr (QK != kMx4) {
            float bc[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) bc[e] = fmaf(kCentre, value(sc, e), value(bi, e));
            const bool own = bc[0] != 0.0f || bc[1] != 0.0f || bc[2] != 0.0f || bc[3] != 0.0f;      // a row has biases that are not the centre's
            if (own) {
              const uint32_t at = sums_at + ((g0 - g_first) * T + t_own) * 4;
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                if (g0 + e < g_first || g0 + e >= g_end) continue;
#pragma unroll
                for (int t = 0; t < kOwn; t += 4) {
                  const float4 f = ldsf128<0>(at + (e * T + t) * 4);
                  fma2(y[t], y[t + 1], bc[e] * (1.0f / kUnit), f.x, f.y);
                  fma2(y[t + 2], y[t + 3], bc[e] * (1.0f / kUnit), f.z, f.w);
                }
              }
            }
            __syncwarp();
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int g = g0 + e;
            // (what lies past the last group has sums of nought)
            const float s = g < p.groups ? value(sc, e) : 0.0f;
#pragma unroll 1
            for (int u = g >= g_first && g < last ? group_units : 0; u > 0; --u) {
              ok = wait(kDFull + 8 * dslot, dphase, 37);
              if (!(ok = __all_sync(0xffffffffu, ok))) break;
              tc_fence_after();
              const uint32_t d = from + dslot * (2 * T);
#pragma unroll
              for (int t = 0; t < kOwn; t += 8) {
                uint32_t hi[8], lo[8];
                tmem_ld(d + t, hi);
                tmem_ld(d + T + t, lo);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 8; j += 2) add_fma2(y[t + j], y[t + j + 1], s, hi + j, lo + j);
              }
              tc_fence_before();
              __syncwarp();
              if (lane == 0) arrive_n(smem + kDEmpty + 8 * dslot, 1);
              if (++dslot == kDSlots) { dslot = 0; dphase ^= 1u; }
            }
            if (!ok) break;
          }
          sc = sc_next;
          bi = bi_next;
          if constexpr (kTwoLevels) {
            const uint32_t back = back_at + (((g0 << p.group_shift) / (kSliceSteps * kStepK) - step0 / kSliceSteps) * T + t_own) * 4;
#pragma unroll
            for (int t = 0; t < kOwn; t += 4) {
              float4 f = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
              if constexpr (kScaled) f = ldsf128<0>(back + t * 4);
              total[t] = fmaf(y[t], f.x, total[t]); total[t + 1] = fmaf(y[t + 1], f.y, total[t + 1]);
              total[t + 2] = fmaf(y[t + 2], f.z, total[t + 2]); total[t + 3] = fmaf(y[t + 3], f.w, total[t + 3]);
              y[t] = y[t + 1] = y[t + 2] = y[t + 3] = 0.0f;
            }
          }
        }
        if (!ok) break;
        if constexpr (kTwoLevels) {
#pragma unroll
          for (int t = 0; t < kOwn; ++t) y[t] = total[t];
        } else if constexpr (kScaled) {
#pragma unroll
          for (int t = 0; t < kOwn; t += 4) {
            const float4 f = ldsf128<0>(back_at + (t_own + t) * 4);
            y[t] *= f.x; y[t + 1] *= f.y; y[t + 2] *= f.z; y[t + 3] *= f.w;
          }
        }
        if constexpr (kUnit != 1.0f) {
#pragma unroll
          for (int t = 0; t < kOwn; ++t) y[t] *= kUnit;
        }
        if (i + 1 < tiles) first_entries(tile + 1);      // (on their way while this tile is passed on)
        // to the CTA that owns this row
        const uint32_t s = p.slots == 1 ? 0u : added & 1u, ph = (p.slots == 1 ? added : added >> 1) & 1u;
        ok = wait_phase<true>(smem + kXFree + 8 * s, ph ^ 1u, abort_at, 38);
        if (!(ok = __all_sync(0xffffffffu, ok))) break;
        const int owner = trow_lane >> own_shift;
        const uint32_t bar = in_cta(smem + kXFull + 8 * s, owner);
        const uint32_t to = in_cta(part_at + s * partial_bytes(T) + ((rank << own_shift) + (trow_lane & (own - 1))) * kRow + t_own * 4, owner);
#pragma unroll
        for (int t = 0; t < kOwn; t += 4) st_async4(to + t * 4, bar, y[t], y[t + 1], y[t + 2], y[t + 3]);
        if (p.slots == 1) {
          if (!(ok = add_up(added, tile, row0))) break;
        } else {
          if (late_tile >= 0 && !(ok = add_up(added - 1, late_tile, late_row))) break;
          late_tile = tile;
          late_row = row0;
        }
        ++added;
      }
    }
    done += tiles;
    __syncthreads();                                     // every role is done with the chunk's activations
    uint32_t gave_up;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(gave_up) : "r"(abort_at) : "memory");
    ok = ok && gave_up == 0;
    if (!ok && warp == 0 && lane == 0)                   // somebody gave up: the boxes on the way land first
      for (uint32_t i = 0; i < static_cast<uint32_t>(p.boxes); ++i) mbar_drain(smem + kWFull + 8 * i, i < slot ? phase : phase ^ 1u);
  }
  if (warp >= kAddWarp && ok && late_tile >= 0) add_up(added - 1, late_tile, late_row);

  tc_fence_before();
  __syncthreads();
  if (csize > 1) {
    __syncwarp();
    cluster_barrier();                                   // nobody leaves while a peer may still write to its shared memory
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
  if (threadIdx.x == 0) {
    int gave_up;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(gave_up) : "r"(abort_at) : "memory");
    if (gave_up) atomicCAS(p.status, 0, gave_up);
  }
}

struct F32Plan {
  int t, cluster, most_steps, slots, boxes;      // t == 0: the activations do not fit
  int64_t items, chunks;                         // (chunk, tile) items, chunks of t rows
};

// The plan of the least load, in clocks of the busiest cluster: rounds of tiles x (its K blocks, plus what a tile costs besides: the push, the sum), and the
// conversion of the activations. What it picked against the best of all plans when it was fitted, us (float32 tables, the few-rows kernel last; since then scaled pieces and the tree have
// changed these by up to 6 %): 33 rows 4096 x 4096 24.0 / 24.0 / 34.8,
// 64 rows 14336 x 4096 82.8 / 82.8 / 178, 4096 x 14336 114 / 114 / 234, 8-bit 64 rows 16384 x 1536 41 / 41 / 102, mxfp4 33 rows 5760 x 2880 26.2 / 26.2 / 47.3,
// 12 rows 65536 x 512 21.0 / 20.9 / 35.4, 1024 x 14336 18.1 / 18.0 / 20.4, 10 rows 4096 x 4096 13.9 / 13.9 / 17.0, 20 rows 2048 x 1024 in groups of 32 8.0 / 8.0 / 8.2.
F32Plan plan_of(const qmm_problem& p) {
  const int64_t steps_all = (p.K + kStepK - 1) / kStepK, tiles = (p.N + kTileRows - 1) / kTileRows;
  const int sms = device_sm_count(), bits = p.mode != QMM_MODE_MXFP4 && p.bits == 8 ? 8 : 4;
  F32Plan best = {};
  double least = 0.0;
  for (int c = kMaxCluster; c >= 1; c /= 2) {
    if (c > steps_all) continue;
    const int steps = static_cast<int>((steps_all + c - 1) / c);
    for (int t = 48; t >= 16; t -= 16) {
      // (48 rows' sums and slices are of 512 codes at most: see kTwoLevels)
      if ((t == 48 && steps > 4) || smem_of(t, steps, 1, kASlots, bits) > kSmemLimit) continue;
      const int64_t chunks = (p.M + t - 1) / t, items = chunks * tiles, clusters = sms / c < items ? sms / c : items, rounds = (items + clusters - 1) / clusters;
      const double passes = static_cast<double>(chunks < rounds ? chunks : rounds);
      const double load = rounds * (steps * 2 * (180.0 + 2.0 * t) + (c > 1 ? 250.0 + 200.0 * c : 400.0) + 10.0 * t) + passes * steps * t * 10.0;
      if (!best.t || load < least) {
        least = load;
        const int slots = smem_of(t, steps, 2, kASlots, bits) <= kSmemLimit ? 2 : 1, boxes = static_cast<int>((kSmemLimit - smem_of(t, steps, slots, 0, bits)) / box_bytes(bits));
        best = {t, c, steps, slots, boxes < kMaxBoxes ? boxes : kMaxBoxes, items, chunks};
      }
    }
  }
  return best;
}

// What a plan is expected to take, in us: rounds of tiles -- a step's codes, its accumulators (one a group; reading, scaling and adding T columns of each),
// the rows passed on -- and the conversion of the activations for every chunk that a cluster meets. GPCs differ in their SMs, so that fewer clusters fit than
// their CTAs would: of eight 14 or 15 of 18, of four 33 of 37. Fitted to 2650 timed plans of 1400 random products (9..100 rows, K 128..14336, N 128..32000, all
// kinds); root mean square error 10 %.
double estimate(const qmm_problem& p, const F32Plan& pl) {
  const bool mx = p.mode == QMM_MODE_MXFP4, bytes = !mx && p.bits == 8;
  const int sms = device_sm_count(), step_units = mx ? 4 : bytes && p.group_size == 128 ? 2 : kStepK / p.group_size;
  const int64_t fit = pl.cluster == 8 ? sms * 14 / 148 : pl.cluster == 4 ? sms * 33 / 148 : sms / pl.cluster, clusters = fit < pl.items ? fit > 0 ? fit : 1 : pl.items;
  const int64_t rounds = (pl.items + clusters - 1) / clusters, tiles = pl.items / pl.chunks, meets = rounds > 1 ? (rounds + tiles - 2) / tiles + 1 : 1;
  const int64_t passes = pl.chunks < meets ? pl.chunks : meets, steps = pl.most_steps;
  return 3.6 + rounds * (0.75 + steps * (bytes ? 0.46 : 0.31) + steps * step_units * (0.14 + 0.0013 * pl.t) + 0.048 * pl.t) +
         passes * steps * pl.t * (mx || bytes ? 0.026 : 0.014);
}

template <int QK, int T, bool WIDE>
int launch_w(const qmm_problem& p, const F32Plan& pl, const CUtensorMap& wm, F32Params& fp, cudaStream_t stream) {
  auto kernel = qmm_f32_tc_kernel<QK, T, WIDE>;
  static bool configured[kMaxDevices] = {};     // the attribute is per device
  const int dev = current_device();
  if (dev < 0) return QMM_ERR_DEVICE;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) return fail(QMM_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    configured[dev] = true;
  }
  const int64_t items = (p.M + T - 1) / T * fp.tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem_of(T, pl.most_steps, pl.slots, pl.boxes, QK == kAff8 ? 8 : 4);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = pl.cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int64_t clusters = device_sm_count() / pl.cluster;
  if (pl.cluster > 1) {
    cfg.gridDim = dim3(static_cast<unsigned>(clusters * pl.cluster));
    const int most = max_active_clusters(reinterpret_cast<const void*>(kernel), cfg, pl.cluster);
    if (most > 0 && clusters > most) clusters = most;
  }
  if (clusters > items) clusters = items;
  if (clusters < 1) clusters = 1;
  cfg.gridDim = dim3(static_cast<unsigned>(clusters * pl.cluster));
  fp.share = static_cast<unsigned>(items / clusters);
  fp.share_more = static_cast<unsigned>(items % clusters);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, wm, fp);
  if (e != cudaSuccess) return fail(QMM_ERR_CUDA, "qmm_f32_tc_kernel launch: %s", cudaGetErrorString(e));
  count_launch();
  return check_launch("qmm_f32_tc_kernel");
}

template <int QK, int T>
int launch_t(const qmm_problem& p, const F32Plan& pl, const CUtensorMap& wm, F32Params& fp, cudaStream_t stream) {
  if constexpr (QK != kMx4)
    if (p.table_dtype == QMM_F32) return launch_w<QK, T, true>(p, pl, wm, fp, stream);
  return launch_w<QK, T, false>(p, pl, wm, fp, stream);
}

template <int QK>
int launch_kind(const qmm_problem& p, const F32Plan& pl, const CUtensorMap& wm, F32Params& fp, cudaStream_t stream) {
  if (pl.t == 48) return launch_t<QK, 48>(p, pl, wm, fp, stream);
  if (pl.t == 32) return launch_t<QK, 32>(p, pl, wm, fp, stream);
  return launch_t<QK, 16>(p, pl, wm, fp, stream);
}

// One weight, no gather; and K as far as 16 rows' pieces fit shared memory (14336 with 4-bit codes, 12288 with 8-bit ones), which the plan says.
bool may_take(const qmm_problem& p) {
  if (p.x_dtype != QMM_F32 || p.batch != 1 || p.lhs_idx || p.rhs_idx || p.group_sizes || p.mode == QMM_MODE_FLOAT) return false;
  if (p.M < 1 || p.K < kBK || p.K % 32 || p.K >= (1LL << 24) || p.N < 1 || p.N >= (1LL << 31) - 256) return false;
  return (p.M + 15) / 16 * ((p.N + kTileRows - 1) / kTileRows) < (1LL << 31);
}

}  // namespace

bool f32_tc_supports(const qmm_problem& p) { return may_take(p) && plan_of(p).t != 0; }

// Up to eight rows are two passes of the few-rows kernel, which a pass here does not beat (5 rows of 4096 x 4096 12.6 us). From nine on the two estimates decide. Of
// 1214 random products (as above) 224 were more than 3 % slower here than there, up to 2.4 times (few tiles of little K, groups of 32, whose accumulators are
// many: 9 rows mxfp4 160 x 8576 16.5 / 9.0 us); as decided 28 are, and all take 1 % more than the better kernel of each would.
bool f32_tc_pays(const qmm_problem& p) {
  if (p.M <= 8 || !may_take(p)) return false;
  const F32Plan pl = plan_of(p);
  return pl.t != 0 && (!rows_supports(p) || estimate(p, pl) <= 0.97 * rows_estimate(p));
}

void f32_tc_plan(const qmm_problem& p, int plan[3]) {
  const F32Plan pl = plan_of(p);
  plan[0] = pl.t; plan[1] = pl.cluster; plan[2] = pl.slots;
}

int launch_f32_tc(const qmm_problem& p, cudaStream_t stream) {
  const F32Plan pl = plan_of(p);
  const bool mx = p.mode == QMM_MODE_MXFP4;
  const int bits = !mx && p.bits == 8 ? 8 : 4, group = mx ? 32 : p.group_size;
  F32Params fp = {};
  fp.x = static_cast<const float*>(p.x); fp.scales = p.scales; fp.biases = p.biases; fp.y = p.y;
  fp.status = device_status_word();
  if (!fp.status) return fail(QMM_ERR_CUDA, "could not allocate the device status word");
  fp.M = p.M; fp.N = p.N; fp.K = static_cast<int>(p.K);
  fp.groups = fp.K / group;
  fp.group_shift = group == 128 ? 7 : group == 64 ? 6 : 5;
  fp.table_dtype = p.table_dtype; fp.y_dtype = p.y_dtype;
  fp.tiles = static_cast<int>((p.N + kTileRows - 1) / kTileRows);
  fp.steps = (fp.K + kStepK - 1) / kStepK;
  fp.most_steps = pl.most_steps; fp.cluster = pl.cluster; fp.slots = pl.slots; fp.boxes = pl.boxes;
  fp.most_inverse = 0xFFFFFFFFu / (16 * pl.most_steps) + 1;
  fp.less_inverse = 0xFFFFFFFFu / (16 * (pl.most_steps > 1 ? pl.most_steps - 1 : 1)) + 1;
  const uint64_t row_bytes = static_cast<uint64_t>(p.K) * bits / 8;
  CUtensorMap wm;
  const int rc = tensor_map_2d(&wm, QMM_U8, p.w, row_bytes, static_cast<uint64_t>(p.N), row_bytes, kStepK * bits / 8, kTileRows, bits == 8 ? 1 : 2);
  if (rc) return rc;
  if (mx) return launch_kind<kMx4>(p, pl, wm, fp, stream);
  if (bits == 8) return launch_kind<kAff8>(p, pl, wm, fp, stream);
  return launch_kind<kAff4>(p, pl, wm, fp, stream);
}

}  // namespace qmm
