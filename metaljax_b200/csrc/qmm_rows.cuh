// The few-rows kernel of the fused dequantize-and-matmul (`y = x . deq(w)^T`,
// src/metaljax/qmm.py:2491): 2..16 rows of 16-bit activations against a streamed weight (and one row
// where the single-row integer kernel declines), unsorted expert gathers, grouped products of a few rows
// per expert, and products of float32 activations: up to 8 rows, and what qmm_f32_tc.cu does not take.
//
// What bounds it. An SM's share of HBM is 23 bytes a clock, 46 4-bit codes: at four instructions a
// clock that leaves 22 warp instructions per 256 codes, two thirds of what a dequantization element by
// element takes, so the budget decides the layout: nothing may be done twice for a code, and nothing that
// belongs to the activations may be done per tile of weights.
//
// Split. A warp owns ONE slice of 512 codes of K for as long as it lives and holds its slice of the
// activations as MMA fragments in registers (64 registers per 8 columns); the warps of a CTA
// (up to 8) are consecutive slices, the CTAs of a cluster (up to 8) consecutive stretches of K. Weight tiles
// of 16 rows pass by: 16 x 128-byte boxes by TMA (128-byte swizzle) through a ring of its own per warp,
// a few boxes ahead across tiles, so the HBM stream never waits for a barrier of the CTA. The warps'
// partial sums of a tile meet in shared memory, one warp (in turn) adds them up in warp order; in
// a cluster the CTAs' sums travel to the tile's leader (in turn) by st.async and are added in rank order, when the leader's next tile comes: waiting for
// them there and then held up a warp for each tile (8 rows of 4096 x 14336 15.9 -> 13.9 us).
// No global scratch, no atomics, fixed order of summation.
//
// Arithmetic. The codes are never dequantized: a nibble pair under a magic exponent is an exact bf16 (128 + q) or f16 (16 + q) A
// fragment of `mma.sync.m16n8k16`, an 8-bit pair an f16 one (1024 + q, a byte permute), an E2M1 pair an exact f16 times 2^-14; scale and bias
// meet the float32 accumulators once per group (the 16 K slots of an MMA lie in one group; the accumulators start at -C sum x, which takes the
// magic number out again; 16 + q, with the code at the top of the mantissa, is a shift more per two words than 1024 + q and leaves that much less to cancel:
// 8 rows of f16, one sign, 4.6e-4 -> 1.2e-6 of the result's norm in float32, grouped products 1.4e-4 -> 5e-7). The bias term is an MMA of its own per 16 rows and slice: the bf16 bias entries against the groups' sums of x
// in three bf16 pieces. Activations that the element type cannot hold as they are become several columns or carry a power of two: float32 is
// three columns (8 + 8 + 8 bits of bf16, or 11 + 11 + 11 of f16) that are added at the end; for f16 fragments of bf16 or float32 activations
// each row of each slice is scaled to [2^14, 2^15) by its largest finite magnitude, and back in its partial sums. The K order inside a group is
// free as long as codes and activations agree: lane t takes 16 consecutive codes (8 in groups of 32), in the pair order one LOP3 extracts.
// Masks and shifts run at half the rate of the issue (16 lanes a clock), so that seven of them in eight codes of a lane are 14 clocks against the
// MMAs' 8: as bf16 the upper nibble of a byte comes out of its place by a mask and an FMA (below), 10 clocks and 4 of another pipe
// (8 rows of 128256 x 4096 64.6 -> 58.0 us, with the sums below and accumulators that start from a register quad).
// The fragments of 16-bit activations are the loaded words, and the groups' sums float32 additions of them that take a 16-bit operand (with a conversion
// each they took 800 instructions a warp, some 2 us of every launch).
// A launch releases its successor in its first instruction: the way from there to the next launch's CTAs bounds the rate of small products (2 rows of 4096 x 4096
// 6.3 -> 5.5 us, 4 rows of 5632 x 2048 5.7 -> 4.8, 8 rows of 1024 x 1024 4.1 -> 3.3).
//
// Where the results are meant to be float32 -- float32 activations, and the 16-bit ones of unsorted gathers of more than 16 rows (EXACT) -- the
// magic number, though it cancels, would cost them the bits in which it is larger than a code. There one exact subtraction a pair makes it q - 8 or q - 128, the accumulators start at nought, and the bias that goes with
// the sum of x is b + 8 s or b + 128 s (nought for most weights). What is left is the tensor core's truncation of a float32 sum. (Codes as f16
// subnormals need neither the magic nor the subtraction, but are aligned as if they had all their bits.)
// Relative error against float64 (2-norm, the largest over K 512 to 14336 and all group sizes) of the SIMT kernel / with the magic number / so, for N(0, 1),
// one sign, outliers of 300: 4-bit 3.8e-7 / 4.9e-6 / 1.1e-7, 6.0e-7 / 1.3e-5 / 0.7e-7, 4.5e-7 / 1.1e-5 / 1.1e-7; 8-bit 2.6e-7 / 3.5e-6 / 1.4e-7,
// 6.8e-7 / 2.2e-4 / 1.3e-7, 3.7e-7 / 5.4e-6 / 3.0e-7. 33 rows of 4096 x 4096: 34.8 us with the magic number, 34.5 so; 8-bit 43 and 47.
// Range: an infinite activation makes its row's results infinite or NaN, as a sum of products does (affine codes: NaN where s (q - C) x and
// the bias term have opposite signs); finite ones up to 2^120 give finite results where those fit. 4-bit codes take float32
// activations below 2^-110 with fewer than 24 bits.
// (8-bit float MMAs would take the codes with a third of the instructions, but `mma.sync` on e4m3 is emulated here with
// conversions to f16: 88 against 67 us for 8 rows of 128256 x 4096.)
//
// Measured (device time, weights from HBM): int4 group 64 8 rows 28672 x 4096 17.2 us (3.8 TB/s; 18.6 a call by itself), 128256 x 4096 58.2 (5.1 TB/s), 4096 x 14336 14.1, 16 rows 128256 x 4096 109,
// 4096 x 4096 7.7; 8-bit 14336 x 4096 13.5 in groups of 64 or 128, bf16 activations and tables. Tried: fragments in tensor memory (tcgen05.st / ld), rolled loops and two CTAs of 8 warps on an SM: 20.1 us at 28672 x 4096 when the above
// was not there yet, 19.1 with it (16 rows a tile cost more instructions a code; the allocation delays the next launch's release); a last tile of 16 rows where a CTA's
// share is not whole tiles: 4096 x 14336 14.8 instead of 13.9 (its code is fetched for it alone).
// Where this kernel came from (before: a kernel with the same fragments under the same kind of magic
// number that read its activations from shared memory for every tile and staged each tile's tables there behind barriers of the CTA; float32: the SIMT kernel), int4 group 64: 8 rows 28672 x 4096 27.1 -> 20.2 us (3.3 TB/s), 128256 x 4096
// 99.5 -> 65.6 (4.5 TB/s), 4096 x 14336 26.8 -> 16.8, 16 rows 128256 x 4096 170 -> 128, 16 rows 4096 x 4096 12.2 -> 9.2; 8-bit 14336 x 4096 22.6
// -> 15.5 (3.9 TB/s); float32 33 rows 4096 x 4096 323 -> 34.5. At the small end (2 rows 4096 x 4096: 5.4 us) it is the chain launch, activations,
// one tile, sum that counts, not a stream.
// Rows of a table that are no multiple of 16 bytes are copied by words, and every such copy but those of float32 entries in groups of 32 is a line a lane: a word more a row
// costs 4 to 20 % of a product (K of 5376, 7936). MXFP4 against such K is 2 to 6 % slower than before the codes' chunks of 64 (8 rows of 37802 x 7936 56.0 -> 58.3 us), other kinds 1 to 5 % faster.
//
// Every wait on an mbarrier is bounded. The kernel is launched with programmatic stream
// serialization: it lets the next kernel of the stream start early and touches only weights and
// tables before `griddepcontrol.wait` (a gather or grouped product waits first: indices decide what it reads).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "qmm_internal.h"
#include "qmm_ptx.cuh"

namespace qmm {
namespace rows {

using namespace ptx;

constexpr int kMaxWarps = 8;
constexpr int kSliceK = 512;            // codes of K per warp
constexpr int kBlockRows = 16;          // weight rows of an MMA; a tile is one or two blocks (see plan_rows)
constexpr int kBoxBytes = 128;          // bytes of a weight row in a TMA box
constexpr int kMaxRing = 6;
constexpr int kMaxCluster = 8;
constexpr int kExchangeSlots = 2;       // tiles a leader may have on the way from its peers
constexpr int kMaxSegments = 1024;      // experts of a grouped product
constexpr int kSmemLimit = 226 * 1024;

enum { kAff4 = 0, kAff8 = 1, kMx4 = 2 };
enum { kTabBf16 = 0, kTabF16 = 1, kTabF32 = 2, kTabE8 = 3 };           // table entries
constexpr int entry_bytes(int tt) { return tt == kTabF32 ? 4 : tt == kTabE8 ? 1 : 2; }

struct RowsParams {
  const void* x;
  const void* scales;
  const void* biases;
  void* y;
  const int32_t* lhs_idx;        // gather: x batch and weight of segment s
  const int32_t* rhs_idx;
  const int32_t* group_sizes;    // grouped: rows of segment s (they follow one another in x and y)
  const int32_t* x_rows;         // grouped: the row of x behind row r of the product (NULL: r)
  int* status;
  int64_t x_batch_stride, y_batch_stride, num_weights, x_batches, M;
  int K, N, segs, groups;        // groups = K / group_size
  int weight_rows;               // weight rows between segments (N, or 0: one weight)
  int table_dtype, y_dtype;
  int tiles;                     // tiles per weight
  int cluster, slices_per_cta, slices_per_warp;
  unsigned share, share_more;    // dense: (chunk, tile) items of every cluster, and how many clusters have one more
  int ring, red_bufs;
  int table_unit;                // bytes on which every row's table entries of every slice start: 16, 8, 4, or less
  int64_t table_bytes;           // of a whole table
  int64_t total_x_rows;          // grouped: rows of x that x_rows may name
  const void* scales2;           // a pair of weights of one shape (two blocks): block 0 of a tile is 16 rows of the first, block 1 the same
  const void* biases2;           //   rows of the second, and y is silu(first) * second; NULL: one weight
};

// d (+)= A (16 rows of weights) * B (8 columns of activations), K 16.
template <typename AT>
struct Mma;
template <>
struct Mma<__nv_bfloat16> {
  static __device__ __forceinline__ void run(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  // ... starting from c (its two columns in both rows: the same two floats twice)
  static __device__ __forceinline__ void first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
  }
};
template <>
struct Mma<__half> {
  static __device__ __forceinline__ void run(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ void first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
  }
};

// (a & b) | c in one LOP3 with all three operands in registers.
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// y0, y1 += s * a0, s * a1 in one instruction.
__device__ __forceinline__ void fma2(float& y0, float& y1, float s, float a0, float a1) {
  asm("{ .reg .b64 y, s, a; mov.b64 y, {%0, %1}; mov.b64 s, {%2, %2}; mov.b64 a, {%3, %4}; fma.rn.f32x2 y, s, a, y; mov.b64 {%0, %1}, y; }"
      : "+f"(y0), "+f"(y1) : "f"(s), "f"(a0), "f"(a1));
}

__device__ __forceinline__ void store_y(void* p, int dtype, int64_t i, float v) {
  if (dtype == QMM_BF16) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else if (dtype == QMM_F16) reinterpret_cast<__half*>(p)[i] = __float2half_rn(v);
  else reinterpret_cast<float*>(p)[i] = v;
}

template <int N, int I = 0, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<N, I + 1>(f);
  }
}

// Two floats as a pair of AT, and the floats the pair stands for.
template <typename AT>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (std::is_same<AT, __nv_bfloat16>::value) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}
template <typename AT>
__device__ __forceinline__ float2 unpack2(uint32_t u) {
  if constexpr (std::is_same<AT, __nv_bfloat16>::value) return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
  else return __half22float2(*reinterpret_cast<const __half2*>(&u));
}

// What `got`, a value rounded to fewer bits, leaves of it (exact; nothing of an infinity).
constexpr float kMaxFloat = 3.402823466e38f;
__device__ __forceinline__ float left_of(float value, float got) { return fabsf(got) > kMaxFloat ? 0.0f : value - got; }

// A pair of bf16: a * b + c. (Bits 0 to 7 of a bf16 whose others are nought are a whole number times 2^-133, subnormal or not: a nibble comes out
// of either place by one mask and one of these, exactly and on the pipe that the masks leave idle.)
__device__ __forceinline__ uint32_t fma_bf16(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// a + the lower, + the upper of a pair, rounded after each.
template <typename AT>
__device__ __forceinline__ float add_pair(float a, uint32_t pair) {
  const uint16_t lower = static_cast<uint16_t>(pair), upper = static_cast<uint16_t>(pair >> 16);
  if constexpr (std::is_same<AT, __half>::value) {
    asm("add.rn.f32.f16 %0, %1, %0;" : "+f"(a) : "h"(lower));
    asm("add.rn.f32.f16 %0, %1, %0;" : "+f"(a) : "h"(upper));
  } else {
    asm("add.rn.f32.bf16 %0, %1, %0;" : "+f"(a) : "h"(lower));
    asm("add.rn.f32.bf16 %0, %1, %0;" : "+f"(a) : "h"(upper));
  }
  return a;
}

// The codes under the magic exponent minus (magic + centre): exact.
template <typename AT>
__device__ __forceinline__ uint32_t centred(uint32_t pair, float offset) {
  if constexpr (std::is_same<AT, __nv_bfloat16>::value) {
    const __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&pair), __float2bfloat162_rn(offset));
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&pair), __float2half2_rn(offset));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t remote(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void remote_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// mbar_wait for a barrier that another CTA of the cluster arrives on (its reads happened before our writes).
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, uint32_t abort_flag, int where) {
  const long long t0 = clock64();
  for (int spins = 1;; ++spins) {
    uint32_t done;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if ((spins & 255) == 0) {
      uint32_t gave_up;
      asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(gave_up) : "r"(abort_flag) : "memory");
      if (gave_up) return false;
      if (clock64() - t0 > kSpinLimit) {
        asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(abort_flag), "r"(where) : "memory");
        return false;
      }
    }
  }
}
__device__ __forceinline__ void st_async4(uint32_t addr, uint32_t bar, const float (&v)[4]) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "f"(v[0]),
               "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar)
               : "memory");
}

// Shared memory, from the (1024-byte aligned) start: barriers and small state, then per warp its ring, then
// what the CTA shares. Fixed places first: an address that is a constant costs no register.
constexpr int kFullAt = 0;                                             // [kMaxWarps][kMaxRing] a box has landed
constexpr int kRedFullAt = kMaxWarps * kMaxRing * 8;                   // [4] every warp's share of a tile is there
constexpr int kRedEmptyAt = kRedFullAt + 4 * 8;                        // [4] ... and has been added up
constexpr int kXFullAt = kRedEmptyAt + 4 * 8;                          // [kExchangeSlots] the peers' sums of a tile this CTA leads
constexpr int kXFreeAt = kXFullAt + kExchangeSlots * 8;                // [kMaxCluster][kExchangeSlots] leader r has read slot s
constexpr int kAbortAt = kXFreeAt + kMaxCluster * kExchangeSlots * 8;  // the abort flag, the number of chunks of a grouped product
constexpr int kStateAt = kAbortAt + 16;                                // [kMaxWarps][2] where a warp's consumer is
constexpr int kStateBytes = 32;
constexpr int kAheadAt = kStateAt + kMaxWarps * 2 * kStateBytes;       // [kMaxWarps] where its requests are: segment, chunk
constexpr int kLedAt = kAheadAt + kMaxWarps * 8;                                   // [kExchangeSlots] where a tile that this CTA leads goes: element of y, rows, tile
constexpr int kHeadBytes = (kLedAt + kExchangeSlots * 16 + 1023) / 1024 * 1024;

struct Place {            // one chunk of the walk: 8 NT columns against every row of one weight
  int64_t y0;             // element of y that its first column's first weight row goes to
  int seg, chunk;
  int rows_left;          // activation rows of it that exist
  int weight_row;         // first row of its weight
};
static_assert(sizeof(Place) <= kStateBytes, "");

// 16-row blocks of a tile: two halve what a tile costs apart from its codes, one halves the wait for a lone tile (plan_rows).
constexpr int kMaxBlocks = 2;

// A tile's table entries travel with its codes: per weight row the slice's entries as they are in memory, so far apart that reads of a word of eight rows meet
// all banks, with a word to spare for entries that do not start on a word. QUADS (affine tables): rows of 16 bytes and more lie on
// multiples of 16, for one copy to take that many, every few rows another 16 bytes further on, and the spare words behind the rows. MXFP4's scales are copied by
// eights at most (K of no multiple of 512 2 % slower else). (A pitch of the row and 16 bytes for all of them took memory that rings and
// plans were made of: steps of 2 sequences 251 -> 271 us, float32 against 8-bit codes 28480 x 2048 17.3 -> 25.7. By eights alone 8 rows of 28672 x 4096 take
// 17.4 us instead of 17.1, in groups of 32 with float32 tables 30.0 instead of 24.4, float32 activations there 17 % more.)
constexpr int table_row_bytes(int groups, int tt) { return groups * entry_bytes(tt); }
constexpr bool table_quads(int groups, int tt) { return tt != kTabE8 && table_row_bytes(groups, tt) >= 16; }
constexpr int table_at(int row, int groups, int tt, bool quads) {
  const int bytes = table_row_bytes(groups, tt);
  return quads ? row * bytes + (bytes == 32 ? (row >> 2) * 16 : bytes == 64 ? (row >> 1) * 16 : 0) : row * (bytes == 8 ? 16 : bytes + 8);
}
constexpr int table_bytes(int rows, int groups, int tt, bool quads) { return table_at(rows, groups, tt, quads) + (quads && entry_bytes(tt) < 4 ? rows * 4 : 0); }
constexpr int table_stage_bytes(int blocks, int groups, int tt, bool quads) { return table_bytes(kBlockRows * blocks, groups, tt, quads) * (tt == kTabE8 ? 1 : 2); }
// The groups' sums of a slice's columns; a pair of columns twice where accumulators of two rows start there (one read, no moves, and no spills: 16-bit tables in groups of
// 32 11 % slower without), but not where no plan has the memory for it.
constexpr bool sums_twice(int qk, int groups, int tt, bool centred) { return qk != kMx4 && !centred && !(groups == 16 && tt == kTabF32) && !(qk == kAff8 && groups == 4 && tt != kTabF32); }
constexpr int sums_bytes(int groups, bool twice) { return groups * (twice ? 64 : 32); }
// Fragments of a second column group (the third piece of float32): they would not fit the registers.
constexpr int more_x_bytes(int tokens) { return tokens == 8 ? 0 : kSliceK * 16; }

// QK: quantization kind. XT: activation type in memory. T: activation rows (tokens) of a chunk, 8 (16-bit) or 4 (float32). SPG: 32-code
// steps per quantization group (1, 2, 4). TT: what the table entries are. R: 16-row blocks of a tile. EXACT: the magic number is taken off the codes, not
// off the sums (affine codes).
// With a second weight (scales2; two blocks, 16-bit activations) the two blocks of a tile are the same rows of both, and y is silu(first) * second: three launches
// as one. 4 rows of a feed-forward block of 2048 x 5632 23.1 -> 17.0 us. It is no kernel of its own, though that would cost plain products nothing (18.0 against 18.3 us, 8 rows of
// 28672 x 4096): where this one and another of its size take turns, each launch is slower (16.6 -> 22.3 us a launch of two kernels in turn; the feed-forward
// block 20.3, 8 tokens through 8 experts 198 against 178).
template <int QK, typename XT, int T, int SPG, int TT, int R, bool EXACT>
__global__ void __launch_bounds__(kMaxWarps * 32, 1)
qmm_rows_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap w2_map, const RowsParams p) {
  using AT = typename std::conditional<QK == kAff4, typename std::conditional<std::is_same<XT, float>::value, __nv_bfloat16, XT>::type, __half>::type;
  constexpr bool kScaled = std::is_same<AT, __half>::value && !std::is_same<XT, __half>::value;
  // A pair of codes under this exponent is kMagicValue + code.
  constexpr uint32_t kMagic = QK == kAff8 ? 0x64006400u : std::is_same<AT, __half>::value ? 0x4C004C00u : 0x43004300u;
  constexpr float kMagicValue = QK == kAff8 ? 1024.0f : std::is_same<AT, __half>::value ? 16.0f : 128.0f;
  constexpr bool kCentred = EXACT && QK != kMx4, kMayPair = !EXACT && R == 2 && sizeof(XT) == 2;
  // 4-bit codes as bf16: of each pair of nibbles the upper one by an FMA, as (128 + q) / 4 against four times the activation, or both as (q - 8) / 64.
  constexpr bool kNibbles = QK == kAff4 && std::is_same<AT, __nv_bfloat16>::value, kQuarters = kNibbles && !kCentred;
  constexpr float kCentre = QK == kAff8 ? 128.0f : 8.0f;
  constexpr float kSumIs = kCentred ? 1.0f : -kMagicValue;   // the groups' sums of x are kept times this
  // Columns: piece i of the tokens is column group i, its column c token c. With 4 tokens two pieces share
  // a group: column c is token c & 3 of piece 2 h + (c >> 2).
  constexpr int kPieces = std::is_same<XT, float>::value ? 3 : 1;
  constexpr bool kHalf = T == 4;
  constexpr int NT = kHalf ? (kPieces + 1) / 2 : kPieces;
  constexpr int kBits = QK == kAff8 ? 8 : 4;
  constexpr int kTileRows = kBlockRows * R;
  constexpr int kBoxSmem = kTileRows * kBoxBytes;
  constexpr int kBoxes = kSliceK * kBits / 8 / kBoxBytes;             // boxes side by side in a slice
  constexpr int kStage = kBoxes * kBoxSmem;
  constexpr int kBlk = SPG == 1 ? 32 : 64;                            // codes that four lanes read together
  constexpr int kBlocks = kSliceK / kBlk;
  constexpr int kLane = kBlk / 4;                                     // consecutive codes of a lane in a block
  constexpr int kMmas = kBlk / 16;
  constexpr int kGroups = kSliceK / (32 * SPG);                       // groups of a slice
  // The codes are worked through in chunks of 64 (eight fragment registers of a column group), four to a half of the slice.
  constexpr int kChunkBlocks = 64 / kBlk;
  constexpr int kHalfGroups = kGroups / 2;
  constexpr int kChunkWords = 64 * kBits / 128;                       // words of a lane and row in a chunk
  constexpr bool kBiasMma = TT == kTabBf16 && !kCentred;              // the bias term is an MMA of its own (see load_x)
  constexpr int kBiasMmas = kGroups == 16 ? 3 : kGroups == 8 ? 2 : 1;
  constexpr int kEntry = entry_bytes(TT);
  constexpr int kRowBytes = table_row_bytes(kGroups, TT);             // a weight row's table entries in a slice
  constexpr bool kQuads = table_quads(kGroups, TT), kTwice = sums_twice(QK, kGroups, TT, kCentred);
  constexpr int kSums = sums_bytes(1, kTwice);                        // the columns' sums of a group
  constexpr int kTable = table_bytes(kTileRows, kGroups, TT, kQuads); // one table of a tile
  constexpr int kEight = table_at(8, kGroups, TT, kQuads);            // its next eight rows
  // Rows of float32 entries in groups of 32 that do not start on 16 bytes: a word a lane. A word a copy of a row a lane is sixteen copies that touch 32 rows each (2 rows of 52352 x 5568 85.4 -> 69.0 us,
  // 28672 x 3200 29.2 -> 21.9, float32 activations 52083 x 5760 216 -> 159). Shorter rows are left to that: MXFP4 and 8-bit codes were up to 4 % slower so.
  constexpr bool kByWords = kRowBytes == 64;
  constexpr int kSlot = kStage + table_stage_bytes(R, kGroups, TT, kQuads);   // codes, scales, biases: a place of the ring
  constexpr float kUnit = QK == kMx4 ? 16384.0f : kNibbles && kCentred ? 64.0f : 1.0f;               // (the E2M1 fragments are the values times 2^-14)

  // The next launch may be made ready from here on: it touches nothing of this one's before its own wait, and the way from here to its CTAs' start is what
  // bounds the rate of small products (see the head of the file).
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ uint8_t rows_smem_raw[];
  const uint32_t smem = (smem_u32(rows_smem_raw) + 1023) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rho = ((g & 1) << 2) | (g & 2) | (g >> 2);                // weight row of MMA row g: bit-reversed, which makes the
                                                                      // swizzled reads of 4, 8 and 16 bytes free of bank conflicts
  const int csize = p.cluster;
  const int rank = csize > 1 ? static_cast<int>(cluster_rank()) : 0;

  // (every access below goes through 32-bit shared addresses)
  const uint32_t ring_at = smem + kHeadBytes + warp * p.ring * kStage;
  const uint32_t tables_at = smem + kHeadBytes + warps * p.ring * kStage + warp * p.ring * (kSlot - kStage);
  const uint32_t red_at = smem + kHeadBytes + warps * p.ring * kSlot;                           // [bufs][warps][R][32] float4
  const uint32_t xbuf_at = red_at + p.red_bufs * warps * R * 512;                          // [slots][cluster][R][32] float4
  const uint32_t own_at = xbuf_at + (csize > 1 ? kExchangeSlots * csize * R * 512 : 0);
  const uint32_t sums_at = own_at + warp * sums_bytes(kGroups, kTwice);                              // [warps] sums of x
  const uint32_t more_x_at = own_at + warps * sums_bytes(kGroups, kTwice) + warp * more_x_bytes(T) + lane * 16;      // [warps][MMA pairs][32] 16 bytes
  const uint32_t segs_at = own_at + warps * (sums_bytes(kGroups, kTwice) + more_x_bytes(T));         // grouped: [segs] chunks, [segs + 1] first rows
  int* seg_chunks = reinterpret_cast<int*>(rows_smem_raw + (segs_at - smem_u32(rows_smem_raw)));
  int* seg_row = seg_chunks + p.segs;
  uint8_t* head = rows_smem_raw + (smem - smem_u32(rows_smem_raw));
  const uint32_t my_full = smem + kFullAt + warp * kMaxRing * 8, abort_at = smem + kAbortAt;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(head + kAbortAt);
  Place* place = reinterpret_cast<Place*>(head + kStateAt + warp * 2 * kStateBytes);
  int* ahead_at = reinterpret_cast<int*>(head + kAheadAt) + warp * 2;

  if (lane == 0) {
    if (warp == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&w_map)) : "memory");
    *abort_flag = 0;
  }
  {
    auto init = [](uint32_t bar, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n)); };
    if (lane < p.ring) init(my_full + lane * 8, 1 + 32);               // the boxes, and every lane's table entries
    if (warp == 0) {                                                   // (a lane a barrier, of those that follow one another)
      static_assert(kRedEmptyAt == kRedFullAt + 32 && kXFullAt == kRedEmptyAt + 32 && kXFreeAt == kXFullAt + kExchangeSlots * 8 && kExchangeSlots * (kMaxCluster + 1) <= 24, "");
      if (lane < 8 + kExchangeSlots * (kMaxCluster + 1)) init(smem + kRedFullAt + lane * 8, lane < 4 ? warps : 1);
    }
    mbar_init_fence();
  }
  __syncwarp();

  // ---- which work is this CTA's: a contiguous share of (chunk, tile), tiles fastest ----
  const bool grouped = p.group_sizes != nullptr;
  const int dense_chunks = static_cast<int>((p.M + T - 1) / T);
  if (grouped || p.lhs_idx) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (grouped) {
    // chunks of every expert and the rows before it (at most p.M in all, as if the sizes were cut off there)
    for (int s = threadIdx.x; s < p.segs; s += blockDim.x) seg_row[s + 1] = p.group_sizes[s] > 0 ? p.group_sizes[s] : 0;
    __syncthreads();
    if (warp == 0) {
      int64_t before = 0;
      int chunks_before = 0;
      for (int s0 = 0; s0 < p.segs; s0 += 32) {
        const int s = s0 + lane;
        const int64_t own = s < p.segs ? seg_row[s + 1] : 0;
        int64_t run = own;
        for (int o = 1; o < 32; o <<= 1) {
          const int64_t v = __shfl_up_sync(0xffffffffu, run, o);
          if (lane >= o) run += v;
        }
        const int64_t lo = before + run - own < p.M ? before + run - own : p.M, hi = before + run < p.M ? before + run : p.M;
        const int c = static_cast<int>((hi - lo + T - 1) / T);
        __syncwarp();
        if (s < p.segs) {
          seg_chunks[s] = c;
          seg_row[s] = static_cast<int>(lo);
          if (s == p.segs - 1) seg_row[p.segs] = static_cast<int>(hi);
        }
        chunks_before += __reduce_add_sync(0xffffffffu, c);
        before += __shfl_sync(0xffffffffu, run, 31);
      }
      if (lane == 0) abort_flag[1] = chunks_before;
    }
    __syncthreads();
  }
  auto chunks_of = [&](int seg) -> int { return grouped ? seg_chunks[seg] : dense_chunks; };
  auto weight_row_of = [&](int seg) -> int {
    int64_t r = p.weight_rows ? seg : 0;
    if (p.rhs_idx) {
      r = p.rhs_idx[seg];
      if (r < 0 || r >= p.num_weights) {
        if (lane == 0) atomicCAS(p.status, 0, QMM_DEVICE_BAD_INDEX);
        r = 0;
      }
    }
    return static_cast<int>(r * p.N);
  };
  int left, tile0, seg0 = 0, chunk0;
  {
    const unsigned cluster = csize > 1 ? blockIdx.x / csize : blockIdx.x;
    unsigned share = p.share, more = p.share_more;                     // (32 bits all the way: a 64-bit division is a hundred instructions)
    if (grouped) {
      const unsigned total = static_cast<unsigned>(abort_flag[1]) * p.tiles, clusters = csize > 1 ? gridDim.x / csize : gridDim.x;
      share = total / clusters;
      more = total - share * clusters;
    }
    const unsigned lo = cluster * share + min(cluster, more);
    left = static_cast<int>(share + (cluster < more ? 1u : 0u));
    unsigned c = lo < static_cast<unsigned>(p.tiles) ? 0u : lo / p.tiles;
    tile0 = static_cast<int>(lo - c * p.tiles);
    if (grouped) {
      while (seg0 + 1 < p.segs && c >= static_cast<unsigned>(seg_chunks[seg0])) c -= seg_chunks[seg0++];
    } else if (p.segs > 1) {
      seg0 = static_cast<int>(c / dense_chunks);
      c -= static_cast<unsigned>(seg0) * dense_chunks;
    }
    chunk0 = static_cast<int>(c);
  }
  // the chunk after (seg, chunk); only asked while there is one
  auto next_chunk = [&](int& seg, int& chunk) {
    if (++chunk < chunks_of(seg)) return;
    chunk = 0;
    do { ++seg; } while (seg + 1 < p.segs && chunks_of(seg) == 0);
  };

  const bool pair = kMayPair && p.scales2 != nullptr;
  const int step_rows = pair ? kBlockRows : kTileRows;             // weight rows from a tile to the next

  // ---- the ring: boxes in the order they are consumed, a few ahead ----
  const int first_slice = rank * p.slices_per_cta + warp * p.slices_per_warp;
  int ahead_left = left * p.slices_per_warp, ahead_row = 0, ahead_last = 0, ahead_tiles = p.tiles - tile0, ahead_sub = 0;
  uint32_t ahead_slot = 0;
  if (left > 0) {
    ahead_row = weight_row_of(seg0);
    ahead_last = ahead_row + p.N - 1;
    ahead_row += tile0 * step_rows;
    if (lane == 0) { ahead_at[0] = seg0; ahead_at[1] = chunk0; }
    __syncwarp();
  }
  // (a slice past the end of K is given the row's first entries: what they multiply is zero)
  auto first_entry = [&](int slice) -> int { return slice * kGroups < p.groups ? slice * kGroups : 0; };
  constexpr bool kBothTables = R == 2 || TT == kTabE8;
  const int table_row = kTileRows == 32 ? lane : lane & 15, table_row_size = p.groups * kEntry;
  const uint8_t* my_table = static_cast<const uint8_t*>(kBothTables || lane < 16 ? p.scales : p.biases);
  // (where the word behind a row's entries goes)
  const int spare = kQuads && kEntry < 4 ? table_at(kTileRows, kGroups, TT, kQuads) + table_row * 4 - table_at(table_row, kGroups, TT, kQuads) : kRowBytes;
  const uint32_t my_tables = tables_at + table_at(table_row, kGroups, TT, kQuads) + (kBothTables || lane < 16 ? 0 : kTable);
  auto request = [&]() {               // the whole warp; ahead_left > 0
    const uint32_t bar = my_full + ahead_slot * 8;
    const int slice = first_slice + ahead_sub;
    if (lane == 0) {
      const uint32_t dst = ring_at + ahead_slot * kStage;
      mbar_expect_tx(bar, kStage);
#pragma unroll
      for (int b = 0; b < kBoxes; ++b) {
        tma_load_2d(&w_map, dst + b * kBoxSmem, bar, (slice * kBoxes + b) * kBoxBytes, ahead_row);
        if (pair) tma_load_2d(&w2_map, dst + b * kBoxSmem + kBlockRows * kBoxBytes, bar, (slice * kBoxes + b) * kBoxBytes, ahead_row);
      }
    }
    {
      // Entries past the end of a row are some other entry of it: what they multiply is zero.
      const uint32_t stage_at = ahead_slot * (kSlot - kStage);
      // a word a lane, the lanes of a row side by side
      auto words = [&]() {
        constexpr int kWords = kRowBytes / 4, kAtOnce = 32 / kWords, kStep = table_at(kAtOnce, kGroups, TT, kQuads);
        const int row = lane / kWords, word = lane % kWords * 4, first = first_entry(slice) * kEntry;
        const int from = first + (slice * kGroups * kEntry + word < table_row_size ? word : 0);
        const uint32_t dst = tables_at + stage_at + table_at(row, kGroups, TT, kQuads) + word;
        static_for<kTileRows / kAtOnce>([&](auto jc) {
          constexpr int j = decltype(jc)::value;
          const bool second = pair && j * kAtOnce >= kBlockRows;
          const int64_t at = static_cast<int64_t>(min(ahead_row + row + (second ? j * kAtOnce - kBlockRows : j * kAtOnce), ahead_last)) * table_row_size + from;
          cp_async4(dst + j * kStep, static_cast<const uint8_t*>(second ? p.scales2 : p.scales) + at);
          cp_async4(dst + j * kStep + kTable, static_cast<const uint8_t*>(second ? p.biases2 : p.biases) + at);
        });
      };
      // a lane's share: a weight row of one table, or (two blocks) of both
      auto rows = [&]() {
        const int64_t at = static_cast<int64_t>(min(ahead_row + (pair ? table_row & 15 : table_row), ahead_last)) * table_row_size + first_entry(slice) * kEntry;
        const bool second = pair && lane >= 16;
        const uint32_t dst = my_tables + stage_at;
        auto copy = [&](const uint8_t* table, uint32_t to) {
          const uint8_t* src = table + at;
          constexpr int kWhole = kQuads ? 16 : 8;
          if (kByWords || (p.table_unit >= kWhole && kRowBytes >= kWhole)) {
#pragma unroll
            for (int i = 0; i < kRowBytes; i += kWhole) {
              if constexpr (kQuads) cp_async16(to + i, src + i);
              else cp_async8(to + i, src + i);
            }
          } else if (kEntry == 4 || p.table_unit >= 4) {
#pragma unroll
            for (int i = 0; i < kRowBytes; i += 4) cp_async4(to + i, slice * kGroups * kEntry + i < table_row_size ? src + i : src);
          } else {                         // from the word the first entry lies in; nothing past the table's end is read
            const int skew = static_cast<int>(at & 3);
#pragma unroll
            for (int i = 0; i <= kRowBytes; i += 4) {
              const int64_t room = p.table_bytes - (at - skew + i);
              cp_async4(to + (i < kRowBytes ? i : spare), room > 0 ? src - skew + i : src - skew, room >= 4 ? 4 : room > 0 ? static_cast<int>(room) : 0);
            }
          }
        };
        if (kBothTables) {
          if (kTileRows == 32 || lane < 16) copy(static_cast<const uint8_t*>(second ? p.scales2 : p.scales), dst);
          if (TT != kTabE8) copy(static_cast<const uint8_t*>(second ? p.biases2 : p.biases), dst + kTable);
        } else {
          copy(my_table, dst);
        }
      };
      if (kByWords && p.table_unit == 4) words();
      else rows();
      cp_async_arrive(bar);
    }
    --ahead_left;
    if (++ahead_slot == static_cast<uint32_t>(p.ring)) ahead_slot = 0;
    if (p.slices_per_warp > 1) {
      if (++ahead_sub < p.slices_per_warp) return;
      ahead_sub = 0;
    }
    ahead_row += step_rows;
    if (--ahead_tiles == 0) {
      ahead_tiles = p.tiles;
      if (ahead_left > 0) {
        int seg = ahead_at[0], chunk = ahead_at[1];
        next_chunk(seg, chunk);
        ahead_row = weight_row_of(seg);
        ahead_last = ahead_row + p.N - 1;
        __syncwarp();
        if (lane == 0) { ahead_at[0] = seg; ahead_at[1] = chunk; }
        __syncwarp();
      }
    }
  };
  // (a warp past the end of K computes on zeros: its boxes are zero-filled)
  for (int i = 0; i < p.ring && ahead_left > 0; ++i) request();

  auto set_place = [&](int which, int seg, int chunk) {               // the whole warp
    const int rows = grouped ? seg_row[seg + 1] - seg_row[seg] : static_cast<int>(p.M);
    const int weight_row = weight_row_of(seg);
    __syncwarp();
    if (lane == 0) {
      Place pl;
      const int64_t m0 = static_cast<int64_t>(chunk) * T;
      pl.y0 = grouped ? (seg_row[seg] + m0) * p.N : seg * p.y_batch_stride + m0 * p.N;
      pl.seg = seg;
      pl.chunk = chunk;
      pl.rows_left = rows - chunk * T;
      pl.weight_row = weight_row;
      place[which] = pl;
    }
    __syncwarp();
  };
  if (left > 0) set_place(0, seg0, chunk0);
  __syncthreads();                                 // the shared barriers are initialised
  if (csize > 1) {                                 // ... in every CTA of the cluster
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (!grouped && !p.lhs_idx) asm volatile("griddepcontrol.wait;" ::: "memory");

  // ---- activations: this warp's slice as MMA fragments ----
  static_assert(NT <= 2, "one column group in registers, one in shared memory");
  uint32_t xf[kSliceK / 8];                        // column group 0: two registers per MMA of the slice
  // The bias term sum_g bias[n, g] sum x_g of a slice is an MMA of 16 K slots: bias entries as they are in the table
  // (bf16) against the groups' sums of x, each split into three bf16 pieces (24 bits) that take a slot of their own.
  [[maybe_unused]] uint32_t bf[kBiasMmas][2];
  float back[2];                                   // what a unit of the scaled activations of output columns 2t, 2t + 1 is worth
  back[0] = back[1] = 1.0f;
  [[maybe_unused]] uint32_t least_e = 15u;
  auto load_x = [&](const Place& pl, int slice, int sub) {
    int64_t base = 0;
    if (!grouped) {
      int64_t b = pl.seg;
      if (p.lhs_idx) {
        b = p.lhs_idx[pl.seg];
        if (b < 0 || (p.x_batches > 0 && b >= p.x_batches)) {
          if (lane == 0) atomicCAS(p.status, 0, QMM_DEVICE_BAD_INDEX);
          b = 0;
        }
      }
      base = b * p.x_batch_stride;
    }
    __syncwarp();                                  // (the sums below may still be read)
    const int m = kHalf ? g & 3 : g;
    const bool live = m < pl.rows_left;
    int64_t xr = pl.chunk * T + m;
    if (grouped && live) {
      xr += seg_row[pl.seg];
      if (p.x_rows) {
        xr = p.x_rows[xr];
        if (xr < 0 || xr >= p.total_x_rows) {
          if (t == 0) atomicCAS(p.status, 0, QMM_DEVICE_BAD_INDEX);
          xr = 0;
        }
      }
    }
    const XT* src = reinterpret_cast<const XT*>(p.x) + base + (live ? xr : 0) * p.K;
    const int k0 = slice * kSliceK + t * kLane;
    auto element_of = [&](int c) -> int { return k0 + (c / (kLane / 8)) * kBlk + (c % (kLane / 8)) * 8; };      // the lane's c-th eight elements
    auto arranged = [](uint32_t (&u)[4]) {         // in the order in which codes come apart: (0,4) (1,5) (2,6) (3,7) of 4 bits, (0,1) (2,3) of 8
      if constexpr (QK != kAff8) {
        const uint32_t v[4] = {u[0], u[1], u[2], u[3]};
        u[0] = __byte_perm(v[0], v[2], 0x5410); u[1] = __byte_perm(v[0], v[2], 0x7632);
        u[2] = __byte_perm(v[1], v[3], 0x5410); u[3] = __byte_perm(v[1], v[3], 0x7632);
      }
    };
    constexpr int kPer = kSliceK / 32 / kGroups;   // eights per group
    auto sum_at = [](int column) -> int { return kTwice ? (column >> 1) * 16 + (column & 1) * 4 : column * 4; };
    if constexpr (kPieces == 1) {
      // 16-bit activations: fragments as they are (or scaled), and the groups' sums of them in float32, by additions that take a 16-bit operand and
      // round. (Conversions and additions of float32 took 800 instructions a warp, 2 us of every launch. MMAs of the fragments against ones are 0.1 us faster in
      // small launches, but each cuts off: activations of 22 binades and both signs were 14 % further from the exact sums, and 8-bit codes against bf16 spilled
      // up to 232 bytes, 8 rows of 14336 x 4096 in groups of 64 with f16 tables 16.8 us instead of 13.7.)
      // (all of the lane's elements are asked for at once: a trip to L2 is a third of what this takes)
      constexpr int kPart = kSliceK / 32;
      uint4 v[kPart];
#pragma unroll
      for (int c = 0; c < kPart; ++c) {
        const int k = element_of(c);
        v[c] = live && k < p.K ? __ldg(reinterpret_cast<const uint4*>(src + k)) : make_uint4(0u, 0u, 0u, 0u);
      }
      float up = 1.0f;
      if constexpr (kScaled) {
        // largest finite magnitude of the row's slice (of a pair of bf16 patterns, as whole numbers)
        auto over_row = [&](uint32_t big) -> uint32_t {
          big = max(big & 0xffffu, big >> 16);
          big = max(big, __shfl_xor_sync(0xffffffffu, big, 1));
          return max(big, __shfl_xor_sync(0xffffffffu, big, 2));
        };
        auto largest = [&](auto finite) -> uint32_t {
          uint32_t pair = 0u;
#pragma unroll
          for (int c = 0; c < kPart; ++c) {
            const uint32_t u[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t m = u[j] & 0x7fff7fffu;
              if (decltype(finite)::value) m = ((m & 0xffffu) >= 0x7f80u ? 0u : m & 0xffffu) | (m >= 0x7f800000u ? 0u : m & 0xffff0000u);
              pair = __vmaxu2(pair, m);
            }
          }
          return over_row(pair);
        };
        uint32_t big = largest(std::false_type());
        if (__any_sync(0xffffffffu, big >= 0x7f80u)) big = largest(std::true_type());      // an infinity or a NaN somewhere
        // largest magnitude to [2^14, 2^15); a warp's later slices no finer than its earlier ones, whose sums are brought to their units
        const uint32_t e = max(big >> 7, sub > 0 ? least_e : 15u);
        least_e = e;
        up = __uint_as_float((268u - e) << 23);
        const float down = __uint_as_float((e - 14u) << 23);
        back[0] = __shfl_sync(0xffffffffu, down, 8 * t);
        back[1] = __shfl_sync(0xffffffffu, down, 8 * t + 4);
      }
      float sum = 0.0f;
#pragma unroll
      for (int c = 0; c < kPart; ++c) {
        uint32_t u[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
        if constexpr (kScaled) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = unpack2<XT>(u[j]);
            u[j] = pack2<AT>(f.x * up, f.y * up);
          }
        }
        if constexpr (QK != kMx4) {
#pragma unroll
          for (int j = 0; j < 4; ++j) sum = add_pair<AT>(sum, u[j]);
          if (c % kPer == kPer - 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            // (kept as -C sum x where the group's accumulators start there)
            if (t < (kTwice ? 2 : 1)) sts32(sums_at + (c / kPer) * kSums + sum_at(g) + t * 8, kSumIs * sum);
            sum = 0.0f;
          }
        }
        arranged(u);
        if constexpr (kQuarters) {               // (what goes with the codes that are (128 + q) / 4)
          u[1] = fma_bf16(u[1], 0x40804080u, 0x80008000u);
          u[3] = fma_bf16(u[3], 0x40804080u, 0x80008000u);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) xf[c * 4 + j] = u[j];
      }
    } else {
      auto load8 = [&](int c, float (&f)[8]) {
        const int k = element_of(c);
        if (live && k < p.K) {
          const float4 a = __ldg(reinterpret_cast<const float4*>(src + k)), b = __ldg(reinterpret_cast<const float4*>(src + k) + 1);
          f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = 0.0f;
        }
      };
      float up = 1.0f;
      [[maybe_unused]] bool infinite = false;      // some row's slice has an infinity in it
      if constexpr (kScaled) {
        auto largest = [&](auto finite) -> float {
          float big = 0.0f;                                            // (a NaN is no larger than anything, and one in any unit)
#pragma unroll
          for (int c = 0; c < kSliceK / 32; ++c) {
            float f[8];
            load8(c, f);
#pragma unroll
            for (int i = 0; i < 8; ++i) big = fmaxf(big, !decltype(finite)::value || fabsf(f[i]) <= kMaxFloat ? fabsf(f[i]) : 0.0f);
          }
          big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 1));
          return fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 2));
        };
        float big = largest(std::false_type());
        if (__any_sync(0xffffffffu, big > kMaxFloat)) {
          infinite = true;
          big = largest(std::true_type());
        }
        // largest magnitude to [2^14, 2^15); a warp's later slices no finer than its earlier ones, whose sums are brought to their units
        const uint32_t e = max(__float_as_uint(big) >> 23, sub > 0 ? least_e : 15u);
        least_e = e;
        up = __uint_as_float((268u - e) << 23);
        const float down = __uint_as_float((e - 14u) << 23);
        back[0] = __shfl_sync(0xffffffffu, down, 8 * t);
        back[1] = __shfl_sync(0xffffffffu, down, 8 * t + 4);
      }
      // CAREFUL: the second piece of an infinity is nought (it would be a NaN), for its results to be what a sum of products makes of them. (A
      // comparison for every element costs a scaled row more than what its largest magnitude already tells: 33 rows of float32 against MXFP4,
      // 4096 x 4096, 98 us with it everywhere, 74 so; 69 without.)
      auto fragments = [&](auto careful) {
        float sum = 0.0f;
#pragma unroll
        for (int c = 0; c < kSliceK / 32; ++c) {
          float f[8];
          load8(c, f);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if constexpr (kScaled) f[i] *= up;
            sum += f[i];
          }
          if constexpr (QK != kMx4) {
            if (c % kPer == kPer - 1) {
              sum += __shfl_xor_sync(0xffffffffu, sum, 1);
              sum += __shfl_xor_sync(0xffffffffu, sum, 2);
              // (kept as -C sum x where the group's accumulators start there)
              if (t < (kTwice ? 2 : 1)) sts32(sums_at + (c / kPer) * kSums + sum_at(g) + t * 8, kSumIs * sum);
              sum = 0.0f;
            }
          }
          [[maybe_unused]] uint32_t frag[4];
#pragma unroll
          for (int i = 0; i < kPieces; ++i) {
            const bool here = !kHalf || (g >> 2) == (i & 1);             // (4 tokens: which of the two pieces this lane's column is)
            uint32_t u[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) u[j] = pack2<AT>(f[2 * j], f[2 * j + 1]);
            if (i + 1 < kPieces) {                                       // what this piece leaves over (exact)
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 got = unpack2<AT>(u[j]);
                if (decltype(careful)::value && i == 0) {
                  f[2 * j] = left_of(f[2 * j], got.x); f[2 * j + 1] = left_of(f[2 * j + 1], got.y);
                } else {
                  f[2 * j] -= got.x; f[2 * j + 1] -= got.y;
                }
              }
            }
            arranged(u);
            if (kHalf) {                                                 // (the half of the last group that no piece is left for: nought)
#pragma unroll
              for (int j = 0; j < 4; ++j) frag[j] = here ? u[j] : i % 2 ? frag[j] : 0u;
              if (i == 1) {
#pragma unroll
                for (int j = 0; j < 4; ++j) xf[c * 4 + j] = frag[j];
              } else if (i + 1 == kPieces) {
                sts128(more_x_at + c * 512, __uint_as_float(frag[0]), __uint_as_float(frag[1]), __uint_as_float(frag[2]), __uint_as_float(frag[3]));
              }
            }
          }
        }
      };
      if constexpr (!kScaled) {
        fragments(std::true_type());
      } else {
        if (infinite) fragments(std::true_type());
        else fragments(std::false_type());
      }
    }
    __syncwarp();                                  // the sums are there
    if constexpr (kBiasMma) {
      // K slots of the bias MMAs: 16 groups -- one MMA per piece of the sums (lane t: groups 2t, 2t + 1, 2t + 8, 2t + 9);
      // 8 groups -- (hi | mid) and (lo | 0) with lane t's groups 2t, 2t + 1; 4 groups -- lanes t < 2 (hi | mid), t >= 2 (lo | 0)
      // with groups 2 (t & 1), 2 (t & 1) + 1
      auto pick = [&](int first) -> float {        // sum of x of column g in group first + 2 t
        return __uint_as_float(lds32<0>(sums_at + (first + 2 * (kGroups == 4 ? t & 1 : t)) * kSums + sum_at(g))) * (1.0f / kSumIs);
      };
      using B16 = __nv_bfloat16;
      auto split = [&](float a, float b, uint32_t (&piece)[3]) {
        piece[0] = pack2<B16>(a, b);
        const float2 f0 = unpack2<B16>(piece[0]);
        const float a1 = left_of(a, f0.x), b1 = left_of(b, f0.y);
        piece[1] = pack2<B16>(a1, b1);
        const float2 f1 = unpack2<B16>(piece[1]);
        piece[2] = pack2<B16>(a1 - f1.x, b1 - f1.y);
      };
      uint32_t lower[3];
      split(pick(0), pick(1), lower);
      if constexpr (kGroups == 16) {
        uint32_t upper[3];
        split(pick(8), pick(9), upper);
#pragma unroll
        for (int i = 0; i < 3; ++i) { bf[i][0] = lower[i]; bf[i][1] = upper[i]; }
      } else if constexpr (kGroups == 8) {
        bf[0][0] = lower[0]; bf[0][1] = lower[1];
        bf[kBiasMmas - 1][0] = lower[2]; bf[kBiasMmas - 1][1] = 0u;
      } else {
        bf[0][0] = t < 2 ? lower[0] : lower[2]; bf[0][1] = t < 2 ? lower[1] : 0u;
      }
    }
    __syncwarp();
  };

  // ---- the tiles ----
  // A lane's bytes of block 0 of row rho in a slot; block j is at this address XOR its chunk term.
  const uint32_t wthread = ring_at + rho * kBoxBytes +
                           (QK == kAff8 ? (SPG == 1 ? ((((t >> 1) ^ rho) << 4) + (t & 1) * 8) : ((t ^ rho) << 4))
                                        : (SPG == 1 ? ((rho << 4) + t * 4) : ((((t >> 1) ^ rho) << 4) + (t & 1) * 8)));
  uint32_t nib_mask = std::is_same<AT, __half>::value ? 0x03C003C0u : 0x000F000Fu, magic = kMagic;
  [[maybe_unused]] uint32_t upper_mask = 0x00F000F0u, times = 0x7F007F00u;       // (2^127)
  asm volatile("" : "+r"(nib_mask), "+r"(magic));                      // constants in registers: one LOP3 per use
  const uint32_t tthread = tables_at + table_at(rho, kGroups, TT, kQuads), scol = sums_at + (kTwice ? 16 : 8) * t;
  int turn = 0, which = 0, tile = tile0, sub = 0, count = 0;
  uint32_t slot = 0, slot_phase = 0, buf = 0, buf_phase = 0;
  // the tile that is to be added up next
  int done_tile = 0, done_which = 0, lap = 0, leader = 0;
  uint32_t done_buf = 0, done_phase = 0;
  auto store_tile = [&](const float (&v)[R][4], int64_t y0, int rows_left, int at_tile) {
    if (pair) {                                    // rounded as products, gate and their product are when each is a launch of its own
      auto gated = [&](auto type, int i) {
        using YT = decltype(type);
        const float gate = static_cast<float>(static_cast<YT>(v[0][i])), up = static_cast<float>(static_cast<YT>(v[1][i]));
        return static_cast<float>(static_cast<YT>(gate / (1.0f + __expf(-gate)))) * up;
      };
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = 2 * t + (i & 1), n = at_tile * kBlockRows + rho + (i >> 1) * 8;
        if (col < rows_left && n < p.N)
          store_y(p.y, p.y_dtype, y0 + static_cast<int64_t>(col) * p.N + n, p.y_dtype == QMM_BF16 ? gated(__nv_bfloat16(), i) : gated(__half(), i));
      }
      return;
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = 2 * t + (i & 1), n = at_tile * kTileRows + r * kBlockRows + rho + (i >> 1) * 8;
        if (col < rows_left && col < T && n < p.N) store_y(p.y, p.y_dtype, y0 + static_cast<int64_t>(col) * p.N + n, v[r][i]);
      }
  };
  // A tile that this CTA leads: the CTAs' sums in rank order.
  auto finish = [&](int led) -> bool {
    const int xs = led % kExchangeSlots;
    if (!mbar_wait_cluster(smem + kXFullAt + xs * 8, static_cast<uint32_t>(led / kExchangeSlots) & 1u, abort_at, 15)) return false;
    __syncwarp();
    const uint32_t xslot = xbuf_at + xs * csize * (R * 512) + lane * 16;
    float v[R][4];
#pragma unroll
    for (int h = 0; h < R; ++h) v[h][0] = v[h][1] = v[h][2] = v[h][3] = 0.0f;
    for (int r = 0; r < csize; ++r)
#pragma unroll
      for (int h = 0; h < R; ++h) {
        const float4 f = ldsf128<0>(xslot + (r * R + h) * 512);
        v[h][0] += f.x; v[h][1] += f.y; v[h][2] += f.z; v[h][3] += f.w;
      }
    const uint4 to = lds128<kLedAt>(smem + xs * 16);
    __syncwarp();
    if (lane < csize && lane != rank) remote_arrive(remote(smem + kXFreeAt + (rank * kExchangeSlots + xs) * 8, lane));
    store_tile(v, static_cast<int64_t>(static_cast<uint64_t>(to.y) << 32 | to.x), static_cast<int>(to.z), static_cast<int>(to.w));
    return true;
  };
  auto add_up = [&]() -> bool {
    // ---- the warps' shares, in warp order ----
    const uint32_t shares = red_at + done_buf * warps * (R * 512) + lane * 16;
    if (!mbar_wait(smem + kRedFullAt + done_buf * 8, done_phase, abort_at, 13)) return false;
    __syncwarp();
    float v[R][4];
#pragma unroll
    for (int h = 0; h < R; ++h) v[h][0] = v[h][1] = v[h][2] = v[h][3] = 0.0f;
#pragma unroll 4
    for (int i = 0; i < warps; ++i)
#pragma unroll
      for (int h = 0; h < R; ++h) {
        const float4 f = ldsf128<0>(shares + (i * R + h) * 512);
        v[h][0] += f.x; v[h][1] += f.y; v[h][2] += f.z; v[h][3] += f.w;
      }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem + kRedEmptyAt + done_buf * 8);
    const int rows_left = place[done_which].rows_left;
    const int64_t y0 = place[done_which].y0;
    if (csize == 1) {
      store_tile(v, y0, rows_left, done_tile);
      return true;
    }
    // ---- the CTAs' sums meet at the tile's leader (in turn; `lap` counts its tiles), who adds them up when its next tile comes: by then they are there ----
    const int xs = lap % kExchangeSlots;
    const uint32_t xslot = xbuf_at + xs * csize * (R * 512) + lane * 16;
    if (leader != rank) {
      if (!mbar_wait_cluster(smem + kXFreeAt + (leader * kExchangeSlots + xs) * 8, (static_cast<uint32_t>(lap / kExchangeSlots) & 1u) ^ 1u, abort_at, 14)) return false;
      __syncwarp();
      const uint32_t bar = remote(smem + kXFullAt + xs * 8, leader), to = remote(xslot + rank * (R * 512), leader);
#pragma unroll
      for (int h = 0; h < R; ++h) st_async4(to + h * 512, bar, v[h]);
      return true;
    }
    if (lap > 0 && !finish(lap - 1)) return false;
#pragma unroll
    for (int h = 0; h < R; ++h) sts128(xslot + rank * (R * 512) + h * 512, v[h][0], v[h][1], v[h][2], v[h][3]);
    if (lane == 0)
      sts128(smem + kLedAt + xs * 16, __uint_as_float(static_cast<uint32_t>(y0)), __uint_as_float(static_cast<uint32_t>(y0 >> 32)), __int_as_float(rows_left), __int_as_float(done_tile));
    __syncwarp();
    if (lane == 0) mbar_expect_tx(smem + kXFullAt + xs * 8, (csize - 1) * R * 512);      // (what finishes the tile sees the above as well)
    return true;
  };
  bool ok = true, stale = true;
  float y[R][NT][4];                               // per column group: sums of scale * codes * digits
  [[maybe_unused]] float yb[R][4];                 // ... and, where it is no MMA, the bias term per output column
  while (left > 0) {
    if (stale) {
      const float unit[2] = {back[0], back[1]};
      load_x(place[which], first_slice + sub, sub);
      if (kScaled && sub > 0) {                    // the sums so far in the new slice's units (a power of two)
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int h = 0; h < NT; ++h) {
              // (with 4 tokens the upper lanes' columns are the lower lanes' tokens)
              float u0 = unit[i & 1] / back[i & 1];
              if (kHalf) u0 = __shfl_sync(0xffffffffu, u0, lane & ~2);
              y[r][h][i] *= u0;
            }
            if constexpr (QK != kMx4) yb[r][i] *= unit[i & 1] / back[i & 1];
          }
      }
      stale = p.slices_per_warp > 1;
    }
    if (sub == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int h = 0; h < NT; ++h) y[r][h][0] = y[r][h][1] = y[r][h][2] = y[r][h][3] = 0.0f;
        yb[r][0] = yb[r][1] = yb[r][2] = yb[r][3] = 0.0f;
      }
    }
    // where this warp goes next
    const bool last_sub = sub + 1 == p.slices_per_warp;
    const bool wraps = last_sub && tile + 1 == p.tiles;
    const int next_tile = !last_sub ? tile : (wraps ? 0 : tile + 1);

    if (!(ok = mbar_wait(my_full + slot * 8, slot_phase, abort_at, 11))) break;
    __syncwarp();
    const uint32_t wrow = wthread + slot * kStage, trow = tthread + slot * (kSlot - kStage);
    if (kEntry < 4 && p.table_unit < 4) {          // entries that do not start on words: shifted to where they would, once per tile
      const int row = kTileRows == 32 ? lane : lane & 15;
      auto straighten = [&](uint32_t at) {
        const int wr = place[which].weight_row + min(tile * step_rows + (pair ? row & 15 : row), p.N - 1);
        const uint32_t skew = ((static_cast<uint32_t>(wr) * static_cast<uint32_t>(p.groups) + first_entry(first_slice + sub)) * kEntry & 3u) * 8;
        uint32_t word = lds32<0>(at);
#pragma unroll
        for (int i = 0; i < kRowBytes; i += 4) {
          const uint32_t next = lds32<0>(at + (i + 4 < kRowBytes ? i + 4 : spare));
          sts32(at + i, __uint_as_float(__funnelshift_r(word, next, skew)));
          word = next;
        }
      };
      const uint32_t at = tables_at + slot * (kSlot - kStage) + table_at(row, kGroups, TT, kQuads);
      if (R == 2 || TT == kTabE8) {
        if (kTileRows == 32 || lane < 16) straighten(at);
        if (TT != kTabE8) straighten(at + kTable);
      } else {
        straighten(at + (lane < 16 ? 0 : kTable));
      }
      __syncwarp();
    }
    if constexpr (kBiasMma) {
      static_for<R>([&](auto rc) {
        constexpr int r = decltype(rc)::value, kAt = kTable + r * 2 * kEight;
        const uint32_t at = trow + (kGroups == 4 ? t & 1 : t) * 4;
        const uint32_t b0 = lds32<kAt>(at), b1 = lds32<kAt + kEight>(at);
        uint32_t a[4] = {b0, b1, b0, b1};
        if constexpr (kGroups == 16) { a[2] = lds32<kAt + 16>(at); a[3] = lds32<kAt + kEight + 16>(at); }
#pragma unroll
        for (int i = 0; i < kBiasMmas; ++i) Mma<__nv_bfloat16>::run(yb[r], a, bf[i][0], bf[i][1]);
      });
    }
    // Chunks of 64 codes; a chunk's codes are requested while the one before it is worked on.
    constexpr int kChunks = kSliceK / 64;
    uint32_t cw[2][R][2][kChunkWords];
    auto fetch = [&](auto qc, auto& c) {
      static_for<kChunkBlocks>([&](auto bc) {
        constexpr int jj = decltype(bc)::value, j = decltype(qc)::value * kChunkBlocks + jj;  // block of the slice
        constexpr int kLaneWords = kLane * kBits / 32;
        constexpr int kPerBox = kBoxBytes * 8 / kBits / kBlk, kBlkBytes = kBlk * kBits / 8;   // blocks of a box, bytes of a row in a block
        constexpr int kBoxAt = (j / kPerBox) * kBoxSmem;
        const uint32_t a0 = wrow ^ ((j % kPerBox) * kBlkBytes);
        static_for<2 * R>([&](auto rc) {
          constexpr int r = decltype(rc)::value / 2, i = decltype(rc)::value % 2, kRow = kBoxAt + (r * kBlockRows + i * 8) * kBoxBytes;      // rows rho and rho + 8 of block r
          uint32_t* u = &c[r][i][jj * kLaneWords];
          if constexpr (kLaneWords == 1) {
            u[0] = lds32<kRow>(a0);
          } else if constexpr (kLaneWords == 2) {
            const uint2 v = lds64<kRow>(a0);
            u[0] = v.x; u[1] = v.y;
          } else {
            const uint4 v = lds128<kRow>(a0);
            u[0] = v.x; u[1] = v.y; u[2] = v.z; u[3] = v.w;
          }
        });
      });
    };
    fetch(std::integral_constant<int, 0>(), cw[0]);
    static_for<2>([&](auto hc) {
      constexpr int half = decltype(hc)::value;
      const uint32_t thalf = trow + half * (kHalfGroups * kEntry), shalf = scol + half * (kHalfGroups * kSums);
      float acc[R][NT][4], start[4];
      constexpr bool kStarts = QK != kMx4 && !kCentred;
      const float nought[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      // (16-bit and 8-bit entries of the half's groups, rows rho and rho + 8)
      constexpr int kHalfWords = kEntry < 4 ? kHalfGroups * kEntry / 4 : 0;
      [[maybe_unused]] uint32_t sw[R][2][kHalfWords ? kHalfWords : 1];
      static_for<kHalfWords ? 2 * R : 0>([&](auto ic) {
        constexpr int r = decltype(ic)::value / 2, i = decltype(ic)::value % 2, kAt = r * 2 * kEight + i * kEight;
        if constexpr (kHalfWords == 1) {
          sw[r][i][0] = lds32<kAt>(thalf);
        } else {
          static_for<kHalfWords / 2>([&](auto jc) {
            constexpr int j = decltype(jc)::value;
            const uint2 v = lds64<kAt + j * 8>(thalf);
            sw[r][i][2 * j] = v.x; sw[r][i][2 * j + 1] = v.y;
          });
        }
      });
      static_for<4>([&](auto qc) {
        constexpr int q = decltype(qc)::value, qq = half * 4 + q;
        auto& c = cw[q % 2];
        if constexpr (qq + 1 < kChunks) fetch(std::integral_constant<int, qq + 1>(), cw[(q + 1) % 2]);
        [[maybe_unused]] uint4 more = make_uint4(0u, 0u, 0u, 0u);
        static_for<4>([&](auto mc) {
          constexpr int m = decltype(mc)::value;                       // MMA of the chunk
          constexpr int kPerGroup = 2 * SPG, at = q * 4 + m, gi = at / kPerGroup;      // MMAs of a group; MMA and group of the half
          constexpr bool kFirst = at % kPerGroup == 0, kLast = at % kPerGroup == kPerGroup - 1;
          if constexpr (kFirst && QK != kMx4) {    // kSumIs * sum x of the group
            if constexpr (kTwice) {
              const float4 sr = ldsf128<gi * kSums>(shalf);
              start[0] = sr.x; start[1] = sr.y; start[2] = sr.z; start[3] = sr.w;
            } else {
              const uint2 sr = lds64<gi * kSums>(shalf);
              start[0] = start[2] = __uint_as_float(sr.x); start[1] = start[3] = __uint_as_float(sr.y);
            }
          }
          if constexpr (NT > 1 && m % 2 == 0) more = lds128<((qq * 4 + m) / 2) * 512>(more_x_at);
          static_for<R>([&](auto rc) {
            constexpr int r = decltype(rc)::value;
            uint32_t a[4];
            if constexpr (QK == kAff8) {                                  // one word: codes (0,1) and (2,3)
              const uint32_t v0 = c[r][0][m], v1 = c[r][1][m];
              a[0] = __byte_perm(v0, 0x64646464u, 0x4140); a[1] = __byte_perm(v1, 0x64646464u, 0x4140);
              a[2] = __byte_perm(v0, 0x64646464u, 0x4342); a[3] = __byte_perm(v1, 0x64646464u, 0x4342);
            } else {                                                      // half a word: nibbles (0,4) (1,5), or (2,6) (3,7)
              const uint32_t v0 = c[r][0][m / 2], v1 = c[r][1][m / 2];
              constexpr int n0 = (m & 1) * 2;
              if constexpr (kNibbles) {            // bytes 0 and 2 of the word, then 1 and 3
                const uint32_t b0 = m & 1 ? v0 >> 8 : v0, b1 = m & 1 ? v1 >> 8 : v1;
                if constexpr (kCentred) {
                  a[0] = fma_bf16(b0 & nib_mask, times, 0xBE00BE00u);
                  a[1] = fma_bf16(b1 & nib_mask, times, 0xBE00BE00u);
                  a[2] = fma_bf16(b0 & upper_mask, 0x7D007D00u, 0xBE00BE00u);      // 2^123
                  a[3] = fma_bf16(b1 & upper_mask, 0x7D007D00u, 0xBE00BE00u);
                } else {
                  a[0] = and_or(b0, nib_mask, magic);
                  a[1] = and_or(b1, nib_mask, magic);
                  a[2] = fma_bf16(b0 & upper_mask, times, 0x42004200u);            // 32
                  a[3] = fma_bf16(b1 & upper_mask, times, 0x42004200u);
                }
              } else if constexpr (QK == kAff4) {
                auto codes = [&](uint32_t v, int nib) -> uint32_t {
                  const int right = 4 * nib - (std::is_same<AT, __half>::value ? 6 : 0);
                  return and_or(right < 0 ? v << -right : v >> right, nib_mask, magic);
                };
                a[0] = codes(v0, n0);     a[1] = codes(v1, n0);
                a[2] = codes(v0, n0 + 1); a[3] = codes(v1, n0 + 1);
              } else {
                // magnitude bits of an E2M1 code at f16's exponent / mantissa boundary (the value times 2^-14,
                // the subnormal 0.5 included), its sign at the sign
                auto place_bits = [](uint32_t v, int nib) -> uint32_t {
                  const uint32_t mag = nib == 3 ? v >> 3 : v << (9 - 4 * nib);
                  return (mag & 0x0E000E00u) | ((v << (12 - 4 * nib)) & 0x80008000u);
                };
                a[0] = place_bits(v0, n0); a[1] = place_bits(v1, n0); a[2] = place_bits(v0, n0 + 1); a[3] = place_bits(v1, n0 + 1);
              }
            }
            if constexpr (kCentred && !kNibbles) {
#pragma unroll
              for (int i = 0; i < 4; ++i) a[i] = centred<AT>(a[i], kMagicValue + kCentre);
            }
#pragma unroll
            for (int h = 0; h < NT; ++h) {
              const uint32_t x0 = h ? (m & 1 ? more.z : more.x) : xf[(qq * 4 + m) * 2], x1 = h ? (m & 1 ? more.w : more.y) : xf[(qq * 4 + m) * 2 + 1];
              if constexpr (kFirst && kStarts)      // (what keeps the magic number has one piece)
                Mma<AT>::first(acc[r][h], a, x0, x1, start);
              else if constexpr (kFirst)
                Mma<AT>::first(acc[r][h], a, x0, x1, nought);
              else
                Mma<AT>::run(acc[r][h], a, x0, x1);
            }
          });
          if constexpr (kLast) {
            // fold the group: rows rho (acc 0, 1) and rho + 8 (acc 2, 3), columns 2t and 2t + 1
            static_for<R>([&](auto rc) {
              constexpr int r = decltype(rc)::value;
              constexpr int kWord = gi * kEntry / 4;
              [[maybe_unused]] constexpr int kIn = gi * kEntry % 4;
              constexpr int kAt = r * 2 * kEight + kWord * 4, kAt8 = kAt + kEight;      // rows rho and rho + 8
              auto value = [](uint32_t w) -> float {
                if constexpr (TT == kTabE8) return __uint_as_float(max(((w >> (8 * kIn)) & 0xffu) << 23, 0x00400000u));      // 2^(e8 - 127)
                else if constexpr (TT == kTabF32) return __uint_as_float(w);
                else if constexpr (TT == kTabBf16) return __uint_as_float(kIn ? (w & 0xffff0000u) : (w << 16));
                else return table_value(kIn ? w >> 16 : w & 0xffffu, QMM_F16);
              };
              float s0, s1;
              if constexpr (kHalfWords > 0) {
                s0 = value(sw[r][0][kWord]); s1 = value(sw[r][1][kWord]);
              } else {
                s0 = value(lds32<kAt>(thalf)); s1 = value(lds32<kAt8>(thalf));
              }
#pragma unroll
              for (int h = 0; h < NT; ++h) {
                fma2(y[r][h][0], y[r][h][1], s0, acc[r][h][0], acc[r][h][1]);
                fma2(y[r][h][2], y[r][h][3], s1, acc[r][h][2], acc[r][h][3]);
              }
              if constexpr (QK != kMx4 && !kBiasMma) {
                float b0 = value(lds32<kTable + kAt>(thalf)), b1 = value(lds32<kTable + kAt8>(thalf));
                if constexpr (kCentred) {
                  b0 = fmaf(kCentre, s0, b0); b1 = fmaf(kCentre, s1, b1);
                } else {
                  b0 *= 1.0f / kSumIs; b1 *= 1.0f / kSumIs;
                }
                fma2(yb[r][0], yb[r][1], b0, start[0], start[1]);
                fma2(yb[r][2], yb[r][3], b1, start[0], start[1]);
              }
            });
          }
        });
      });
    });
    // every read of the slot has been consumed above: the warp's next box may land in it
    __syncwarp();
    if (ahead_left > 0) request();
    if (++slot == static_cast<uint32_t>(p.ring)) { slot = 0; slot_phase ^= 1u; }
    if (!last_sub) {
      ++sub;
      continue;
    }
    sub = 0;

    // ---- this warp's share of the tile ----
    if (!(ok = mbar_wait(smem + kRedEmptyAt + buf * 8, buf_phase ^ 1u, abort_at, 12))) break;
    // the pieces of a column together, the bias term, the scale
    const uint32_t rbuf = red_at + (buf * warps + warp) * (R * 512) + lane * 16;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float s = y[r][NT - 1][i];
#pragma unroll
        for (int h = NT - 2; h >= 0; --h) s += y[r][h][i];
        if constexpr (kHalf) s += __shfl_xor_sync(0xffffffffu, s, 2);
        v[i] = fmaf(s, kUnit, yb[r][i]) * back[i & 1];
      }
      sts128(rbuf + r * 512, v[0], v[1], v[2], v[3]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem + kRedFullAt + buf * 8);
    // the tile before this one: its shares have all been written by now, or nearly (adding up this very tile would make each adder wait
    // for the warp that has just been one: a tile then costs its codes plus the adding up)
    if (warp == turn && count > 0 && !(ok = add_up())) break;
    done_tile = tile;
    done_which = which;
    if (count > 0) {
      if (++turn == warps) turn = 0;
      if (++done_buf == static_cast<uint32_t>(p.red_bufs)) { done_buf = 0; done_phase ^= 1u; }
      if (++leader == csize) { leader = 0; ++lap; }
    }
    ++count;
    if (++buf == static_cast<uint32_t>(p.red_bufs)) { buf = 0; buf_phase ^= 1u; }
    --left;
    tile = next_tile;
    if (wraps && left > 0) {
      int seg = place[which].seg, chunk = place[which].chunk;
      next_chunk(seg, chunk);
      which ^= 1;
      set_place(which, seg, chunk);
      stale = true;
    }
  }

  if (ok && count > 0 && warp == turn) {
    ok = add_up();                                 // the last tile
    // ... and the last one that this CTA leads (the tile `leader` is at stands for the cluster's last)
    const int last_led = leader >= rank ? lap : lap - 1;
    if (ok && csize > 1 && last_led >= 0) ok = finish(last_led);
  }

  // ---- rows past the last expert's are zero ----
  if (grouped) {
    const int64_t used = static_cast<int64_t>(seg_row[p.segs]) * p.N, all = p.M * p.N;
    for (int64_t i = used + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < all; i += static_cast<int64_t>(gridDim.x) * blockDim.x)
      store_y(p.y, p.y_dtype, i, 0.0f);
  }
  if (!ok) {                                       // gave up: the boxes on the way land first
    cp_async_drain();
    if (lane == 0) {
      atomicCAS(p.status, 0, *abort_flag);
      for (uint32_t i = 0; i < static_cast<uint32_t>(p.ring); ++i) mbar_drain(my_full + i * 8, i < slot ? slot_phase ^ 1u : slot_phase);
    }
  }
  if (csize > 1) {                                 // nobody leaves while a peer may still write to its shared memory
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// ---- host side ---------------------------------------------------------------------------

struct RowsPlan {
  int blocks, cluster, warps, slices_per_cta, slices_per_warp, ring, red_bufs, grid;
  int64_t items;                 // (chunk, tile) items of a dense product
  size_t smem;
  double load;                   // what it is expected to take (see plan_rows)
};

struct RowsShape {
  int tokens, groups, tt, stage;         // rows of a chunk; groups per slice; bytes of codes of a 16-row block and slice
  bool exact;                            // 16-bit activations, results in plain float32 (tiles of kMaxBlocks only)
};

template <int QK, typename XT, int T, int SPG, int TT, int R, bool EXACT>
int launch_kernel_of(const CUtensorMap& wm, const CUtensorMap& wm2, RowsParams& rp, RowsPlan& pl, bool early, cudaStream_t stream) {
  auto kernel = qmm_rows_kernel<QK, XT, T, SPG, TT, R, EXACT>;
  static bool configured[kMaxDevices] = {};     // the attribute is per device
  const int dev = current_device();
  if (dev < 0) return QMM_ERR_DEVICE;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) return fail(QMM_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(pl.warps * 32);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  cfg.numAttrs = 0;
  if (pl.cluster > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = pl.cluster;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
    cfg.gridDim = dim3(pl.grid);
    // (a GPC's SMs do not always divide by the cluster size: more clusters than fit at once would be a second wave of persistent CTAs)
    const int most = max_active_clusters(reinterpret_cast<const void*>(kernel), cfg, pl.cluster);
    if (pl.grid > most * pl.cluster) pl.grid = most > 0 ? most * pl.cluster : pl.cluster;
  }
  cfg.gridDim = dim3(pl.grid);
  const unsigned clusters = static_cast<unsigned>(pl.grid / pl.cluster);
  rp.share = static_cast<unsigned>(pl.items / clusters);
  rp.share_more = static_cast<unsigned>(pl.items - static_cast<int64_t>(rp.share) * clusters);
  if (early) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, wm, wm2, rp);
  if (e != cudaSuccess) return fail(QMM_ERR_CUDA, "qmm_rows_kernel launch: %s", cudaGetErrorString(e));
  count_launch();
  return check_launch("qmm_rows_kernel");
}

template <int QK, typename XT, int T, int SPG, int TT>
int launch_kernel(const CUtensorMap& wm, const CUtensorMap& wm2, RowsParams& rp, RowsPlan& pl, const RowsShape& sh, bool early, cudaStream_t stream) {
  constexpr bool kFloat = std::is_same<XT, float>::value;
  if constexpr (QK != kMx4 && !kFloat)
    if (sh.exact) return launch_kernel_of<QK, XT, T, SPG, TT, kMaxBlocks, true>(wm, wm2, rp, pl, early, stream);
  if (pl.blocks == 1) return launch_kernel_of<QK, XT, T, SPG, TT, 1, kFloat>(wm, wm2, rp, pl, early, stream);
  return launch_kernel_of<QK, XT, T, SPG, TT, kMaxBlocks, kFloat>(wm, wm2, rp, pl, early, stream);
}

// (QK, XT) by T, group size and table type.
template <int QK, typename XT, int T, int SPG>
int launch_tt(const CUtensorMap& wm, const CUtensorMap& wm2, RowsParams& rp, RowsPlan& pl, const RowsShape& sh, bool early, cudaStream_t stream) {
  if constexpr (QK == kMx4) {
    return launch_kernel<QK, XT, T, SPG, kTabE8>(wm, wm2, rp, pl, sh, early, stream);
  } else {
    if (sh.tt == kTabBf16) return launch_kernel<QK, XT, T, SPG, kTabBf16>(wm, wm2, rp, pl, sh, early, stream);
    if (sh.tt == kTabF16) return launch_kernel<QK, XT, T, SPG, kTabF16>(wm, wm2, rp, pl, sh, early, stream);
    return launch_kernel<QK, XT, T, SPG, kTabF32>(wm, wm2, rp, pl, sh, early, stream);
  }
}

template <int QK, typename XT, int T>
int launch_spg(const CUtensorMap& wm, const CUtensorMap& wm2, RowsParams& rp, RowsPlan& pl, const RowsShape& sh, bool early, cudaStream_t stream) {
  if constexpr (QK == kMx4) {
    return launch_tt<QK, XT, T, 1>(wm, wm2, rp, pl, sh, early, stream);
  } else {
    if (sh.groups == kSliceK / 32) return launch_tt<QK, XT, T, 1>(wm, wm2, rp, pl, sh, early, stream);
    if (sh.groups == kSliceK / 64) return launch_tt<QK, XT, T, 2>(wm, wm2, rp, pl, sh, early, stream);
    return launch_tt<QK, XT, T, 4>(wm, wm2, rp, pl, sh, early, stream);
  }
}

template <int QK, typename XT>
int launch_rows_kernel(const CUtensorMap& wm, const CUtensorMap& wm2, RowsParams& rp, RowsPlan& pl, const RowsShape& sh, bool early, cudaStream_t stream) {
  if constexpr (sizeof(XT) == 4) {
    return launch_spg<QK, XT, 4>(wm, wm2, rp, pl, sh, early, stream);
  } else {
    return launch_spg<QK, XT, 8>(wm, wm2, rp, pl, sh, early, stream);
  }
}

}  // namespace rows
}  // namespace qmm
