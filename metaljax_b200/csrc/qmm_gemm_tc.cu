// Prefill kernel of the fused dequantize-and-matmul on the 5th-generation tensor cores.
//
//   y[t, f] = sum_k x[t, k] * deq(w)[f, k]          (transpose=True of the reference's call,
//                                                    src/metaljax/qmm.py:2491)
//
// The WEIGHT is the MMA's A operand and lives in tensor memory: a CTA's tile is 128 output
// features (= 128 TMEM lanes), so one dequantizing thread owns one weight row, reads its packed bytes of
// 64 K-elements from shared memory, applies its own per-group scale and bias in registers, and writes the
// bf16/f16 result straight to TMEM with tcgen05.st -- the dequantized weight never exists in shared or
// global memory. The ACTIVATIONS are the B operand: TMA brings [tokens x 64 K] tiles into shared memory in
// the 128-byte-swizzled K-major layout tcgen05.mma reads. The accumulator D[feature, token]
// (float32) sits in TMEM; the epilogue reads it back with tcgen05.ld, casts and stores y[token, feature].
//
// Wide token tiles (256) are worked on by PAIRS of CTAs (`cta_group::2`): 256 features x 256 tokens, each CTA
// dequantizes its own 128 features and holds half of the tokens' activations, so an SM reads 16 KB of activations per 64 K
// instead of 32: a lone CTA's 36 KB per 64 K were what L2 could not deliver (42 bytes a clock and SM at 974 TFLOP/s).
//
// Scales and biases travel with the boxes, 32 bytes of a table row at a time (cp.async by the weights' producer, two lanes to a row): read by the
// dequantizing threads from global memory they thrashed what is left of L1 next to 200 KB of shared memory, and their
// latency was the dequantization's. Packed weights come in boxes of 128 rows x 128 bytes (256 4-bit K-elements, 128 8-bit ones, 64 float ones) through a
// ring of their own: a box of 32 bytes a row for 64 4-bit elements costs the TMA unit and L2 a request per 32 bytes.
//
// Warp roles (19 warps): 0 = activations' producer, 1 = MMA issuer (+ TMEM allocation), 2..17 = sixteen
// dequant/epilogue warps in four teams of four (one warp per TMEM lane quarter) that take K blocks round-robin,
// 18 = weights' producer.
//
// Persistent workers (a CTA or a pair) walk a list of tiles (segment, token tile, feature tile).
// A segment is a run of x rows that meets one weight matrix: the whole of x for the plain
// op, one batch of a batched weight, or one expert's rows of a ragged (grouped) product,
// in which case the per-expert row offsets are prefix sums of `group_sizes` computed here.
// Tiles that do not fill the workers evenly are shared out by weight boxes (every worker an equal, contiguous stretch of K over
// consecutive tiles): a tile's pieces meet through float32 partial tiles in scratch, which the worker that holds the
// tile's last piece adds up in K order. A worker walks its stretch from the end, so the piece another worker waits for is
// the first that it makes, and waits only on lower-numbered workers, which were scheduled before it.
//
// Measured (device time, before: one CTA per tile at every width, 32-byte boxes, tables from global memory, an issuer behind a branch, split
// products added up by a second kernel), int4 group 64: 2048 rows 14336 x 4096 248 -> 181..189 us (the clock under load decides), 4096 x 14336
// 219 -> 167..174; 512 rows 28672 x 4096 130 -> 97; 64 rows 28672 x 4096 59.7 -> 33.1, 4096 x 4096 16.4 -> 10.5, 4096 x 14336 31.2 -> 19.4; 128 rows
// 4096 x 14336 47 -> 21; 8-bit group 128, 45 rows 14336 x 4096 33 -> 20.6. Table entries a sector of a row at a time instead of the 8 bytes of
// every box (a row a lane: 32 lines an instruction; without the dequantization 64 rows then took 345 clocks a K block and SM, 204 without those copies):
// 64 rows 28672 x 4096 33.3 -> 30.6, 65760 x 2880 (rows of 90 table bytes) 79.3 -> 48.7, float32 tables in groups of 32 14336 x 4096 42 -> 33. What an epilogue
// costs: 4.6 us a tile of 256 x 256 with 2-byte stores behind a check each (2.1 at 64 tokens); drained into registers and rounded first, stored in pairs of features: 64 rows 28672 x
// 4096 30.6 -> 27.0, 512 rows mxfp4 5760 x 2880 22.8 -> 20.6, 2048 rows 14336 x 4096 183 -> 172. The weights' producer on its way before the rest is set up: 64 rows 28672 x 4096 27.0 ->
// 26.3, 4096 x 14336 17.6 -> 17.2. MXFP4 codes looked up: 64 rows 65760 x 2880 48.1 -> 43.0; and shorter tiles where there are few: 512 rows 5760 x 2880 20.5 -> 18.8.
// What bounds it: at 64 rows memory and the dequantizing warps together (335 clocks a K block and SM; 260 without the dequantization, 210 of them the weights' bytes) and some
// 6 us of a launch's ends, at 256 the tensor cores (500 clocks a block between a tile's ends, under the power cap) and the ends,
// where the accumulator is drained by the warps that would dequantize for the next tile. (Draining it after the first steps of the next
// tile was built: the state that lives across the epilogue then spills, and every size lost.)
//
// Every wait is bounded: when a barrier does not flip within ~2 s of SM clock the kernel
// records the place in a status word, stops issuing work and drains.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>
#include <type_traits>

#include "qmm_internal.h"
#include "qmm_ptx.cuh"
#include "qmm_tcgen05.cuh"

namespace qmm {
namespace {

using namespace ptx;
using namespace tc;

constexpr int kBF = 128;        // features of a CTA's tile (TMEM lanes)
constexpr int kBK = 64;         // K elements of a K block
constexpr int kTeams = 4;       // dequant / epilogue teams of four warps (one per TMEM lane quarter)
constexpr int kDequantWarps = 4 * kTeams;
constexpr int kWarps = 3 + kDequantWarps;
constexpr int kThreads = kWarps * 32;
constexpr int kMaxSegments = 256;
constexpr int kBoxBytes = 128;  // bytes of a weight row in a box
constexpr int kChunkBytes = 32; // bytes of a table row in a chunk: a sector of memory ...
constexpr int kTablePitch = 48; // ... and in shared memory, where they keep their distance from a 16-byte boundary

enum { kAff4 = 0, kAff8 = 1, kMx4 = 2, kFloat = 3 };    // kFloat: the weight holds values of the activation type (nothing to dequantize)

struct TcParams {
  const void* scales;
  const void* biases;
  void* y;
  const int32_t* group_sizes;  // ragged: [segments]; else NULL
  int* status;                 // device status word (0 = ok)
  int64_t M;                   // rows of x per segment (dense) or total rows (ragged)
  int64_t N;
  int64_t w_seg_rows;          // rows of the packed weight between segments (N, or 0 = shared)
  int K, segments, group_shift, table_dtype, y_dtype;
  int w_stages, t_stages;      // places of the weight ring, and of the ring of table chunks
  unsigned w_inverse, t_inverse;              // 2^32 / w_stages and t_stages, rounded up: counts are divided by a multiplication
  int table_entry, skewed;     // bytes of a table entry; whether some chunk's entries start off a 16-byte boundary
  int chunk_shift;             // weight boxes per table chunk (log2)
  int64_t table_bytes;         // of a whole table
  int tile_rows;               // token rows of a tile: the template's, or fewer where that fills the machine in one round
  int split;                   // > 1: `split` consecutive workers share the K of each tile (and the walk is one tile long): a cluster that
  int cluster_adds;            // adds up over distributed shared memory, or partial tiles for the kernel that follows
  int shared_tiles;            // the first tiles of the walk are shared out by weight boxes ...
  unsigned share, share_more;  // ... `share` to every worker, one more to the first `share_more`
  float* partial;              // [CTA][tokens of a tile][128]: a CTA's partial tile
  unsigned long long* ready;   // [CTA][dequant warps]: == epoch when that warp's part of the partial tile is there
  unsigned long long epoch;    // a value that no earlier launch used
};

// ---- dequantization of one weight row's K block into 32 packed 16-bit pairs ---------------

// (a & mask) | bits in one LOP3: with both constants known the compiler makes two of it, an immediate each.
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t bits) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(mask), "r"(bits));
  return d;
}
__device__ __forceinline__ uint32_t in_register(uint32_t v) {
  asm volatile("" : "+r"(v));
  return v;
}

// 4-bit affine, NW packed words -> NW*4 pairs; s2, b2 are scale and bias as pairs of the type.
//
// bf16: the even and the odd nibbles of a word under a byte mask each; PRMT takes byte i of either into bytes 0 and 2 of a
// pair and zeros (the sign of the even one's byte) into 1 and 3. A code in bits 0 to 3 is the subnormal q 2^-133, one in bits 4 to 7 q 2^-129 (bit 7 is the first
// exponent's, where numbers go on as the subnormals do): a product with 2^127 or 2^123 makes it the
// exact q / 64, and one FMA with (64 s, 64 s), (b, b) rounds once. (Scales below 2^121.) 14 instructions a word, 6 of them on the
// half-rate logic pipe; with the odd nibbles shifted down 15 and 7, with a magic exponent per pair 17 and 9.
//
// f16 has no factor for that: there PRMT takes a byte from the word (even element in its low nibble) into byte 0 and from
// the word shifted right by four into byte 2, one LOP3 keeps the two nibbles under the magic exponent (1024 + q, exact),
// an exact subtraction removes the magic, and the FMA rounds once.
template <typename XT, int NW>
__device__ __forceinline__ void dequant_aff4(const uint32_t (&w)[NW], uint32_t s2, uint32_t b2, uint32_t mask, uint32_t magic, uint32_t* out) {
  using H = Half2Ops<XT>;
  if constexpr (std::is_same<XT, __nv_bfloat16>::value) {
    const uint32_t s64 = H::mul(s2, 0x42804280u);
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      const uint32_t even = w[j] & 0x0F0F0F0Fu, odd = w[j] & 0xF0F0F0F0u;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t q = permute(even, odd, i | ((8 + i) << 4) | ((4 + i) << 8) | ((8 + i) << 12));
        out[j * 4 + i] = H::fma(H::mul(q, 0x7D007F00u), s64, b2);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      const uint32_t hi = w[j] >> 4;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t t = __byte_perm(w[j], hi, i | ((4 + i) << 8));
        const uint32_t v = and_or(t, mask, magic);
        out[j * 4 + i] = H::fma(H::sub(v, magic), s2, b2);
      }
    }
  }
}

// The same for float32 tables (what the packer emits when a bias is not exactly
// representable in the narrow type): the magic pair is widened to float32, one float32 FMA
// per element with (s, b - C s), one rounding to the pair type.
template <typename XT, int NW>
__device__ __forceinline__ void dequant_aff4_wide(const uint32_t (&w)[NW], float s, float b, uint32_t* out) {
  using H = Half2Ops<XT>;
  const float c = std::is_same<XT, __nv_bfloat16>::value ? 128.0f : 1024.0f;
  const float bc = fmaf(-c, s, b);
#pragma unroll
  for (int j = 0; j < NW; ++j) {
    const uint32_t hi = w[j] >> 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t t = __byte_perm(w[j], hi, i | ((4 + i) << 8));
      const uint32_t v = (t & 0x000F000Fu) | H::kMagic;
      float lo, up;
      if constexpr (std::is_same<XT, __nv_bfloat16>::value) {
        lo = __uint_as_float(v << 16);
        up = __uint_as_float(v & 0xffff0000u);
      } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
        lo = f.x; up = f.y;
      }
      out[j * 4 + i] = H::pack(fmaf(s, lo, bc), fmaf(s, up, bc));
    }
  }
}

// x0, x1 = s * (x0 - 2^23) + b, the same for x1: two elements per instruction.
__device__ __forceinline__ void take_magic_and_scale(float& x0, float& x1, float s, float b) {
  asm("{ .reg .b64 x, m, s, b; mov.b64 x, {%0, %1}; mov.b64 m, {%2, %2}; mov.b64 s, {%3, %3}; mov.b64 b, {%4, %4};"
      "  add.rn.f32x2 x, x, m; fma.rn.f32x2 x, x, s, b; mov.b64 {%0, %1}, x; }"
      : "+f"(x0), "+f"(x1) : "f"(-8388608.0f), "f"(s), "f"(b));
}

// 8-bit affine, NW packed words -> NW*2 pairs, f16; s2, b2 are scale and bias as pairs. Two bytes of the word under a magic exponent are the f16 1024 + q; an exact subtraction and one
// FMA, which rounds once. Six instructions a word; in float32 (below) ten, four of them byte permutes at half rate, and two roundings: 45 rows of 4096 x 14336 20.6 -> 19.2 us, 2048 rows of
// 14336 x 4096 192.8 -> 186.2. bf16 has no such exponent: its bytes are q 2^-133 as they stand, which takes 64 times the scale, and a way of its own for scales from 2^121 on: with
// both in a kernel 2048 rows took 181.8 instead of 185.0 us, but 24 rows of 4096 x 4096 12.6 instead of 11.4, and it stays in float32.
template <int NW>
__device__ __forceinline__ void dequant_aff8_f16(const uint32_t (&w)[NW], uint32_t s2, uint32_t b2, uint32_t* out) {
  using H = Half2Ops<__half>;
#pragma unroll
  for (int j = 0; j < NW; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) out[j * 2 + h] = H::fma(H::sub(__byte_perm(w[j], 0x64646464u, h ? 0x4342 : 0x4140), H::kMagic), s2, b2);
}

// The same in float32, for bf16 and for other tables: an FMA per element, rounded to the 16-bit type in pairs.
template <typename XT, int NW>
__device__ __forceinline__ void dequant_aff8(const uint32_t (&w)[NW], float s, float b, uint32_t* out) {
  using H = Half2Ops<XT>;
#pragma unroll
  for (int j = 0; j < NW; ++j) {
    float q[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) q[e] = __uint_as_float(__byte_perm(w[j], 0x4B000000u, 0x7540u + e));
    take_magic_and_scale(q[0], q[1], s, b);
    take_magic_and_scale(q[2], q[3], s, b);
    out[j * 2] = H::pack(q[0], q[1]);
    out[j * 2 + 1] = H::pack(q[2], q[3]);
  }
}

// MXFP4, NW packed words of one 32-element group -> NW*4 pairs. The group's eight magnitudes, each times the group's E8M0 scale (a product of exact values, rounded
// once where the type cannot hold it), are made once and split into their low and their high bytes: a byte permute then looks four codes up at a time,
// and their signs go in on top. 15 instructions a word and 8 a group; with the bits of each pair moved to the exponent's place and multiplied twice they were 29 a word.
template <typename XT, int NW>
__device__ __forceinline__ void dequant_mx4(const uint32_t (&w)[NW], uint32_t e8, uint32_t* out) {
  using H = Half2Ops<XT>;
  constexpr bool kBf = std::is_same<XT, __nv_bfloat16>::value;
  // 0, 1/2 | 1, 3/2 | 2, 3 | 4, 6
  constexpr uint32_t kMagnitudes[4] = {kBf ? 0x3F000000u : 0x38000000u, kBf ? 0x3FC03F80u : 0x3E003C00u, kBf ? 0x40404000u : 0x42004000u, kBf ? 0x40C04080u : 0x46004400u};
  const float sc = __uint_as_float(e8 ? (e8 << 23) : 0x00400000u);
  const uint32_t s2 = H::pack(sc, sc);
  uint32_t m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = H::mul(kMagnitudes[i], s2);
  const uint32_t low[2] = {permute(m[0], m[1], 0x6420), permute(m[2], m[3], 0x6420)}, high[2] = {permute(m[0], m[1], 0x7531), permute(m[2], m[3], 0x7531)};
#pragma unroll
  for (int j = 0; j < NW; ++j) {
    const uint32_t codes = w[j] & 0x77777777u, even = w[j] << 4;       // (a byte of `even` has the sign of its even code on top, one of the word that of its odd one)
#pragma unroll
    for (int h = 0; h < 2; ++h) {                  // four codes
      const uint32_t at = h ? codes >> 16 : codes;
      const uint32_t lo = permute(low[0], low[1], at), hi = and_or(permute(even, w[j], h ? 0x7362 : 0x5140), 0x80808080u, permute(high[0], high[1], at));
      out[j * 4 + 2 * h] = permute(lo, hi, 0x5140);
      out[j * 4 + 2 * h + 1] = permute(lo, hi, 0x7362);
    }
  }
}

// ---- shared-memory plan -----------------------------------------------------------------

// Rings of activation tiles (each with a 32-column slot of dequantized weights in tensor memory per K block) and of
// weight boxes. A step is what a team dequantizes and the issuer waits for and commits at once: two K blocks, since the waits,
// fences and arrivals around a step cost a team about as much as one block's arithmetic.
template <int QK, int BT>
struct Plan {
  static constexpr bool kPair = BT == 256;
  static constexpr int kCtas = kPair ? 2 : 1;
  static constexpr int kBits = (QK == kFloat) ? 16 : ((QK == kAff8) ? 8 : 4);
  static constexpr int kRowBytes = kBK * kBits / 8;           // of a weight row in a K block: 32, 64 or (float weights) 128
  static constexpr int kPer = kBoxBytes / kRowBytes;          // K blocks of a box
  static constexpr int kStep = QK == kFloat && BT > 64 ? 1 : 2;      // (float weights' boxes leave no room for four of two)
  static constexpr int kStepsPerBox = kPer >= kStep ? kPer / kStep : 1;
  static constexpr int kXBlock = (BT / kCtas) * kBK * 2;      // a K block of this CTA's activations
  static constexpr int kXBytes = kStep * kXBlock;
  static constexpr int kWBytes = kBF * kBoxBytes;
  static constexpr int kACol0 = BT;                           // the A ring starts behind D's columns [0, BT)
  static constexpr int kTeamCols = BT / kTeams;               // columns of D that a team drains ...
  // ... so many at a time. At 128 tokens 32 spill some 200 bytes and are the faster for 4-bit codes all the same (us, 32 / 16: 96 rows 28672 x 4096 31.8 / 33.8, mxfp4 35.3 /
  // 37.7, 4096 x 14336 19.5 / 20.6), but not for 8-bit ones (44.2 / 42.8, 128 rows 4096 x 4096 13.7 / 13.5) and float weights (8 x 100 rows 2880 x 2880 45.5 / 43.5).
  static constexpr int kCols = BT == 128 && kBits == 4 ? 32 : 16;
  // A tile goes into registers rounded, whole, before it is stored. (Not float weights' 256 tokens: they spilled 156 bytes; 8 x 2048 rows 4096 x 4096 409 us, 388 so.)
  static constexpr bool kHeld = !(QK == kFloat && BT == 256);
  static constexpr int kStages = kStep == 1 || (BT <= 64 && QK != kFloat) ? 6 : 4;
  static constexpr int kBarBytes = 1024;
  static constexpr int kBudget = 227 * 1024 - 4608;           // dynamic shared memory (the tile tables are static)
  static constexpr int kFixed = kStages * kXBytes + kBarBytes + 1024 /* alignment slack */;
  static constexpr int kMostBoxes = 10;
  static constexpr bool kMaySplit = kStages * kXBytes >= BT * kBF * 4;      // a cluster's partial tile goes where the activations were
  // A team need not touch every box, and a parity wait cannot tell a box from the one two rounds before it: the team's wait for
  // its A slot, which comes first, has to imply that the box before in the same place has been used up.
  static constexpr int kLeastPlaces = (kStages * kStep + (kPer > kStep ? kPer - kStep : 0) + kPer - 1) / kPer;
  // ... and a team that waits for its next A slot must not be able to lag that slot's barrier by two phases.
  static_assert(kStages >= kTeams, "");
  static_assert(kACol0 + kStages * kStep * 32 <= 512, "the A ring fits tensor memory");
  static_assert(kFixed + kLeastPlaces * kWBytes <= kBudget, "");
  // (the next launch may start before this one's tensor memory is allocated: none of its CTAs may get onto the SM with some of it)
  static_assert(kFixed + kLeastPlaces * kWBytes > 128 * 1024, "one CTA an SM, and none of qmm_f32_tc.cu's (100 KB and more) beside it");
  static_assert(kTeams * kStep % kPer == 0, "a team's next step lies whole boxes ahead");
  static_assert((2 * kMostBoxes + 3 * kStages + 2) * 8 + 16 <= kBarBytes, "");
};

// A piece of work: K blocks [kb_lo, kb_hi) of a tile.
struct Piece {
  int kb_lo, kb_hi, tile;
  bool begins, ends;           // it holds the tile's first / last K block
  int seg, rows;               // rows: token rows of the tile that exist
  int64_t row0, f0;            // first x / y row, first feature (of the whole tile)
};

// The walk of worker `w` of `workers`: its stretch of the shared tiles from the end, then every workers-th tile.
template <int BT, int kPer>
struct Walk {
  int lo, hi, next, w, workers, boxes, num_kb, tiles, tile_rows;
  __device__ __forceinline__ Walk(const TcParams& p, int w_, int workers_, int num_kb_, int tiles_) : w(w_), workers(workers_), num_kb(num_kb_), tiles(tiles_) {
    boxes = (num_kb + kPer - 1) / kPer;
    tile_rows = p.tile_rows;
    lo = hi = 0;
    if (p.split > 1) {                             // one piece, its stretch of K of the cluster's tile
      const int tile = w / p.split, part = w - tile * p.split;
      lo = tile * boxes + boxes * part / p.split;
      hi = tile * boxes + boxes * (part + 1) / p.split;
      next = 0x7fffffff;
      return;
    }
    if (p.shared_tiles) {
      lo = first_box(p, w);
      hi = lo + static_cast<int>(p.share) + (static_cast<unsigned>(w) < p.share_more ? 1 : 0);
    }
    next = p.shared_tiles + w;
  }
  static __device__ __forceinline__ int first_box(const TcParams& p, int w) {
    return static_cast<int>(static_cast<unsigned>(w) * p.share + min(static_cast<unsigned>(w), p.share_more));
  }
  __device__ __forceinline__ bool take(Piece* out, const int* seg_tile0, const int64_t* seg_row0, int nseg, int ftiles, int features) {
    int t, b0, b1;
    if (hi > lo) {
      t = static_cast<int>(static_cast<unsigned>(hi - 1) / static_cast<unsigned>(boxes));
      const int base = t * boxes;
      b0 = (lo > base ? lo : base) - base;
      b1 = hi - base;
      hi = base + b0;
    } else {
      t = next;
      next = static_cast<int>(static_cast<unsigned>(next) + static_cast<unsigned>(workers));
      if (static_cast<unsigned>(t) >= static_cast<unsigned>(tiles)) return false;
      b0 = 0;
      b1 = boxes;
    }
    out->tile = t;
    out->begins = b0 == 0;
    out->ends = b1 == boxes;
    out->kb_lo = b0 * kPer;
    out->kb_hi = b1 * kPer < num_kb ? b1 * kPer : num_kb;
    int s = 0;
    while (t >= seg_tile0[s + 1]) ++s;
    const unsigned local = static_cast<unsigned>(t - seg_tile0[s]);
    // feature tiles vary fastest inside a token tile, so that concurrently running workers share the activation
    // tile and stream disjoint weight rows
    const unsigned tt = local / static_cast<unsigned>(ftiles), ft = local - tt * static_cast<unsigned>(ftiles);
    out->seg = s;
    out->row0 = seg_row0[s] + static_cast<int64_t>(tt) * static_cast<unsigned>(tile_rows);
    const int64_t left = seg_row0[s + 1] - out->row0;
    out->rows = static_cast<int>(left < tile_rows ? left : tile_rows);
    out->f0 = static_cast<int64_t>(ft) * features;
    return true;
  }
};

// SAME: the tables are of the activation type (the pairs for the arithmetic are the entries themselves).
template <int QK, typename XT, int BT, bool SAME>
__global__ void __launch_bounds__(kThreads, 1)
qmm_gemm_tc_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const TcParams p) {
  using P = Plan<QK, BT>;
  constexpr bool kPair = P::kPair;
  constexpr int kCtas = P::kCtas, kPer = P::kPer, kStep = P::kStep, kStages = P::kStages, kMostBoxes = P::kMostBoxes;
  constexpr int kTables = QK == kMx4 ? 1 : 2;
  extern __shared__ uint8_t smem_raw[];
  __shared__ int seg_tile0[kMaxSegments + 1];
  __shared__ int64_t seg_row0[kMaxSegments + 1];

  const uint32_t smem = (smem_u32(smem_raw) + 1023) & ~1023u;
  const uint32_t x_at = smem, bars = smem + kStages * P::kXBytes, w_at = bars + P::kBarBytes, t_at = w_at + p.w_stages * P::kWBytes;
  const uint32_t wfull = bars, wempty = wfull + 8 * kMostBoxes;         // a weight box and its table entries have landed / have been read
  const uint32_t xfull = wempty + 8 * kMostBoxes;                         // a step's activations have landed
  const uint32_t empty = xfull + 8 * kStages;                           // a step's MMAs are done: its activations and its A slot are free
  const uint32_t a_full = empty + 8 * kStages;                          // (a pair's leader) a step's dequantized weights are in TMEM
  const uint32_t d_full = a_full + 8 * kStages, d_empty = d_full + 8;   // accumulator complete / (leader) drained
  const uint32_t tmem_slot = d_empty + 8, abort_at = tmem_slot + 4;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int in_cluster = kPair || p.cluster_adds ? static_cast<int>(cluster_rank()) : 0;
  const int rank = kPair ? in_cluster & 1 : 0, leader = in_cluster - rank;            // within the pair
  [[maybe_unused]] const uint16_t pair_mask = static_cast<uint16_t>(3 << leader);
  const int worker = static_cast<int>(blockIdx.x) / kCtas, workers = static_cast<int>(gridDim.x) / kCtas;
  const int nseg = p.segments;
  const int ftiles = static_cast<int>((p.N + kBF * kCtas - 1) / (kBF * kCtas));
  const int num_kb = (p.K + kBK - 1) / kBK;

  // Programmatic dependent launch: the grid that follows may be scheduled as soon as every CTA
  // of this one has got here (it touches memory only after its own griddepcontrol.wait). This
  // grid sets itself up, and requests its first weight boxes, while the grid it depends on is
  // still running; what that grid produces -- the activations, the group sizes of a ragged
  // product -- is read only after a griddepcontrol.wait, and everything this grid writes is
  // downstream of those reads.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  auto init = [](uint32_t bar, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n)); };
  uint32_t tmem_base = 0;
  if (warp == kWarps - 1) {
    // The weights' producer lays out the walk and its own barriers and does not wait for the rest: its first boxes are on their way (a trip to
    // memory, 2 us when every CTA asks at once) while the others set up tensor memory and their barriers (0.7 us).
    if (p.group_sizes) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      for (int s = lane; s < nseg; s += 32) seg_row0[s + 1] = p.group_sizes[s] > 0 ? p.group_sizes[s] : 0;
      __syncwarp();
    }
    if (lane == 0) {
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(abort_at), "r"(0) : "memory");
      int64_t rows = 0;
      int tiles = 0;
      seg_row0[0] = 0;
      seg_tile0[0] = 0;
      for (int s = 0; s < nseg; ++s) {
        int64_t r = p.group_sizes ? seg_row0[s + 1] : p.M;
        if (p.group_sizes && rows + r > p.M) r = p.M - rows;
        rows += r;
        tiles += static_cast<int>((r + p.tile_rows - 1) / p.tile_rows) * ftiles;
        seg_tile0[s + 1] = tiles;
        seg_row0[s + 1] = rows;
      }
      for (int i = 0; i < p.w_stages; ++i) {
        init(wfull + 8 * i, QK == kFloat ? 1 : 1 + 32);
        init(wempty + 8 * i, 4 * P::kStepsPerBox);
      }
      mbar_init_fence();
    }
    __syncwarp();
    asm volatile("bar.arrive 1, %0;" ::"n"(kThreads) : "memory");
    if constexpr (kPair) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  } else {
    if (threadIdx.x == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&x_map)) : "memory");
      for (int i = 0; i < kStages; ++i) {
        init(xfull + 8 * i, 1);
        init(empty + 8 * i, 1);
        init(a_full + 8 * i, 4 * kCtas);
      }
      init(d_full, 1);
      init(d_empty, kDequantWarps * kCtas);
      mbar_init_fence();
    }
    if (warp == 1) {
      if constexpr (kPair) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
      } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
      }
    }
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
    if constexpr (kPair) cluster_barrier();        // the partner's barriers and tensor memory are there
    tc_fence_after();
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot) : "memory");
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);
  }
  const int tiles = seg_tile0[nseg];
  Walk<BT, kPer> walk(p, worker, workers, num_kb, tiles);
  Piece pc = {};
  auto wait = [&](uint32_t bar, uint32_t parity, int where) -> bool { return wait_phase(bar, parity, abort_at, where); };
  // Columns of the MMA: the token rows that exist, in the widths the instruction takes (a pair's CTAs hold half each).
  auto columns = [&]() -> int { return kPair ? (pc.rows + 31) & ~31 : (pc.rows + 15) & ~15; };

  if (warp == 0) {
    // ---------------- activations ----------------
    if (lane == 0) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      uint32_t s = 0, ph = 0;
      bool ok = true;
      while (ok && walk.take(&pc, seg_tile0, seg_row0, nseg, ftiles, kBF * kCtas)) {
        const int row = static_cast<int>(pc.row0) + (kPair ? rank * (columns() / 2) : 0);
        for (int kb = pc.kb_lo; kb < pc.kb_hi; kb += kStep) {
          if (!(ok = wait(empty + 8 * s, ph ^ 1u, 1))) break;
          const uint32_t bar = xfull + 8 * s;
          const int blocks = kStep == 1 || kb + 1 < pc.kb_hi ? kStep : 1;
          mbar_expect_tx(bar, blocks * P::kXBlock);
          for (int i = 0; i < blocks; ++i) tma_load_2d(&x_map, x_at + s * P::kXBytes + i * P::kXBlock, bar, (kb + i) * kBK, row);
          if (++s == static_cast<uint32_t>(kStages)) { s = 0; ph ^= 1u; }
        }
      }
      if (!ok)                                     // gave up: what is on the way lands first (of each place, its last load)
        for (uint32_t i = 0; i < static_cast<uint32_t>(kStages); ++i) mbar_drain(xfull + 8 * i, i < s ? ph : ph ^ 1u);
    }
  } else if (warp == kWarps - 1) {
    // ---------------- weights and tables (nothing the grid before writes: they need not wait for it) ----------------
    const int groups = QK == kFloat ? 1 : p.K >> p.group_shift;
    int s = 0;
    [[maybe_unused]] int ts = -1;                  // place of the chunk that is being read
    [[maybe_unused]] uint32_t issued = 0, chunks = 0, last_box = 0;    // boxes and chunks so far; (lane i) the last box of the chunk in place i
    uint32_t ph = 0;
    bool ok = true;
    while (ok && walk.take(&pc, seg_tile0, seg_row0, nseg, ftiles, kBF * kCtas)) {
      const int row = static_cast<int>(pc.seg * p.w_seg_rows + pc.f0) + rank * kBF;
      const int last = static_cast<int>(p.N - pc.f0) - rank * kBF - 1;                  // the tile's last row of this weight (or before its first)
      for (int kb = pc.kb_lo; kb < pc.kb_hi; kb += kPer) {
        if (!(ok = wait(wempty + 8 * s, ph ^ 1u, 3))) break;
        const uint32_t bar = wfull + 8 * s;
        if (lane == 0) {
          mbar_expect_tx(bar, P::kWBytes);
          tma_load_2d(&w_map, w_at + s * P::kWBytes, bar, QK == kFloat ? kb * kBK : kb * P::kRowBytes, row);
        }
        if constexpr (QK != kFloat) {
          // A chunk of table entries with its first box (or the piece's). Every box's barrier gets the lanes' arrivals: they come
          // when all of a lane's earlier copies have landed, so any box of a chunk answers for its entries.
          const int box = kb / kPer, chunk = box >> p.chunk_shift;
          if (kb == pc.kb_lo || (box & ((1 << p.chunk_shift) - 1)) == 0) {
            if (++ts == p.t_stages) ts = 0;
            if (chunks >= static_cast<uint32_t>(p.t_stages)) {        // the last box of the chunk that was here has been read
              const uint32_t was = __shfl_sync(0xffffffffu, last_box, ts), lap = __umulhi(was, p.w_inverse);
              if (issued - was < static_cast<uint32_t>(p.w_stages) && !(ok = wait(wempty + 8 * (was - lap * p.w_stages), lap & 1u, 3))) {
                ++s;                               // (its codes are on the way: see below)
                break;
              }
            }
            ++chunks;
            const int g0 = ((chunk << p.chunk_shift) * (kPer * kBK)) >> p.group_shift, most = (kPer * kBK << p.chunk_shift) >> p.group_shift;
            const int bytes = (groups - g0 < most ? groups - g0 : most) * p.table_entry;
            const uint32_t slot = t_at + ts * (kTables * kBF * kTablePitch);
            const int64_t row_bytes = static_cast<int64_t>(groups) * p.table_entry, at0 = row * row_bytes + g0 * p.table_entry;
            // 16 bytes a lane, neighbouring lanes to a row: an instruction meets as few lines of memory as it can. Entries that start off a
            // 16-byte boundary come with what lies before them; nothing past the table's end is read.
            auto copy = [&](const void* table, uint32_t to) {
              const uint8_t* src = static_cast<const uint8_t*>(table) + at0;
              if (!p.skewed) {
                const int o = (lane & 1) * 16;
                if (o < bytes)
#pragma unroll
                  for (int i = lane >> 1; i < kBF; i += 16) cp_async16(to + i * kTablePitch + o, src + min(i, last) * row_bytes + o, 16);
              } else {
                const int o = (lane & 3) * 16;
                const uint64_t end = reinterpret_cast<uint64_t>(table) + p.table_bytes;
#pragma unroll 4
                for (int i = lane >> 2; i < kBF; i += 8) {
                  const uint64_t at = reinterpret_cast<uint64_t>(src) + min(i, last) * row_bytes, from = (at & ~15ull) + o;
                  if (from < at + bytes) cp_async16(to + i * kTablePitch + o, reinterpret_cast<const void*>(from), end - from < 16 ? static_cast<int>(end - from) : 16);
                }
              }
            };
            copy(p.scales, slot);
            if constexpr (QK != kMx4) copy(p.biases, slot + kBF * kTablePitch);
          }
          if (lane == ts) last_box = issued;
          ++issued;
          cp_async_arrive(bar);
        }
        if (++s == p.w_stages) { s = 0; ph ^= 1u; }
      }
    }
    if (!ok) {
      cp_async_drain();
      for (int i = 0; i < p.w_stages; ++i) mbar_drain(wfull + 8 * i, i < s ? ph : ph ^ 1u);
    }
    if constexpr (kPair) {
      __syncwarp();
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // (of the arrival above)
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (of a pair: the leader's) ----------------
    if (!kPair || rank == 0) {
      constexpr uint32_t idesc0 = instr_desc(std::is_same<XT, __nv_bfloat16>::value ? 1 : 0, kBF * kCtas);
      uint32_t s = 0, ph = 0, piece = 0;
      bool issued = false;
      for (; walk.take(&pc, seg_tile0, seg_row0, nseg, ftiles, kBF * kCtas); ++piece) {
        const uint32_t idesc = __shfl_sync(0xffffffffu, idesc0 | (static_cast<uint32_t>(columns() >> 3) << 17), 0);
        const int nkb = __shfl_sync(0xffffffffu, pc.kb_hi - pc.kb_lo, 0);
        bool ok = kPair ? wait_phase<true>(d_empty, (piece & 1) ^ 1, abort_at, 2) : wait(d_empty, (piece & 1) ^ 1, 2);
        if (!__all_sync(0xffffffffu, ok)) break;
        for (int j = 0; j < nkb; j += kStep) {
          // (a pair's dequantizing warps answer for their own CTA's activations: see there)
          if constexpr (kPair) ok = wait_phase<true>(a_full + 8 * s, ph, abort_at, 4);
          else ok = wait(xfull + 8 * s, ph, 5) && wait(a_full + 8 * s, ph, 4);
          if (!__all_sync(0xffffffffu, ok)) break;
          tc_fence_after();
          const uint32_t blo = desc_low(x_at + s * P::kXBytes), acol = tmem_base + P::kACol0 + s * (32 * kStep);
          tc_mma_block<kPair>(tmem_base, acol, blo, kDescHigh, idesc, j ? 1u : 0u);
          if (kStep == 2 && j + 1 < nkb) tc_mma_block<kPair>(tmem_base, acol + 32, blo + P::kXBlock / 16, kDescHigh, idesc, 1u);
          tc_commit<kPair>(empty + 8 * s, pair_mask);
          issued = true;
          if (++s == static_cast<uint32_t>(kStages)) { s = 0; ph ^= 1u; }
        }
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_commit<kPair>(d_full, pair_mask);
      }
      // gave up, or done: the MMAs issued last complete before tensor memory is given back (they complete in order)
      if (issued) mbar_drain(empty + 8 * (s ? s - 1 : kStages - 1), s ? ph : ph ^ 1u);
    }
  } else {
    // ---------------- dequant + epilogue warps ----------------
    const int team = (warp - 2) >> 2;            // takes steps i of a piece with i % kTeams == team
    const int quarter = warp & 3;                // TMEM lane quarter this warp may touch
    const int frow = quarter * 32 + lane;        // feature row within the CTA's tile
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const int groups = QK == kFloat ? 1 : p.K >> p.group_shift;
    const bool twide = !SAME && p.table_dtype == QMM_F32;
    const int entry = QK == kMx4 ? 1 : SAME ? 2 : p.table_entry;
    [[maybe_unused]] const uint32_t mask = in_register(0x000F000Fu), magic = in_register(Half2Ops<XT>::kMagic);
    const uint32_t swizzle = (frow & 7) << 4;
    const uint32_t a_bar = kPair ? in_cta(a_full, leader) : a_full, d_bar = kPair ? in_cta(d_empty, leader) : d_empty;
    const uint32_t wthread = w_at + frow * kBoxBytes;
    uint32_t wbase = 0, sbase = 0, cbase = 0, piece = 0;    // boxes, steps and table chunks before this piece
    bool ok = true;
    for (; ok && walk.take(&pc, seg_tile0, seg_row0, nseg, ftiles, kBF * kCtas); ++piece) {
      int64_t feat = pc.f0 + rank * kBF + frow;
      const bool feat_ok = feat < p.N;
      if (!feat_ok) feat = p.N - 1;
      const uint32_t trow = static_cast<uint32_t>(pc.seg * p.w_seg_rows + feat) * static_cast<uint32_t>(groups);   // row of the tables (its low bits count)
      const int nkb = pc.kb_hi - pc.kb_lo, steps = (nkb + kStep - 1) / kStep;
      constexpr int kHalfBytes = P::kRowBytes / 2;                 // packed bytes of a half block
      // where the team's next step is in the rings: slot, box (and how often round)
      uint32_t s = (sbase + team) % kStages, ph = (sbase + team) / kStages & 1u;
      uint32_t wi = wbase + team * kStep / kPer, wph = __umulhi(wi, p.w_inverse), ws = wi - wph * p.w_stages;
      for (int i = team; i < steps; i += kTeams) {
        const int j = i * kStep;                   // first K block of the step
        if (!(ok = wait(empty + 8 * s, ph ^ 1u, 7))) break;
        if (!(ok = wait(wfull + 8 * ws, wph & 1u, 6))) break;
        __syncwarp();
        tc_fence_after();
        // This row's entries of the chunk: where the first is, and which is the last of the whole row
        const int chunk = (pc.kb_lo + j) / kPer >> p.chunk_shift, chunk_k = (chunk << p.chunk_shift) * (kPer * kBK);
        const int g0 = chunk_k >> p.group_shift, glast = groups - 1 - g0;
        const int k0 = (pc.kb_lo + j) * kBK - chunk_k;                 // the step's first element in the chunk
        const uint32_t ci = cbase + chunk - (pc.kb_lo / kPer >> p.chunk_shift), ts = ci - __umulhi(ci, p.t_inverse) * p.t_stages;
        uint32_t tbox = t_at + ts * (kTables * kBF * kTablePitch) + frow * kTablePitch, bias_off = kBF * kTablePitch;
        if (p.skewed) {
          const uint32_t at = (trow + g0) * entry, skew = (at + static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.scales))) & 15u;
          tbox += skew;
          if constexpr (QK != kMx4) bias_off += ((at + static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.biases))) & 15u) - skew;
        }
        // (a block at a time, not the whole step unrolled: the sixteen warps are at sixteen places of this code, and much more of it
        // no longer stays in the instruction caches)
        const int blocks = nkb - j < kStep ? nkb - j : kStep;
#pragma unroll 1
        for (int b = 0; b < blocks; ++b) {
          if (kPer == 1 && b == 1) {               // (float weights: a box is one block)
            __syncwarp();
            if (lane == 0) arrive_n(wempty + 8 * ws, 1);
            if (++ws == static_cast<uint32_t>(p.w_stages)) { ws = 0; ++wph; }
            if (!(ok = wait(wfull + 8 * ws, wph & 1u, 6))) break;
            __syncwarp();
          }
          // 16-byte chunk c of row r sits at chunk c ^ (r & 7) (the TMA unit's 128-byte swizzle): eight lanes read distinct banks
          const uint32_t first = wthread + ws * P::kWBytes + (static_cast<uint32_t>((j + b) % kPer * P::kRowBytes) ^ swizzle);
          uint32_t sc = 0u, bi = 0u;               // the half block's table entries
          auto entries = [&](int k) {
            const uint32_t at = tbox + min(k >> p.group_shift, glast) * entry;
            if constexpr (QK == kMx4) {
              sc = lds8(at);
            } else if (twide) {
              sc = lds32<0>(at);
              bi = lds32<0>(at + bias_off);
            } else {
              sc = lds16(at);
              bi = lds16(at + bias_off);
            }
          };
          if constexpr (QK != kFloat) entries(k0 + b * kBK);
#pragma unroll(QK == kAff8 ? 1 : 2)
          for (int h = 0; h < 2; ++h) {
            uint32_t packed[kHalfBytes / 4], out[16];
#pragma unroll
            for (int c = 0; c < kHalfBytes / 16; ++c) {
              const uint4 v = lds128<0>(first ^ ((h * (kHalfBytes / 16) + c) << 4));
              packed[c * 4] = v.x; packed[c * 4 + 1] = v.y; packed[c * 4 + 2] = v.z; packed[c * 4 + 3] = v.w;
            }
            if constexpr (QK != kFloat)
              if (h == 1 && p.group_shift == 5) entries(k0 + b * kBK + 32);
            if constexpr (QK == kFloat) {
#pragma unroll
              for (int e = 0; e < 16; ++e) out[e] = packed[e];
            } else if constexpr (QK == kMx4) {
              dequant_mx4<XT>(packed, sc, out);
            } else if constexpr (QK == kAff4 && SAME) {
              dequant_aff4<XT>(packed, __byte_perm(sc, sc, 0x1010), __byte_perm(bi, bi, 0x1010), mask, magic, out);
            } else if constexpr (QK == kAff8 && SAME && std::is_same<XT, __half>::value) {
              dequant_aff8_f16(packed, __byte_perm(sc, sc, 0x1010), __byte_perm(bi, bi, 0x1010), out);
            } else {
              const int td = SAME ? (std::is_same<XT, __nv_bfloat16>::value ? QMM_BF16 : QMM_F16) : p.table_dtype;
              const float fs = twide ? __uint_as_float(sc) : table_value(sc, td);
              const float fb = twide ? __uint_as_float(bi) : table_value(bi, td);
              if constexpr (QK == kAff8) dequant_aff8<XT>(packed, fs, fb, out);
              else if (twide) dequant_aff4_wide<XT>(packed, fs, fb, out);
              else dequant_aff4<XT>(packed, Half2Ops<XT>::pack(fs, fs), Half2Ops<XT>::pack(fb, fb), mask, magic, out);
            }
            tmem_st16(tmem_base + lane_addr + P::kACol0 + s * (32 * kStep) + b * 32 + h * 16, out);
          }
        }
        if (!ok) break;
        __syncwarp();
        // this warp's share of the step's part of the box has been read (a piece's last box may have fewer steps than its barrier counts)
        if (lane == 0) arrive_n(wempty + 8 * ws, kPer > 1 && i + 1 == steps ? P::kStepsPerBox - (j % kPer) / kStep : 1);
        tmem_wait_st();
        tc_fence_before();
        if constexpr (kPair) {                     // ... and this CTA's activations of the step have landed
          if (!(ok = wait(xfull + 8 * s, ph, 5))) break;
        }
        __syncwarp();
        if (lane == 0) {
          if constexpr (kPair) remote_arrive_n(a_bar + 8 * s, 1);
          else arrive_n(a_bar + 8 * s, 1);
        }
        s += kTeams;
        if (s >= static_cast<uint32_t>(kStages)) { s -= kStages; ph ^= 1u; }
        ws += kPer == 1 ? kTeams * kStep - (kStep - 1) : kTeams * kStep / kPer;
        while (ws >= static_cast<uint32_t>(p.w_stages)) { ws -= p.w_stages; ++wph; }
      }
      wbase += static_cast<uint32_t>(nkb + kPer - 1) / kPer;
      sbase += static_cast<uint32_t>(nkb + kStep - 1) / kStep;
      cbase += ((pc.kb_hi - 1) / kPer >> p.chunk_shift) - (pc.kb_lo / kPer >> p.chunk_shift) + 1;
      if (!ok) break;
      // ---- epilogue: the teams drain disjoint 32-column chunks of the accumulator ----
      if (!(ok = wait(d_full, piece & 1, 8))) break;
      __syncwarp();      // lanes leave the wait loop one by one; tcgen05.ld needs the whole warp
      tc_fence_after();
      constexpr int kCols = P::kCols;
      const int first_col = team * P::kTeamCols, end_col = min(first_col + P::kTeamCols, pc.rows);
      if (P::kMaySplit && p.cluster_adds) {        // this worker's share of the sums, over its activation ring (which is done with)
#pragma unroll 1
        for (int c0 = first_col; c0 < end_col; c0 += kCols) {
          uint32_t r[kCols];
          tmem_ld(tmem_base + lane_addr + c0, r);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < kCols; ++j) sts32(x_at + ((c0 + j) * kBF + frow) * 4, __uint_as_float(r[j]));
        }
        break;
      }
      auto drained = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (kPair) remote_arrive_n(d_bar, 1);
          else arrive_n(d_bar, 1);
        }
      };
      const bool mine = first_col < pc.rows;
      const bool whole = pc.begins && pc.ends, part_only = !pc.ends || p.split > 1;
      if (mine && !part_only && !whole) {          // the tile's earlier pieces, made by the workers before this one
        const int tile_box0 = pc.tile * walk.boxes;
        for (int v = worker - 1; ok && v >= 0; --v) {
          const unsigned long long* flag = p.ready + (static_cast<int64_t>(v) * kCtas + rank) * kDequantWarps + (warp - 2);
          const long long t0 = clock64();
          for (;;) {
            unsigned long long got;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(got) : "l"(flag) : "memory");
            if (got == p.epoch) break;
            if (clock64() - t0 > kSpinLimit) {
              asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(abort_at), "r"(9) : "memory");
              ok = false;
              break;
            }
          }
          if (Walk<BT, kPer>::first_box(p, v) <= tile_box0) break;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      // COLS rounded columns of the tile, two to a word, stored. Even N: neighbouring lanes (features) swap halves, so that
      // the even one stores both features of one token and the odd one those of the next.
      auto store_halves = [&](const auto& h, int c0) {
        constexpr int kPairs = sizeof(h) / 4;
        const int rows_left = feat_ok ? pc.rows - c0 : 0, n = static_cast<int>(p.N);
        uint16_t* y = reinterpret_cast<uint16_t*>(p.y) + ((pc.row0 + c0) * p.N + feat);
        if ((n & 1) == 0) {
          const int odd = lane & 1;
          const uint32_t swap = odd ? 0x3276u : 0x5410u;
          if (odd) y += n - 1;
#pragma unroll
          for (int j = 0; j < kPairs; ++j) {
            const uint32_t v = __byte_perm(h[j], __shfl_xor_sync(0xffffffffu, h[j], 1), swap);
            if (2 * j + odd < rows_left) *reinterpret_cast<uint32_t*>(y) = v;
            y += 2 * static_cast<int64_t>(n);
          }
        } else {
#pragma unroll
          for (int j = 0; j < kPairs; ++j) {
            if (2 * j < rows_left) y[0] = static_cast<uint16_t>(h[j]);
            if (2 * j + 1 < rows_left) y[n] = static_cast<uint16_t>(h[j] >> 16);
            y += 2 * static_cast<int64_t>(n);
          }
        }
      };
      auto round = [&](const uint32_t (&r)[kCols], uint32_t* h) {
        if (p.y_dtype == QMM_BF16) {
#pragma unroll
          for (int j = 0; j < kCols; j += 2) h[j / 2] = Half2Ops<__nv_bfloat16>::pack(__uint_as_float(r[j]), __uint_as_float(r[j + 1]));
        } else {
#pragma unroll
          for (int j = 0; j < kCols; j += 2) h[j / 2] = Half2Ops<__half>::pack(__uint_as_float(r[j]), __uint_as_float(r[j + 1]));
        }
      };
      if (P::kHeld && whole && !part_only && p.y_dtype != QMM_F32) {      // all of it into registers first: the next tile's MMAs need not wait for the stores
        uint32_t h[P::kTeamCols / 2];
#pragma unroll
        for (int i = 0; i < P::kTeamCols / kCols; ++i) {
          if (first_col + i * kCols < pc.rows) {
            uint32_t r[kCols];
            tmem_ld(tmem_base + lane_addr + first_col + i * kCols, r);
            tmem_wait_ld();
            round(r, h + i * (kCols / 2));
          }
        }
        drained();
        if (mine) store_halves(h, first_col);
        continue;
      }
#pragma unroll 1
      for (int c0 = first_col; c0 < end_col; c0 += kCols) {
        const int64_t in_partial = static_cast<int64_t>(c0) * kBF + frow;
        float sum[kCols];
        if (!part_only && !whole) {                // in K order: the workers' pieces, then this one
          const int tile_box0 = pc.tile * walk.boxes;
          int v = worker - 1;
          while (Walk<BT, kPer>::first_box(p, v) > tile_box0) --v;
#pragma unroll
          for (int j = 0; j < kCols; ++j) sum[j] = 0.0f;
          for (; v < worker; ++v) {
            const float* part = p.partial + (static_cast<int64_t>(v) * kCtas + rank) * (BT * kBF) + in_partial;
            float f[kCols];
            // (volatile: all requests go out before the first is waited for)
#pragma unroll
            for (int j = 0; j < kCols; ++j) asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(f[j]) : "l"(part + j * kBF));
#pragma unroll
            for (int j = 0; j < kCols; ++j) sum[j] += f[j];
          }
        }
        uint32_t r[kCols];
        tmem_ld(tmem_base + lane_addr + c0, r);
        tmem_wait_ld();
        if (c0 + kCols >= end_col) drained();      // this warp's last columns
        if (part_only) {
          float* part = p.partial + static_cast<int64_t>(blockIdx.x) * (BT * kBF) + in_partial;
#pragma unroll
          for (int j = 0; j < kCols; ++j) __stcg(part + j * kBF, __uint_as_float(r[j]));
          continue;
        }
        if (!whole) {
#pragma unroll
          for (int j = 0; j < kCols; ++j) r[j] = __float_as_uint(sum[j] + __uint_as_float(r[j]));
        }
        if (p.y_dtype == QMM_F32) {
          float* y = reinterpret_cast<float*>(p.y) + ((pc.row0 + c0) * p.N + feat);
          const int rows_left = feat_ok ? pc.rows - c0 : 0;
#pragma unroll
          for (int j = 0; j < kCols; ++j) {
            if (j < rows_left) *y = __uint_as_float(r[j]);
            y += p.N;
          }
        } else {
          uint32_t h[kCols / 2];
          round(r, h);
          store_halves(h, c0);
        }
      }
      if (!mine) drained();
      if (p.split > 1) break;
      if (mine && part_only) {                     // this warp's part of the partial tile is there
        if (lane == 0) {
          __threadfence();
          asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p.ready + static_cast<int64_t>(blockIdx.x) * kDequantWarps + (warp - 2)), "l"(p.epoch) : "memory");
        }
      } else if (mine && !whole) {                 // taken: a replay of this launch starts from flags that say nothing
        const int tile_box0 = pc.tile * walk.boxes;
        for (int v = worker - 1; v >= 0; --v) {
          if (lane == 0) p.ready[(static_cast<int64_t>(v) * kCtas + rank) * kDequantWarps + (warp - 2)] = 0ull;
          if (Walk<BT, kPer>::first_box(p, v) <= tile_box0) break;
        }
      }
    }
    tmem_wait_st();                                // (of a step that was given up)
    // ragged: rows past the last group are zero
    if (p.group_sizes) {
      const int64_t used = seg_row0[nseg];
      const int64_t total = (p.M - used) * p.N;
      constexpr int64_t nth = 32 * kDequantWarps;
      const int64_t tid = static_cast<int64_t>(blockIdx.x) * nth + (threadIdx.x - 64);
      for (int64_t i = tid; i < total; i += static_cast<int64_t>(gridDim.x) * nth) {
        const int64_t o = used * p.N + i;
        if (p.y_dtype == QMM_F32) reinterpret_cast<float*>(p.y)[o] = 0.0f;
        else reinterpret_cast<uint16_t*>(p.y)[o] = 0;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  __syncwarp();
  if (p.cluster_adds) {
    // ---- a cluster's workers add up their shares of the tile: each a stretch of the token rows, in K order ----
    cluster_barrier();
    if (warp >= 2 && warp < 2 + kDequantWarps && pc.rows > 0) {
      const int part = in_cluster / kCtas, c0 = pc.rows * part / p.split, c1 = pc.rows * (part + 1) / p.split;
      const int64_t feat = pc.f0 + rank * kBF + lane * 4;
#pragma unroll 2
      for (int c = c0 + warp - 2; c < c1; c += kDequantWarps) {
        const uint32_t at = x_at + (c * kBF + lane * 4) * 4;
        float4 sum = remote_ld128(in_cta(at, rank));
        for (int v = 1; v < p.split; ++v) {
          const float4 f = remote_ld128(in_cta(at, v * kCtas + rank));
          sum.x += f.x; sum.y += f.y; sum.z += f.z; sum.w += f.w;
        }
        const int64_t o = (pc.row0 + c) * p.N + feat;
        const float out[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (feat + i < p.N) {
            if (p.y_dtype == QMM_BF16) reinterpret_cast<__nv_bfloat16*>(p.y)[o + i] = __float2bfloat16_rn(out[i]);
            else if (p.y_dtype == QMM_F16) reinterpret_cast<__half*>(p.y)[o + i] = __float2half_rn(out[i]);
            else reinterpret_cast<float*>(p.y)[o + i] = out[i];
          }
        }
      }
    }
    __syncwarp();
  }
  if (kPair || p.cluster_adds) cluster_barrier();  // another CTA may still read or signal this one's memory until here
  if (warp == 1) {
    tc_fence_after();
    if constexpr (kPair)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
  if (threadIdx.x == 0) {
    int gave_up;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(gave_up) : "r"(abort_at) : "memory");
    if (gave_up) atomicCAS(p.status, 0, gave_up);
  }
}

// Adds up the partial tiles of a split product in K order and casts to y's type: a thread has four features of a token row.
//   partial [tile][split][CTA of a pair][tokens of a tile][128]
template <int BT>
__global__ void __launch_bounds__(256)
add_partials_kernel(const float* __restrict__ partial, const TcParams p, int ctas, int64_t token_tiles, int64_t ftiles) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");               // the partial tiles come from the grid before
  const int lane = threadIdx.x & 31;
  const int64_t rows = p.M * p.segments, units = rows * ftiles * ctas;
  for (int64_t u = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; u < units; u += static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5)) {
    const int64_t row = u / (ftiles * ctas), rest = u - row * (ftiles * ctas), ft = rest / ctas;
    const int rank = static_cast<int>(rest - ft * ctas);
    const int64_t seg = row / p.M, in_seg = row - seg * p.M, tt = in_seg / p.tile_rows, tile = (seg * token_tiles + tt) * ftiles + ft;
    const float* at = partial + ((tile * p.split * ctas + rank) * BT + (in_seg - tt * p.tile_rows)) * kBF + lane * 4;
    float4 sum = __ldcg(reinterpret_cast<const float4*>(at));
#pragma unroll 4
    for (int v = 1; v < p.split; ++v) {
      const float4 f = __ldcg(reinterpret_cast<const float4*>(at + static_cast<int64_t>(v) * ctas * BT * kBF));
      sum.x += f.x; sum.y += f.y; sum.z += f.z; sum.w += f.w;
    }
    const int64_t feat = (ft * ctas + rank) * kBF + lane * 4, o = row * p.N + feat;
    const float out[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (feat + i < p.N) {
        if (p.y_dtype == QMM_BF16) reinterpret_cast<__nv_bfloat16*>(p.y)[o + i] = __float2bfloat16_rn(out[i]);
        else if (p.y_dtype == QMM_F16) reinterpret_cast<__half*>(p.y)[o + i] = __float2half_rn(out[i]);
        else reinterpret_cast<float*>(p.y)[o + i] = out[i];
      }
    }
  }
}

// ---- host side ---------------------------------------------------------------------------

// A value for TcParams::epoch: no two launches of a process share one, and scratch that held anything else
// (float32 sums, zeros, other launches' values) does not hold it.
unsigned long long next_epoch() {
  static std::atomic<unsigned long long> count{0};
  return (count.fetch_add(1, std::memory_order_relaxed) + 1) * 0x9E3779B97F4A7C15ull;
}

// Shares below this many weight boxes cost more in filling their pipeline than the idle workers.
constexpr int kLeastBoxes = 2;
// (More of them of wide tiles write and read more partial sums than they save.)
constexpr int most_shares(int bt) { return bt >= 256 ? 8 : 16; }
// What handing partial tiles from worker to worker takes, in K blocks (us, shared out / a tile each: 64 rows 28672 x 4096, 224 tiles of 64
// blocks on 148 workers, 29.9 / 27.0 (before the producer's early start; 26.3 with it); 14336 x 4096, 112 tiles, 20.3 / 15.3; 11008 x 4096 18.4 / 14.7; 128 rows 28672 x 4096 35.7 / 33.0; 300 rows 14336 x 4096, 112 tiles on
// 74 pairs, 51 / 43; mxfp4 64 rows 28800 x 2880 27..29 / 25.6).
constexpr int kExchangeBlocks = 32;

// Clusters of `ctas` that fit the device at once.
template <typename Kernel>
int64_t max_clusters(Kernel kernel, int ctas, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = static_cast<unsigned>(ctas);
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return max_active_clusters(reinterpret_cast<const void*>(kernel), cfg, ctas);
}

template <int QK, typename XT, int BT, bool SAME>
int launch_tables(const qmm_problem& p, cudaStream_t stream) {
  using P = Plan<QK, BT>;
  const bool ragged = p.group_sizes != nullptr;
  const int64_t x_rows = ragged ? p.M : p.batch * p.M;
  const int64_t w_rows = (p.w_batch_stride ? p.batch : 1) * p.N;
  CUtensorMap xm, wm;
  int rc;
  if ((rc = tensor_map_2d(&xm, p.x_dtype, p.x, static_cast<uint64_t>(p.K), static_cast<uint64_t>(x_rows), static_cast<uint64_t>(p.K) * 2, kBK, BT / P::kCtas, 1)))
    return rc;
  const uint64_t wrow_bytes = static_cast<uint64_t>(p.K) * P::kBits / 8;
  if (QK == kFloat)
    rc = tensor_map_2d(&wm, p.x_dtype, p.w, static_cast<uint64_t>(p.K), static_cast<uint64_t>(w_rows), wrow_bytes, kBK, kBF, 1);
  else
    rc = tensor_map_2d(&wm, QMM_U8, p.w, wrow_bytes, static_cast<uint64_t>(w_rows), wrow_bytes, kBoxBytes, kBF, 1);
  if (rc) return rc;
  const ScratchBlock* block = scratch_override();
  TcParams tp = {};
  tp.scales = p.scales; tp.biases = p.biases; tp.y = p.y; tp.group_sizes = p.group_sizes;
  tp.status = block ? block->status : device_status_word();
  if (!tp.status) return fail(QMM_ERR_CUDA, "could not allocate the device status word");
  tp.M = p.M; tp.K = static_cast<int>(p.K); tp.N = p.N;
  tp.segments = static_cast<int>(p.batch);
  tp.w_seg_rows = p.w_batch_stride ? p.N : 0;
  const int group = QK == kMx4 ? 32 : p.group_size;
  tp.group_shift = group == 128 ? 7 : group == 64 ? 6 : 5;
  tp.table_dtype = p.table_dtype; tp.y_dtype = p.y_dtype;

  // The rings: as many weight boxes as fit next to the table chunks that go with them. Entries travel a sector of a row at a time: the copies are
  // per row, and what they cost the producer is the lines that they touch (8 bytes of 32 rows an instruction, with every box, was what bound
  // 64 rows: see the head of the file).
  int chunk_boxes = 0, chunk_slot = 0;
  if (QK != kFloat) {
    tp.table_entry = QK == kMx4 ? 1 : (p.table_dtype == QMM_F32 ? 4 : 2);
    const int box_bytes = (P::kPer * kBK >> tp.group_shift) * tp.table_entry, row_table = static_cast<int>(p.K >> tp.group_shift) * tp.table_entry;
    const uintptr_t start = reinterpret_cast<uintptr_t>(p.scales) | (QK == kMx4 ? 0 : reinterpret_cast<uintptr_t>(p.biases));
    tp.skewed = row_table % 16 != 0 || start % 16 != 0;
    while (box_bytes << tp.chunk_shift < kChunkBytes) ++tp.chunk_shift;
    chunk_boxes = 1 << tp.chunk_shift;
    tp.table_bytes = w_rows * row_table;
    chunk_slot = (QK == kMx4 ? 1 : 2) * kBF * kTablePitch;
  }
  // Chunks for every box of the ring that lies ahead of the one that is read, if they fit (with fewer the producer waits a little earlier).
  const int room = P::kBudget - P::kFixed;
  for (tp.w_stages = P::kMostBoxes; tp.w_stages >= P::kLeastPlaces; --tp.w_stages) {
    if (QK == kFloat) {
      if (tp.w_stages * P::kWBytes <= room) break;
      continue;
    }
    tp.t_stages = 1 + (tp.w_stages - 1 + chunk_boxes - 1) / chunk_boxes;
    if (tp.t_stages < 2) tp.t_stages = 2;
    if (tp.w_stages == P::kLeastPlaces)
      while (tp.t_stages > 2 && tp.w_stages * P::kWBytes + tp.t_stages * chunk_slot > room) --tp.t_stages;
    if (tp.w_stages * P::kWBytes + tp.t_stages * chunk_slot <= room) break;
  }
  if (tp.w_stages < P::kLeastPlaces) return fail(QMM_ERR_UNSUPPORTED, "qmm_gemm_tc_kernel: the weight ring does not fit shared memory");
  const size_t smem = P::kFixed + static_cast<size_t>(tp.w_stages) * P::kWBytes + static_cast<size_t>(tp.t_stages) * chunk_slot;
  tp.w_inverse = 0xFFFFFFFFu / tp.w_stages + 1;
  tp.t_inverse = tp.t_stages ? 0xFFFFFFFFu / tp.t_stages + 1 : 0;

  auto kernel = qmm_gemm_tc_kernel<QK, XT, BT, SAME>;
  static bool configured[kMaxDevices] = {};     // the attribute is per device
  const int dev = current_device();
  if (dev < 0) return QMM_ERR_DEVICE;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, P::kBudget);
    if (e != cudaSuccess) return fail(QMM_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    configured[dev] = true;
  }
  const int sms = device_sm_count();
  const int num_kb = static_cast<int>((p.K + kBK - 1) / kBK), boxes = (num_kb + P::kPer - 1) / P::kPer;
  const int64_t ftiles = (p.N + kBF * P::kCtas - 1) / (kBF * P::kCtas), ttiles = (p.M + BT - 1) / BT;
  int64_t tiles = ragged ? (ttiles + p.batch) * ftiles : p.batch * ttiles * ftiles;      // (ragged: at most)
  tp.tile_rows = BT;
  int64_t workers = sms / P::kCtas;
  int64_t shared = 0, split = 1;
  if (ragged) {
    if (tiles < workers) workers = tiles;
  } else if (tiles * 2 <= workers) {
    // Few tiles: several workers share a tile's K, at least kLeastBoxes each. Where clusters of them (8 CTAs at most) fill half of the
    // machine they add up over distributed shared memory: no scratch, one kernel, the sum spread over the cluster (64 rows of
    // 4096 x 14336: 31.4 us with a second kernel, 21.9). Where they do not, more workers to a tile and a second kernel.
    split = workers / tiles;
    if (split > boxes / kLeastBoxes) split = boxes / kLeastBoxes;
    if (split > most_shares(BT)) split = most_shares(BT);
    if (split < 1) split = 1;
    int64_t in_cluster = split < 8 / P::kCtas ? split : 8 / P::kCtas;
    while (in_cluster > 1 && max_clusters(kernel, static_cast<int>(in_cluster) * P::kCtas, smem) < tiles) --in_cluster;
    if (P::kMaySplit && in_cluster > 1 && tiles * in_cluster * 2 >= workers) {
      split = in_cluster;
      tp.cluster_adds = 1;
    }
    workers = tiles * split;
  } else {
    // Otherwise a tile each, in rounds; the last whole round and what is left over are shared out evenly by boxes, if that
    // shortens it by more than the exchange of partial tiles takes.
    const int64_t rest = tiles % workers, rounds = tiles / workers;
    const int64_t region = rounds ? workers + rest : tiles;
    if (rest && (rounds ? 2 : 1) * boxes - region * boxes / workers > kExchangeBlocks / P::kPer) shared = region;
    // Less than a round that is not shared out is as long as its longest tile: the shortest tiles that are one round still take its place (down to
    // 160 tokens, below which the dequantization is what a K block costs). 512 rows mxfp4 5760 x 2880: 46 tiles of 256 tokens on 74 pairs, 69 of 192, 20.5 -> 18.8 us;
    // 300 rows 6144 x 4096: 48, 48 of 160 and 140 instead of 256 and 44, 23.0 -> 19.5; 280 rows mxfp4 5760 x 2880 17.5 -> 16.0; 384 rows 8192 x 2048 8-bit 16.2 -> 15.7.
    if (!shared && !rounds && P::kPair)
      for (int h = 160; h < BT; h += 32) {
        const int64_t shorter = p.batch * ((p.M + h - 1) / h) * ftiles;
        if (shorter > workers) continue;
        tp.tile_rows = h;
        tiles = shorter;
        break;
      }
    if (!shared && tiles < workers) workers = tiles;
  }
  // Partial tiles: the caller's static block (qmm_quantized_matmul_static) or a stream-ordered allocation. No scratch,
  // no sharing.
  void* scratch = nullptr;
  if (shared || (split > 1 && !tp.cluster_adds)) {
    const size_t per_worker = P::kCtas * (static_cast<size_t>(BT) * kBF * sizeof(float) + (shared ? kDequantWarps * sizeof(unsigned long long) : 0));
    if (block) {
      // (a call is refused when the partial results of its K shares as whole float32 matrices exceed the block)
      const int64_t old_tiles = ttiles * ((p.N + kBF - 1) / kBF);
      int64_t s = p.batch != 1 || (p.N & 3) ? 1 : sms / old_tiles;
      if (s > num_kb / 8) s = num_kb / 8;
      if (s > 8) s = 8;
      const size_t need = static_cast<size_t>(s < 2 ? 0 : s) * p.M * p.N * sizeof(float);
      if (need > block->bytes)
        return fail(QMM_ERR_TOO_LARGE, "split product needs %zu bytes of scratch, the static block has %zu", need, block->bytes);
      if (split > 1)
        while (split > 1 && per_worker * tiles * split > block->bytes) --split;
      if (split > 1) workers = tiles * split;
      if (per_worker * workers <= block->bytes) tp.partial = static_cast<float*>(block->ptr);
    } else {
      tp.partial = static_cast<float*>(scratch = scratch_alloc(per_worker * workers, stream));
    }
    if (!tp.partial || (!shared && split == 1)) {
      shared = 0;
      split = 1;
      if (tiles < workers) workers = tiles;
    }
  }
  tp.split = static_cast<int>(split);
  if (shared) {
    tp.ready = reinterpret_cast<unsigned long long*>(tp.partial + static_cast<int64_t>(P::kCtas) * workers * BT * kBF);
    tp.epoch = next_epoch();
    tp.shared_tiles = static_cast<int>(shared);
    tp.share = static_cast<unsigned>(shared * boxes / workers);
    tp.share_more = static_cast<unsigned>(shared * boxes % workers);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(workers * P::kCtas));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  const int cluster = P::kCtas * (tp.cluster_adds ? tp.split : 1);
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kernel, xm, wm, tp);      // a failure stays as the last error: check_launch reports it
  count_launch();
  if (split > 1 && !tp.cluster_adds) {
    const int64_t rows = p.M * p.batch, warps = rows * ftiles * P::kCtas;
    const int64_t most = static_cast<int64_t>(sms) * 8;
    launch_early(add_partials_kernel<BT>, static_cast<unsigned>((warps + 7) / 8 < most ? (warps + 7) / 8 : most), 256, 0, stream,
                 tp.partial, tp, P::kCtas, ttiles, ftiles);
    count_launch();
  }
  if (scratch) scratch_free(scratch, stream);
  return check_launch("qmm_gemm_tc_kernel");
}

template <int QK, typename XT, int BT>
int launch_cfg(const qmm_problem& p, cudaStream_t stream) {
  if constexpr (QK == kAff4 || QK == kAff8)
    if (p.table_dtype != (std::is_same<XT, __nv_bfloat16>::value ? QMM_BF16 : QMM_F16)) return launch_tables<QK, XT, BT, false>(p, stream);
  return launch_tables<QK, XT, BT, true>(p, stream);
}

template <int QK, typename XT>
int launch_bt(const qmm_problem& p, cudaStream_t stream) {
  // Token-tile width: wide tiles amortize the dequantization, narrow ones waste less MMA
  // work on short row runs.
  const int64_t rows = p.group_sizes ? (p.M + p.batch - 1) / (p.batch ? p.batch : 1) : p.M;
  if (rows > 128) return launch_cfg<QK, XT, 256>(p, stream);
  if (rows > 64) return launch_cfg<QK, XT, 128>(p, stream);
  return launch_cfg<QK, XT, 64>(p, stream);
}

template <int QK>
int launch_xt(const qmm_problem& p, cudaStream_t stream) {
  if (p.x_dtype == QMM_BF16) return launch_bt<QK, __nv_bfloat16>(p, stream);
  return launch_bt<QK, __half>(p, stream);
}

}  // namespace

bool gemm_tc_supports(const qmm_problem& p) {
  if (p.x_dtype != QMM_BF16 && p.x_dtype != QMM_F16) return false;
  if (p.lhs_idx || p.rhs_idx) return false;                   // unsorted gathers go elsewhere
  if (p.batch > kMaxSegments) return false;
  if (p.K < kBK || p.K % (p.mode == QMM_MODE_FLOAT ? 8 : 32) || p.K >= (1LL << 30)) return false;
  if ((p.K * 2) % 16) return false;
  if (!p.group_sizes && p.batch > 1 && p.x_batch_stride != p.M * p.K) return false;
  if (!p.group_sizes && p.batch > 1 && p.y_batch_stride != p.M * p.N) return false;
  // (tiles are counted in 32 bits)
  if (((p.M + 63) / 64 + p.batch) * (p.group_sizes ? 1 : p.batch) * ((p.N + 127) / 128) * ((p.K + 63) / 64) >= (1LL << 31)) return false;
  if (p.M * (p.group_sizes ? 1 : p.batch) >= (1LL << 31) || p.N * p.batch >= (1LL << 31)) return false;
  return true;
}

int launch_gemm_tc(const qmm_problem& p, cudaStream_t stream) {
  if (p.mode == QMM_MODE_FLOAT) return launch_xt<kFloat>(p, stream);
  if (p.mode == QMM_MODE_MXFP4) return launch_xt<kMx4>(p, stream);
  if (p.bits == 8) return launch_xt<kAff8>(p, stream);
  return launch_xt<kAff4>(p, stream);
}

}  // namespace qmm
