// Packing a quantized Dense layer's stored arrays on the device (keras' int4 layout: two output columns per byte,
// tables per group of input rows; tests/test_qmm.py:179-199): the code transpose and the table transpose as one
// pass each, with the facts the packer decides from (src/metaljax/qmm.py:206-286, 1204-1247) gathered on the way.
//
// Through generic tensor passes (unpack to int16, transpose, widen to int64, minimum and maximum, repack, expanded
// scale and zero maps, ...) a [4096, 14336] layer took 2.8 ms and a dozen waits for the device; the bytes that have to move
// are 69 MB, 11 us of HBM. As a memset, three kernels, a copy of the facts and an event it took 84 us, 30 of them the kernels'; now one kernel does all
// of it -- a CTA has a tile of codes or of tables -- and its last CTA writes the facts to host memory that the call watches: 42 us a call from Python
// (the codes alone, 59 MB, take 17).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <sched.h>

#include <mutex>
#include <type_traits>
#include <vector>

#include "../../include/qmm.h"
#include "qmm_internal.h"

namespace qmm {
namespace {

constexpr int kTileN = 128, kTileK = 256;          // output rows and codes of a CTA's tile: 64 bytes of an input row, 128-byte output lines
constexpr uint32_t kMix = 2246822519u;

// packed int8 [K, bytes] (byte j of row k: columns 2j, 2j + 1, two's complement nibbles) -> out words [N, K / 8], codes + 8.
// A thread owns 4 bytes (8 columns) x 8 rows, twice: eight 4-byte reads, then the even rows' bytes and the odd rows' as columns, of which
// a select each makes an even and an odd column's word. `digest` accumulates the content digest of the words (the sharing table's key).
// (Five instructions a nibble pair to squeeze each column's nibbles together and a word at a time out of a tile with four-way bank conflicts
// kept it at 22.2 us for the codes of [4096, 14336], 16.9 so; rows that start on no word took four loads for one: [4096, 14337] a whole call 68.6 -> 57.0.)
struct CodeTile {
  alignas(16) uint32_t tile[kTileN * kTileK / 8];  // [column][word], a row of words turned by 4 for every eight columns (see word_at)
  unsigned long long warp_sum[8];
};
constexpr int kTileWords = kTileK / 8;
__device__ __forceinline__ int word_at(int column, int word) { return column * kTileWords + ((word + (column >> 3) * 4) & (kTileWords - 1)); }
__device__ __forceinline__ void transpose_pack(CodeTile& shared, int n0, int k0, const uint8_t* __restrict__ packed, uint32_t* __restrict__ out, int K, int N, int bytes,
                                               bool words4, unsigned long long* digest) {
  auto& tile = shared.tile;
  auto& warp_sum = shared.warp_sum;
  const int q = threadIdx.x & 15, byte0 = n0 / 2 + q * 4;            // which 4 bytes of a row
  const bool whole = words4 && byte0 + 4 <= bytes;
  const uintptr_t first = reinterpret_cast<uintptr_t>(packed), end = first + static_cast<int64_t>(K) * bytes;
  constexpr int kParts = kTileK / 128;                                 // 128 rows at a time, all requests first
  uint32_t r[kParts][8];
#pragma unroll
  for (int h = 0; h < kParts; ++h) {
    const int row0 = k0 + h * 128 + (threadIdx.x >> 4) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      r[h][i] = 0u;
      if (row0 + i < K) {
        const uint8_t* src = packed + static_cast<int64_t>(row0 + i) * bytes + byte0;
        const uintptr_t at = reinterpret_cast<uintptr_t>(src), word = at & ~uintptr_t(3);
        if (whole) {
          r[h][i] = __ldcs(reinterpret_cast<const uint32_t*>(src));
        } else if (byte0 + 4 <= bytes && word >= first && word + 8 <= end) {       // rows that start on no word: out of the two that it lies in
          r[h][i] = __funnelshift_r(__ldg(reinterpret_cast<const uint32_t*>(word)), __ldg(reinterpret_cast<const uint32_t*>(word) + 1), static_cast<unsigned>(at & 3) * 8);
        } else {
          for (int b = 0; b < 4; ++b)
            if (byte0 + b < bytes) r[h][i] |= static_cast<uint32_t>(src[b]) << (8 * b);
        }
      }
    }
  }
  // column c of four rows as one word: bytes transposed
  auto transpose = [](uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&t)[4]) {
    const uint32_t x0 = __byte_perm(a, b, 0x5140), x1 = __byte_perm(a, b, 0x7362), y0 = __byte_perm(c, d, 0x5140), y1 = __byte_perm(c, d, 0x7362);
    t[0] = __byte_perm(x0, y0, 0x5410); t[1] = __byte_perm(x0, y0, 0x7632);
    t[2] = __byte_perm(x1, y1, 0x5410); t[3] = __byte_perm(x1, y1, 0x7632);
  };
#pragma unroll
  for (int h = 0; h < kParts; ++h) {
    const int o = h * 16 + (threadIdx.x >> 4);
    uint32_t even[4], odd[4];                      // of rows 0, 2, 4, 6 and 1, 3, 5, 7; two's complement + 8 is an exclusive or with 8
#pragma unroll
    for (int i = 0; i < 8; ++i) r[h][i] ^= 0x88888888u;
    transpose(r[h][0], r[h][2], r[h][4], r[h][6], even);
    transpose(r[h][1], r[h][3], r[h][5], r[h][7], odd);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      tile[word_at(q * 8 + 2 * c, o)] = (even[c] & 0x0F0F0F0Fu) | ((odd[c] << 4) & 0xF0F0F0F0u);
      tile[word_at(q * 8 + 2 * c + 1, o)] = ((even[c] >> 4) & 0x0F0F0F0Fu) | (odd[c] & 0xF0F0F0F0u);
    }
  }
  __syncthreads();
  // four words of a column at a time
  const int words = K / 8, w = (threadIdx.x & 7) * 4, wk = k0 / 8 + w;
  const bool quads = (reinterpret_cast<uintptr_t>(out) & 15) == 0;     // (K is a multiple of 32: its rows of words then start there too)
  unsigned long long sum = 0;
#pragma unroll 4
  for (int i = threadIdx.x >> 3; i < kTileN; i += 32) {
    const int n = n0 + i;
    if (n < N && wk < words) {
      const uint4 v = *reinterpret_cast<const uint4*>(&tile[word_at(i, w)]);
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
      const int64_t at = static_cast<int64_t>(n) * words + wk;
      if (quads) __stcs(reinterpret_cast<uint4*>(out + at), v);
      const uint32_t mixed = static_cast<uint32_t>(at) * 2654435761u;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (!quads) __stcs(out + at + j, u[j]);
        uint32_t m = (u[j] ^ (mixed + static_cast<uint32_t>(j) * 2654435761u)) * kMix;
        m ^= m >> 15;
        sum += m;
      }
    }
  }
  for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) sum += warp_sum[i];
    atomicAdd(digest, sum);
  }
}
__global__ void __launch_bounds__(256, 8)
transpose_pack_kernel(const uint8_t* __restrict__ packed, uint32_t* __restrict__ out, int K, int N, int bytes, bool words4, unsigned long long* digest) {
  __shared__ CodeTile shared;
  transpose_pack(shared, blockIdx.x * kTileN, blockIdx.y * kTileK, packed, out, K, N, bytes, words4, digest);
}

template <typename T>
__device__ __forceinline__ float as_float(T v) { return static_cast<float>(v); }
template <>
__device__ __forceinline__ float as_float(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float as_float(__half v) { return __half2float(v); }

template <typename T>
__device__ __forceinline__ T to_table(float v) {
  if constexpr (sizeof(T) == 4) return v;
  else if constexpr (std::is_same<T, __nv_bfloat16>::value) return __float2bfloat16_rn(v);
  else return __float2half_rn(v);
}

// Facts about scale / zero [G, N] (group = K / G rows): bit 0 not constant within 128 codes, 1 within 64, 2 the biases do not narrow
// to the scales' type exactly, 3 something the packer has to look at itself (a NaN, a zero point that is no integer or out of range).
template <typename S, typename Z>
__device__ __forceinline__ unsigned facts_of(const S* __restrict__ scale, const Z* __restrict__ zero, int j, int n, int N, int group) {
  unsigned f = 0;
  const int64_t i = static_cast<int64_t>(j) * N + n;
  const float s = as_float(scale[i]), z = zero ? as_float(zero[i]) : 0.0f;
  if (!(s == s) || !(z == z) || rintf(z) != z || fabsf(z) > 32768.0f) f |= 8u;
  const float b = -(s * (z + 8.0f));
  if (as_float(to_table<S>(b)) != b) f |= 4u;
  // blocks of 128 and of 64 codes that this group's first code is not the start of: the same entries as their first group's?
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int g = t ? 64 : 128;
    const int64_t at = static_cast<int64_t>(j) * group;
    const int64_t first = at / g * g / group;      // group of the block's first code
    if (at % g != 0 && first != j) {
      const float s0 = as_float(scale[first * N + n]), z0 = zero ? as_float(zero[first * N + n]) : 0.0f;
      if (!(s == s0) || !(z == z0)) f |= 1u << t;
    }
  }
  return f;
}
template <typename S, typename Z>
__global__ void table_facts_kernel(const S* __restrict__ scale, const Z* __restrict__ zero, int G, int N, int K, unsigned* __restrict__ facts) {
  unsigned f = 0;
  const int64_t total = static_cast<int64_t>(G) * N;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int j = static_cast<int>(i / N);
    f |= facts_of(scale, zero, j, static_cast<int>(i - static_cast<int64_t>(j) * N), N, K / G);
  }
  f = __reduce_or_sync(0xffffffffu, f);
  if ((threadIdx.x & 31) == 0 && f) atomicOr(facts, f);
}

// scale, zero [G, N] -> scales, biases = -scale (zero + 8) [N, K / g], transposed through shared memory.
struct TableTile {
  float ts[32][33], tb[32][33];
};
// The 32 x 32 tile at (n0, j0); FACTS: also what it says about the stored entries that it meets (all of them, where no entry stands for two groups).
template <bool FACTS, typename S, typename Z, typename T>
__device__ __forceinline__ unsigned table_tile(TableTile& shared, int n0, int j0, const S* __restrict__ scale, const Z* __restrict__ zero, T* __restrict__ scales, T* __restrict__ biases,
                                               int G, int N, int K, int g) {
  const int groups = K / g, group = K / G;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  unsigned f = 0;
  for (int i = ty; i < 32; i += 8) {
    const int j = j0 + i, n = n0 + tx;
    if (j < groups && n < N) {
      const int stored = static_cast<int>(static_cast<int64_t>(j) * g / group);
      const int64_t at = static_cast<int64_t>(stored) * N + n;
      const float s = as_float(scale[at]), z = zero ? as_float(zero[at]) : 0.0f;
      shared.ts[i][tx] = s;
      shared.tb[i][tx] = -(s * (z + 8.0f));
      if (FACTS) f |= facts_of(scale, zero, stored, n, N, group);
    }
  }
  __syncthreads();
  for (int i = ty; i < 32; i += 8) {
    const int n = n0 + i, j = j0 + tx;
    if (j < groups && n < N) {
      const int64_t at = static_cast<int64_t>(n) * groups + j;
      scales[at] = to_table<T>(shared.ts[tx][i]);
      biases[at] = to_table<T>(shared.tb[tx][i]);
    }
  }
  return f;
}
template <typename S, typename Z, typename T>
__global__ void __launch_bounds__(256)
tables_kernel(const S* __restrict__ scale, const Z* __restrict__ zero, T* __restrict__ scales, T* __restrict__ biases, int G, int N, int K, int g) {
  __shared__ TableTile shared;
  table_tile<false>(shared, blockIdx.x * 32, blockIdx.y * 32, scale, zero, scales, biases, G, N, K, g);
}

// A whole layer. What its CTAs add up is in `sums` (nought before and after), and the last one reports it to the host.
struct Sums {
  unsigned long long digest;
  unsigned flags, done;
};
struct Told {                        // host memory
  unsigned long long digest, flags, ticket;
};
template <typename S, typename Z, typename T>
__global__ void __launch_bounds__(256, 8)
pack_layer_kernel(const uint8_t* __restrict__ packed, uint32_t* __restrict__ out, const S* __restrict__ scale, const Z* __restrict__ zero, T* __restrict__ scales, T* __restrict__ biases,
                  int K, int N, int G, int g, int bytes, bool words4, int table_tiles, Sums* sums, volatile Told* told, unsigned long long ticket) {
  __shared__ union { CodeTile codes; TableTile tables; } shared;
  int t = static_cast<int>(blockIdx.x);
  if (t < table_tiles) {
    const int across = (N + 31) / 32;
    unsigned f = table_tile<true>(shared.tables, t % across * 32, t / across * 32, scale, zero, scales, biases, G, N, K, g);
    f = __reduce_or_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0 && f) atomicOr(&sums->flags, f);
    __syncthreads();
  } else {
    t -= table_tiles;
    const int across = (N + kTileN - 1) / kTileN;
    transpose_pack(shared.codes, t % across * kTileN, t / across * kTileK, packed, out, K, N, bytes, words4, &sums->digest);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&sums->done, 1u) == gridDim.x - 1) {
      __threadfence();
      told->digest = atomicExch(&sums->digest, 0ull);
      told->flags = atomicExch(&sums->flags, 0u);
      atomicExch(&sums->done, 0u);
      __threadfence_system();
      told->ticket = ticket;
    }
  }
}

// f(S(), Z()) for a scale and a zero type.
template <typename F>
int with_types(int scale_dtype, int zero_dtype, F&& f) {
  auto z = [&](auto s) -> int {
    switch (zero_dtype) {
      case QMM_BF16: return f(s, __nv_bfloat16());
      case QMM_F16: return f(s, __half());
      case QMM_F32: return f(s, float());
      case QMM_U8: return f(s, uint8_t());
      case QMM_I8: return f(s, int8_t());
    }
    return fail(QMM_ERR_DTYPE, "pack_dense: zero points are bf16, f16, f32, int8 or uint8");
  };
  switch (scale_dtype) {
    case QMM_BF16: return z(__nv_bfloat16());
    case QMM_F16: return z(__half());
    case QMM_F32: return z(float());
  }
  return fail(QMM_ERR_DTYPE, "pack_dense: scales are bf16, f16 or f32");
}

// Sums and host words, one pair per call that is under way; they stay for later calls of the device (qmm_release_scratch gives them back).
struct Slot {
  Sums* sums;
  volatile Told* told;
  unsigned long long ticket;
};
std::mutex g_slots_mutex;
std::vector<Slot> g_slots[kMaxDevices];

bool take_slot(int dev, cudaStream_t stream, Slot* out) {
  {
    std::lock_guard<std::mutex> lock(g_slots_mutex);
    if (!g_slots[dev].empty()) {
      *out = g_slots[dev].back();
      g_slots[dev].pop_back();
      ++out->ticket;
      return true;
    }
  }
  void *d = nullptr, *h = nullptr;
  if (cudaMalloc(&d, sizeof(Sums)) != cudaSuccess || cudaMemsetAsync(d, 0, sizeof(Sums), stream) != cudaSuccess ||
      cudaHostAlloc(&h, sizeof(Told), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    if (d) cudaFree(d);
    return false;
  }
  count_alloc();
  out->sums = static_cast<Sums*>(d);
  out->told = static_cast<volatile Told*>(h);
  out->told->ticket = 0;
  out->ticket = 1;
  return true;
}

}  // namespace

void release_pack_slots() {
  const int dev = current_device();
  if (dev < 0) return;
  std::vector<Slot> slots;
  {
    std::lock_guard<std::mutex> lock(g_slots_mutex);
    slots.swap(g_slots[dev]);
  }
  for (const Slot& s : slots) {
    cudaFree(s.sums);
    cudaFreeHost(const_cast<Told*>(s.told));
  }
}

}  // namespace qmm

using namespace qmm;

extern "C" int qmm_pack_dense_layer(const void* packed, uint32_t* words, const void* scale, const void* zero, int scale_dtype, int zero_dtype, void* scales, void* biases, int narrow,
                                    int64_t G, int64_t N, int64_t K, int group_size, uint64_t* digest, uint32_t* facts, void* stream) {
  if (!packed || !words || !scale || !scales || !biases || !digest || !facts) return fail(QMM_ERR_NULL, "pack_dense_layer: null pointer");
  if (K < 32 || K % 32 || N < 1 || K >= (1LL << 24) || N >= (1LL << 30) || G < 1 || K % G || (K / G) % 32) return fail(QMM_ERR_SHAPE, "pack_dense_layer: groups are multiples of 32 codes");
  if (group_size < 32 || (K / G) % group_size) return fail(QMM_ERR_SHAPE, "pack_dense_layer: the group size divides the stored groups");
  const int64_t table_tiles = (N + 31) / 32 * ((K / group_size + 31) / 32), code_tiles = (N + kTileN - 1) / kTileN * ((K + kTileK - 1) / kTileK);
  if (table_tiles + code_tiles >= (1LL << 31)) return fail(QMM_ERR_SHAPE, "pack_dense_layer: the layer is too large");
  const int rt = with_types(scale_dtype, zero ? zero_dtype : QMM_U8, [](auto, auto) -> int { return QMM_OK; });
  if (rt) return rt;                               // (before a slot is taken: one that does not come back is lost)
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone)
    return fail(QMM_ERR_UNSUPPORTED, "pack_dense_layer: waits for the device, which a stream that is being captured cannot");
  const int dev = current_device();
  if (dev < 0) return QMM_ERR_DEVICE;
  Slot slot;
  if (!take_slot(dev, st, &slot)) return fail(QMM_ERR_CUDA, "pack_dense_layer: no memory to report to");
  const int64_t bytes = (N + 1) / 2;
  const bool words4 = bytes % 4 == 0 && reinterpret_cast<uintptr_t>(packed) % 4 == 0;
  const int rc = with_types(scale_dtype, zero ? zero_dtype : QMM_U8, [&](auto s, auto z) -> int {
    using S = decltype(s);
    using Z = decltype(z);
    auto launch = [&](auto t) -> int {
      using T = decltype(t);
      pack_layer_kernel<S, Z, T><<<static_cast<unsigned>(table_tiles + code_tiles), 256, 0, st>>>(
          static_cast<const uint8_t*>(packed), words, static_cast<const S*>(scale), static_cast<const Z*>(zero), static_cast<T*>(scales), static_cast<T*>(biases), static_cast<int>(K),
          static_cast<int>(N), static_cast<int>(G), group_size, static_cast<int>(bytes), words4, static_cast<int>(table_tiles), slot.sums, slot.told, slot.ticket);
      count_launch();
      return check_launch("pack_layer_kernel");
    };
    return narrow ? launch(s) : launch(float());
  });
  if (rc) return rc;                               // (the slot is left out of the pool: its sums may not be nought)
  auto arrived = [&] { return slot.told->ticket == slot.ticket; };
  for (unsigned spins = 1; !arrived(); ++spins) {
    if (spins % 64) continue;
    sched_yield();
    const cudaError_t e = cudaStreamQuery(st);
    if (e != cudaErrorNotReady && !arrived()) return fail(QMM_ERR_CUDA, "pack_dense_layer: the kernel did not report: %s", cudaGetErrorString(e));
  }
  *digest = slot.told->digest;
  *facts = static_cast<uint32_t>(slot.told->flags);
  std::lock_guard<std::mutex> lock(g_slots_mutex);
  g_slots[dev].push_back(slot);
  return QMM_OK;
}

extern "C" int qmm_pack_dense_codes(const void* packed, uint32_t* words, int64_t K, int64_t N, uint64_t* digest, void* stream) {
  if (!packed || !words || !digest) return fail(QMM_ERR_NULL, "pack_dense_codes: null pointer");
  if (K < 32 || K % 32 || N < 1 || K >= (1LL << 24) || N >= (1LL << 30)) return fail(QMM_ERR_SHAPE, "pack_dense_codes: K is a multiple of 32");
  const int64_t bytes = (N + 1) / 2;
  const dim3 grid(static_cast<unsigned>((N + kTileN - 1) / kTileN), static_cast<unsigned>((K + kTileK - 1) / kTileK));
  if (grid.y > 65535) return fail(QMM_ERR_SHAPE, "pack_dense_codes: K is too long");
  const bool words4 = bytes % 4 == 0 && reinterpret_cast<uintptr_t>(packed) % 4 == 0;
  transpose_pack_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint8_t*>(packed), words, static_cast<int>(K), static_cast<int>(N),
                                                                             static_cast<int>(bytes), words4, reinterpret_cast<unsigned long long*>(digest));
  count_launch();
  return check_launch("transpose_pack_kernel");
}

extern "C" int qmm_pack_dense_facts(const void* scale, const void* zero, int scale_dtype, int zero_dtype, int64_t G, int64_t N, int64_t K, uint32_t* facts, void* stream) {
  if (!scale || !facts) return fail(QMM_ERR_NULL, "pack_dense_facts: null pointer");
  if (G < 1 || N < 1 || K % G || (K / G) % 32 || G >= (1LL << 30) || N >= (1LL << 30) || K >= (1LL << 30)) return fail(QMM_ERR_SHAPE, "pack_dense_facts: groups are multiples of 32 codes");
  const int64_t total = G * N, cap = static_cast<int64_t>(device_sm_count()) * 8;
  const int64_t blocks = (total + 255) / 256 < cap ? (total + 255) / 256 : cap;
  return with_types(scale_dtype, zero ? zero_dtype : QMM_U8, [&](auto s, auto z) -> int {
    using S = decltype(s);
    using Z = decltype(z);
    table_facts_kernel<S, Z><<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const S*>(scale), static_cast<const Z*>(zero), static_cast<int>(G), static_cast<int>(N), static_cast<int>(K), facts);
    count_launch();
    return check_launch("table_facts_kernel");
  });
}

extern "C" int qmm_pack_dense_tables(const void* scale, const void* zero, int scale_dtype, int zero_dtype, void* scales, void* biases, int narrow, int64_t G, int64_t N,
                                     int64_t K, int group_size, void* stream) {
  if (!scale || !scales || !biases) return fail(QMM_ERR_NULL, "pack_dense_tables: null pointer");
  if (G < 1 || N < 1 || K % G || group_size < 32 || K % group_size || N >= (1LL << 30) || K >= (1LL << 30)) return fail(QMM_ERR_SHAPE, "pack_dense_tables: bad shape");
  const dim3 grid(static_cast<unsigned>((N + 31) / 32), static_cast<unsigned>((K / group_size + 31) / 32));
  if (grid.y > 65535) return fail(QMM_ERR_SHAPE, "pack_dense_tables: K is too long");
  return with_types(scale_dtype, zero ? zero_dtype : QMM_U8, [&](auto s, auto z) -> int {
    using S = decltype(s);
    using Z = decltype(z);
    if (narrow && scale_dtype != QMM_F32)
      tables_kernel<S, Z, S><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const S*>(scale), static_cast<const Z*>(zero), static_cast<S*>(scales),
                                                                                  static_cast<S*>(biases), static_cast<int>(G), static_cast<int>(N), static_cast<int>(K), group_size);
    else
      tables_kernel<S, Z, float><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const S*>(scale), static_cast<const Z*>(zero), static_cast<float*>(scales),
                                                                                      static_cast<float*>(biases), static_cast<int>(G), static_cast<int>(N), static_cast<int>(K), group_size);
    count_launch();
    return check_launch("tables_kernel");
  });
}
