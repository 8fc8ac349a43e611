// What the tensor-core kernels (qmm_gemm_tc.cu, qmm_f32_tc.cu) share: tcgen05 instructions, bounded waits, arithmetic on pairs. Device code only.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "qmm_ptx.cuh"

namespace qmm {
namespace tc {

using namespace ptx;

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 remote_ld128(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// `n` arrivals on a barrier of this CTA, or (cluster address) of another's. The latter releases nothing wider than the CTA either: what
// it announces are tensor-memory stores (ordered by tcgen05's own fences) and TMA writes, and a cluster-wide release costs a memory barrier.
__device__ __forceinline__ void arrive_n(uint32_t bar, uint32_t n) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0], %1; }" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ void remote_arrive_n(uint32_t bar, uint32_t n) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}
// ... that does: what this thread has read of the other CTA's or its own shared memory may be written over.
__device__ __forceinline__ void remote_arrive_release(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait for a phase of a barrier: false (with `where` recorded at abort_flag) when it does not flip within kSpinLimit clocks, or as
// soon as another waiter of the CTA has given up. CLUSTER: the other CTA of a pair arrives on it. The hint (nanoseconds) lets the
// hardware hold the thread, so that waiting warps do not poll away the issue slots of those that work.
template <bool CLUSTER = false>
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, uint32_t abort_flag, int where) {
  auto poll = [&]() -> bool {
    uint32_t done;
    if constexpr (CLUSTER)
      asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
                   : "=r"(done) : "r"(bar), "r"(parity), "r"(100000) : "memory");
    else
      asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
                   : "=r"(done) : "r"(bar), "r"(parity), "r"(100000) : "memory");
    return done != 0;
  };
  if (poll()) return true;
  const long long t0 = clock64();
  while (!poll()) {
    uint32_t gave_up;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(gave_up) : "r"(abort_flag) : "memory");
    if (gave_up) return false;
    if (clock64() - t0 > kSpinLimit) {
      asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(abort_flag), "r"(where) : "memory");
      return false;
    }
  }
  return true;
}

// The tensor-core instructions are issued by one elected lane, chosen inside the instruction sequence: the warp around it stays
// converged, so that descriptors and addresses are uniform registers (behind a branch on the lane, every operand of every MMA
// was moved into one first: 80 to 110 cycles an MMA, above the 64 that it runs for).

// Arrives on `bar` (of both CTAs of a pair: a mask of their ranks in the cluster) when the MMAs issued so far have completed.
template <bool PAIR>
__device__ __forceinline__ void tc_commit(uint32_t bar, [[maybe_unused]] uint16_t pair) {
  if constexpr (PAIR)
    asm volatile("{ .reg .pred e; elect.sync _|e, 0xffffffff;"
                 "  @e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1; }" ::"r"(bar),
                 "h"(pair) : "memory");
  else
    asm volatile("{ .reg .pred e; elect.sync _|e, 0xffffffff;"
                 "  @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0]; }" ::"r"(bar) : "memory");
}

// D[tmem_d] (+)= A[tmem_a] * B over a K block: A from tensor memory (8 columns per 16 K), B from shared memory (32 bytes per
// 16 K; the descriptor's words).
#define QMM_MMA(GROUP, COL, ADV, ACC)                                    \
  "add.u32 a, %1, " COL "; add.u32 lo, %2, " ADV "; mov.b64 b, {lo, %3};" \
  "@e tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], [a], b, %4, " ACC ";"
template <bool PAIR>
__device__ __forceinline__ void tc_mma_block(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate) {
  if constexpr (PAIR)
    asm volatile("{ .reg .pred e, p, t; .reg .b32 a, lo; .reg .b64 b; elect.sync _|e, 0xffffffff; setp.ne.b32 p, %5, 0; setp.eq.b32 t, 0, 0;"
                 QMM_MMA("2", "0", "0", "p") QMM_MMA("2", "8", "2", "t") QMM_MMA("2", "16", "4", "t") QMM_MMA("2", "24", "6", "t") "}"
                 ::"r"(tmem_d), "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile("{ .reg .pred e, p, t; .reg .b32 a, lo; .reg .b64 b; elect.sync _|e, 0xffffffff; setp.ne.b32 p, %5, 0; setp.eq.b32 t, 0, 0;"
                 QMM_MMA("1", "0", "0", "p") QMM_MMA("1", "8", "2", "t") QMM_MMA("1", "16", "4", "t") QMM_MMA("1", "24", "6", "t") "}"
                 ::"r"(tmem_d), "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory");
}

// ... over half a block.
__device__ __forceinline__ void tc_mma_half(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{ .reg .pred e, p, t; .reg .b32 a, lo; .reg .b64 b; elect.sync _|e, 0xffffffff; setp.ne.b32 p, %5, 0; setp.eq.b32 t, 0, 0;"
               QMM_MMA("1", "0", "0", "p") QMM_MMA("1", "8", "2", "t") "}"
               ::"r"(tmem_d), "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory");
}

#define QMM_ASM_R(o) "r"(r[o]), "r"(r[o + 1]), "r"(r[o + 2]), "r"(r[o + 3]), "r"(r[o + 4]), "r"(r[o + 5]), "r"(r[o + 6]), "r"(r[o + 7])
#define QMM_ASM_W(o) "=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7])

__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds8(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

// 32 lanes x 16 / 32 consecutive 32-bit columns: thread i of the warp owns lane (base + i).
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
               QMM_ASM_R(0), QMM_ASM_R(8)
               : "memory");
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : QMM_ASM_W(0) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : QMM_ASM_W(0), QMM_ASM_W(8)
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : QMM_ASM_W(0), QMM_ASM_W(8), QMM_ASM_W(16), QMM_ASM_W(24)
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Bytes of {a, b}; a selector of 8 + i is byte i's sign, eight times (which __byte_perm does not pass on).
__device__ __forceinline__ uint32_t permute(uint32_t a, uint32_t b, uint32_t selector) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(selector));
  return d;
}

// ---- pairs of 16-bit floats ---------------------------------------------------------------

template <typename XT>
struct Half2Ops;

template <>
struct Half2Ops<__nv_bfloat16> {
  static constexpr uint32_t kMagic = 0x43004300u;  // (128, 128): 7 mantissa bits hold the code
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ uint32_t sub(uint32_t a, uint32_t b) {
    __nv_bfloat162 r = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
  }
  static __device__ __forceinline__ uint32_t fma(uint32_t a, uint32_t b, uint32_t c) {
    __nv_bfloat162 r = __hfma2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b),
                               *reinterpret_cast<__nv_bfloat162*>(&c));
    return *reinterpret_cast<uint32_t*>(&r);
  }
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
  }
};

template <>
struct Half2Ops<__half> {
  static constexpr uint32_t kMagic = 0x64006400u;  // (1024, 1024)
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ uint32_t sub(uint32_t a, uint32_t b) {
    __half2 r = __hsub2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
  }
  static __device__ __forceinline__ uint32_t fma(uint32_t a, uint32_t b, uint32_t c) {
    __half2 r = __hfma2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b),
                        *reinterpret_cast<__half2*>(&c));
    return *reinterpret_cast<uint32_t*>(&r);
  }
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    __half2 r = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
  }
};

// ---- UMMA descriptors ------------------------------------------------------------------

// K-major operand in the 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart. Low word: start address, leading
// byte offset (unused); high word: stride byte offset, descriptor version (sm_100), SWIZZLE_128B.
__device__ __forceinline__ uint32_t desc_low(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }
constexpr uint32_t kDescHigh = (1024u >> 4) | (1u << 14) | (2u << 29);

// kind::f16, float32 accumulate, both operands K-major; N goes in with `<< 17` in eighths.
__host__ __device__ constexpr uint32_t instr_desc(int fmt /*0 f16, 1 bf16*/, int m) {
  return (1u << 4) | (static_cast<uint32_t>(fmt) << 7) | (static_cast<uint32_t>(fmt) << 10) | (static_cast<uint32_t>(m >> 4) << 24);
}

}  // namespace tc
}  // namespace qmm
