// The rotary embedding's rotation of a pair, in one place: the rotary kernel and both attention kernels append the same bits to a cache, whichever of them a
// step runs, and the products that are rounded by themselves are therefore not the compiler's choice.
#pragma once

namespace qmm {

__device__ __forceinline__ float2 rotate_half(float lo, float hi, float sine, float cosine) {
  return make_float2(__fmaf_rn(lo, cosine, -__fmul_rn(hi, sine)), __fmaf_rn(hi, cosine, __fmul_rn(lo, sine)));
}

}  // namespace qmm
