// tc_split.h -- operand splitting of the tensor-core modes: hi = round(x) and
// lo = round(x - hi) (TF32 or BF16, to nearest even), written to packed rows.
//
// The rounding is one conversion per part; on all 2^32 inputs it gives the
// value of adding half a unit of the kept mantissa, ties to even, to the bits
// (infinities stay, NaN stays NaN).  lo of an infinity or NaN is 0.
#pragma once
#include <stdint.h>

#include "tc_common.h"

namespace bgemm {

__device__ __forceinline__ float round_tf32(float x) {
  uint32_t r;
  asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
// {x0, x1} as BF16, x0 in the low half
__device__ __forceinline__ uint32_t round_bf16x2(float x0, float x1) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(x1), "f"(x0));
  return r;
}
__device__ __forceinline__ float zero_nan(float x) { return x == x ? x : 0.0f; }

// One element of a packed row.
template <int KIND, int SPLIT>
__device__ __forceinline__ void put(char* hi, char* lo, long long idx, float x) {
  if constexpr (KIND == kKindTF32) {
    const float h = round_tf32(x);
    reinterpret_cast<float*>(hi)[idx] = h;
    if constexpr (SPLIT) reinterpret_cast<float*>(lo)[idx] = round_tf32(zero_nan(x - h));
  } else {
    const uint32_t h = round_bf16x2(x, 0.0f);
    reinterpret_cast<uint16_t*>(hi)[idx] = (uint16_t)h;
    if constexpr (SPLIT)
      reinterpret_cast<uint16_t*>(lo)[idx] =
          (uint16_t)round_bf16x2(zero_nan(x - __uint_as_float(h << 16)), 0.0f);
  }
}

// Four consecutive k of one packed row, one 16-byte (TF32) or 8-byte (BF16)
// store per part; idx is a multiple of 4.
template <int KIND, int SPLIT>
__device__ __forceinline__ void put4(char* hi, char* lo, long long idx, const float (&x)[4]) {
  if constexpr (KIND == kKindTF32) {
    const float4 h = make_float4(round_tf32(x[0]), round_tf32(x[1]), round_tf32(x[2]),
                                 round_tf32(x[3]));
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(hi) + idx) = h;
    if constexpr (SPLIT)
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(lo) + idx) =
          make_float4(round_tf32(zero_nan(x[0] - h.x)), round_tf32(zero_nan(x[1] - h.y)),
                      round_tf32(zero_nan(x[2] - h.z)), round_tf32(zero_nan(x[3] - h.w)));
  } else {
    const uint2 h = make_uint2(round_bf16x2(x[0], x[1]), round_bf16x2(x[2], x[3]));
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(hi) + idx) = h;
    if constexpr (SPLIT) {
      float l[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t w = i < 2 ? h.x : h.y;
        l[i] = zero_nan(x[i] - __uint_as_float((i & 1) ? w & 0xffff0000u : w << 16));
      }
      *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(lo) + idx) =
          make_uint2(round_bf16x2(l[0], l[1]), round_bf16x2(l[2], l[3]));
    }
  }
}

}  // namespace bgemm
