// fp32 operands of tensor-core products as three bf16 parts: x = x0 + x1 + x2 exactly (3 x 8 significant bits) for every x of
// 2^-110 and more.  Below that a third part, then a second, falls under bf16's smallest number, 2^-133: the parts are off by up to
// 2^-134 then.  Infinities, NaN and numbers that round to infinity as bf16 leave NaN in their results.
#pragma once
#include "sm100_prims.cuh"

namespace saf {

constexpr int SBLK = 64 * 64 * 2;              // one part of a block: 64 rows of 64 values, 128-byte swizzled rows

// A result of n products x y may be off by more than 2^-24 of itself where it is smaller than this: the parts are off by up to
// 2^-134 for each x and y, times the other one, at most `top`, and the accumulator may have lost up to 2^-126 of each of six part
// products.  Tested on the results, this needs the largest operand only, and costs the products of 2048 rows 1 %; what the parts
// leave over of each operand would say the same and cost 12 to 22 %.
__device__ __forceinline__ float split_tiny(int n, float top) { return n * fmaxf(0x1p-99f, 0x1p-109f * top); }

// the largest magnitude of three; NaN is left out
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max_abs(float top, const float4& x) { return max3_abs(max3_abs(top, x.x, x.y), x.z, x.w); }

__device__ __forceinline__ float4 ld4_or_0(const float* p, bool ok) {
  return ok ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
// x - h, exact for h = bf16(x): the mixed-precision FMA takes either half of a packed pair without unpacking it
__device__ __forceinline__ float minus_bf16(float x, uint16_t h) {
  float r;
  asm("fma.rn.f32.bf16 %0, %1, %2, %3;" : "=f"(r) : "h"(h), "h"((uint16_t)0xbf80u), "f"(x));
  return r;
}
// two values -> their three parts, packed
__device__ __forceinline__ void split2(float x, float y, uint32_t (&p)[3]) {
  p[0] = pack_bf16(x, y);
  x = minus_bf16(x, (uint16_t)p[0]);
  y = minus_bf16(y, (uint16_t)(p[0] >> 16));
  p[1] = pack_bf16(x, y);
  x = minus_bf16(x, (uint16_t)p[1]);
  y = minus_bf16(y, (uint16_t)(p[1] >> 16));
  p[2] = pack_bf16(x, y);
}

// 16 bytes of fp32 -> 8 bytes of each part, `stride` bytes apart
__device__ __forceinline__ void split_store(uint8_t* dst, int stride, const float4& x) {
  uint32_t w0[3], w1[3];
  split2(x.x, x.y, w0);
  split2(x.z, x.w, w1);
#pragma unroll
  for (int u = 0; u < 3; ++u) *reinterpret_cast<uint2*>(dst + u * stride) = make_uint2(w0[u], w1[u]);
}

}  // namespace saf
