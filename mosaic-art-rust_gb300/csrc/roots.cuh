// roots.cuh -- the adjacency weights' square root and reciprocal and the
// composite's reciprocal, correctly rounded, without the range branches of the
// general forms: in the ranges given nothing can overflow, underflow or lose bits,
// so the hardware's approximate reciprocal square root (or reciprocal) and one
// correction by fused multiply-adds of the exact residual gives the rounded
// result (the last step of Markstein's method, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 1990).
// tests/test_gpu_roots.py compares every float of those ranges on the device: with
// __frcp_rn, and the weights with __frcp_rn(__fsqrt_rn(s) + 1).
// Two chains of these interleave, where the general forms' branches run one
// after the other.
#pragma once
#include "mg_math.h"

namespace mg {

// x in [1, 1e30].
__device__ __forceinline__ float rcp_in_range(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return __fmaf_rn(y, __fmaf_rn(-x, y, 1.0f), y);
}
// Two at once in packed arithmetic, each in [2^-67, 4).
__device__ __forceinline__ float2 rcp2_in_range(float2 v) {
  float2 y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(v.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(v.y));
  return __ffma2_rn(y, __ffma2_rn(make_float2(-v.x, -v.y), y, make_float2(1.0f, 1.0f)), y);
}

// 1 / (distance + 1) of adjacency.rs:83 from a squared distance, any float: the
// correctly rounded reciprocal equals the correctly rounded 1.0 / x.  Below
// 1e-30 (zero among them) the root is off, but it then vanishes beside the 1.
__device__ __forceinline__ float weight_general(float s) { return __frcp_rn(__fadd_rn(__fsqrt_rn(s), 1.0f)); }
__device__ __forceinline__ float weight_small(float s) {  // s in [0, 1e30]
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaxf(s, 1e-30f)));
  const float g = __fmul_rn(s, y);
  return rcp_in_range(__fadd_rn(__fmaf_rn(__fmaf_rn(-g, g, s), __fmul_rn(0.5f, y), g), 1.0f));
}
__device__ __forceinline__ float weight_of_sq(float s) {
  float w = weight_small(s);
  if (!(s <= 1e30f)) w = weight_general(s);
  return w;
}
// Two at once (their chains interleave).
__device__ __forceinline__ float2 weight_of_sq2(float s, float t) {
  float2 w = make_float2(weight_small(s), weight_small(t));
  if (!(s <= 1e30f && t <= 1e30f)) w = make_float2(weight_general(s), weight_general(t));
  return w;
}

// The adjacency weight of two Lab colours.
__device__ __forceinline__ float wgt(const float4& a, const float4& b) {
  return weight_of_sq(sq_dist(a.x, a.y, a.z, b.x, b.y, b.z));
}

}  // namespace mg
