// What the recurrence kernels share: conversions from and to the model's type, the gates' functions, a step's geometry.
#pragma once
#include "common.cuh"

namespace cvllm {
namespace {

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }
// silu_f without a branch, so that several can be under way at once (a quotient's special cases are a branch each): the
// approximate reciprocal, then one step of P. Markstein's correction q + r (z - d q) with fused multiply-adds.  Denominators above
// 2^120 are scaled, or their reciprocal would be subnormal and flushed to zero.  Where the step has no finite remainder (z or
// the denominator infinite) q itself is right.  The same bits as silu_f for every fp32 number in [-104, 104] (all were compared).
__device__ __forceinline__ float silu_fast(float z) {
  const float e = 1.0f + expf(-z), s = e > 0x1p120f ? 0x1p-32f : 1.0f, d = e * s;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = z * r, rem = fmaf(-d, q, z);
  return (rem == rem ? fmaf(rem, r, q) : q) * s;
}
__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

struct StepGeom {
  const int32_t* cu_q;        // [B + 1] or NULL
  const int32_t* seq_start;   // [B] (with cu_q)
  const int32_t* positions;   // [B] (without cu_q)
  const int32_t* slots;       // [B]
};

__device__ __forceinline__ void portion(const StepGeom& g, int b, int& t0, int& n_new, int& start) {
  if (g.cu_q) {
    t0 = g.cu_q[b];
    n_new = g.cu_q[b + 1] - t0;
    start = g.seq_start[b];
  } else {
    t0 = b;
    n_new = 1;
    start = g.positions[b];
  }
}

}  // namespace
}  // namespace cvllm
