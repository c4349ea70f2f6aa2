// Feature map and single-token state update of the associative attention, shared by its kernels so that all forms give the
// same bits (jarvis_engine/jarvis_model.py:104-196).
#pragma once
#include "common.cuh"

namespace jb {

#if defined(__CUDACC__)

// ELU(x)+1 = max(x, 0) + exp(min(x, 0)) = (x + |x|)/2 + 2^((x - |x|) * log2(e)/2): two adds, one multiply, one
// ex2.approx (flush-to-zero form: a single MUFU, rel. error 2^-22, far below the bf16 rounding of the result) and
// one fused multiply-add, all on the FMA / MUFU pipes - no compare, no select.  For x > 0 the exponent is exactly
// 0 and the result is x + 1 rounded once; for x <= 0 the first term is exactly 0.
__device__ __forceinline__ float elu1(float x) {
  const float ax = fabsf(x);
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"((x - ax) * 0.72134752044448170368f));
  return fmaf(x + ax, 0.5f, e);
}

// One element of the single-token state update, S' = gamma S + v k', with its roundings spelled out so that all
// kernels that take a single token produce the same state bits.
__device__ __forceinline__ float decode_update(float gamma, float s, float v, float k) {
  return __fmaf_rn(gamma, s, __fmul_rn(v, k));
}

// RoPE of a pair (d, d + 32), roundings spelled out for the same reason.
__device__ __forceinline__ float rope_lo(float a, float b, float c, float s) { return __fmaf_rn(a, c, -__fmul_rn(b, s)); }
__device__ __forceinline__ float rope_hi(float a, float b, float c, float s) { return __fmaf_rn(b, c, __fmul_rn(a, s)); }

// Four columns of a state row times the query.
__device__ __forceinline__ float decode_dot4(float4 s, float4 q) { return s.x * q.x + s.y * q.y + s.z * q.z + s.w * q.w; }

#endif

}  // namespace jb
