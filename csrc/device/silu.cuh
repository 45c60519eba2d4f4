// Sigmoid and SiLU in fp32 without a branch, for loops whose elements are independent: eight of them interleave, with `/`
// they ran one after the other (GATE_UP's epilogue: 1100 cycles for a chunk of eight). A Newton step on the approximate
// reciprocal and a residual correction of the quotient (P. Markstein, IBM J. Res. Dev. 34, 1990).
//
// For the arguments that `..._plain` admits the result is that of the division below bit for bit; test_gpu_silu.py
// compares every one of them (silu_sweep). Callers take the division for anything else.
#pragma once

namespace mep {

__device__ __forceinline__ float approx_rcp(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return fmaf(r, fmaf(-d, r, 1.f), r);
}

__device__ __forceinline__ bool sigmoid_plain(float g) { return fabsf(g) < 60.f; }
static __device__ __noinline__ float sigmoid_any(float g) { return 1.f / (1.f + __expf(-g)); }
__device__ __forceinline__ float sigmoid(float g) {
  const float d = 1.f + __expf(-g), r = approx_rcp(d);
  return fmaf(fmaf(-d, r, 1.f), r, r);
}

__device__ __forceinline__ bool silu_plain(float g) { const float m = fabsf(g); return m < 60.f && (m >= 1e-30f || m == 0.f); }
static __device__ __noinline__ float silu_any(float g) { return g / (1.f + __expf(-g)); }
__device__ __forceinline__ float silu(float g) {
  const float d = 1.f + __expf(-g), r = approx_rcp(d), q = g * r;
  return copysignf(fmaf(fmaf(-d, q, g), r, q), g);      // the correction turns -0 into +0
}

}  // namespace mep
