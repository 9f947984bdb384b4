// Activations that more than one kernel applies (element-wise launches and GEMM epilogues).
#pragma once

namespace dgpt {

// e^x and 1 / y as one instruction of the exponential unit each (subnormal results become zero).  __expf and __fdividef take
// care of subnormal operands with several more, which in a GEMM's epilogue are what the tensor cores wait for.
__device__ __forceinline__ float exp_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}
__device__ __forceinline__ float rcp_fast(float y) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}

// z > 0:   alpha_p z^2 + z / 2
// z <= 0:  alpha_n (e^z - 1 - z) + z / 2
// alpha_p = softplus(p) and alpha_n = 1/2 + softplus(q) of the layer's two learned numbers.
__device__ __forceinline__ float xielu_value(float z, float alpha_p, float alpha_n) {
  const float curve = z > 0.f ? alpha_p * z * z : alpha_n * (expm1f(z) - z);
  return fmaf(0.5f, z, curve);
}

// The same for a result that is rounded to bf16: e^z from the exponential unit, with an absolute error near 1e-7 (below
// a bf16 step of the sum wherever that is larger than 1e-4), a third of the instructions.
__device__ __forceinline__ float xielu_fast(float z, float alpha_p, float alpha_n) {
  const bool pos = z > 0.f;
  const float sq = z * z, tail = exp_fast(z) - 1.f - z;  // both, so that no warp splits over the sign
  const float t = pos ? sq : tail;
  return fmaf(pos ? alpha_p : alpha_n, t, 0.5f * z);
}

// gate * sigmoid(gate) * up
__device__ __forceinline__ float silu_mul_value(float gate, float up) { return gate / (1.f + expf(-gate)) * up; }
// The same for a result that is rounded to bf16 (fast exponential and division, relative error near 1e-6).
__device__ __forceinline__ float silu_mul_fast(float gate, float up) { return gate * rcp_fast(1.f + exp_fast(-gate)) * up; }

}  // namespace dgpt
