// Epilogue options that the GEMM kernels share.
#pragma once
#include "ft_ptx.cuh"

namespace ft {

enum GemmFlags : int {
  GEMM_OUT_F32 = 1,     // C is fp32 (default bf16)
  GEMM_ACCUMULATE = 2,  // C += A B^T
  GEMM_BIAS = 4,        // + bias[N] (bf16)
  GEMM_BIAS_F32 = 8,    // bias is fp32
  GEMM_RELU = 16,       // activation fused in the epilogue (after bias)
  GEMM_GELU = 32,
  GEMM_SILU = 64,
  GEMM_RELU2 = 128,     // max(v, 0)^2
  GEMM_ACT_MASK = GEMM_RELU | GEMM_GELU | GEMM_SILU | GEMM_RELU2,
  GEMM_EPI_DIRECT = 1 << 16,  // internal: per-lane read-modify-write epilogue
};

__device__ __forceinline__ float apply_act(float v, int flags) {
  if (flags & GEMM_RELU) return fmaxf(v, 0.f);
  if (flags & GEMM_GELU) return 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
  if (flags & GEMM_SILU) return v / (1.f + __expf(-v));
  if (flags & GEMM_RELU2) return fmaxf(v, 0.f) * fmaxf(v, 0.f);
  return v;
}

// act(gate) * up, the activations of the SwiGLU kernel (norm_act.cu).  kind: 1 silu, 2 relu, 3 gelu (tanh form).
__device__ __forceinline__ float glu(float g, float u, int kind) {
  if (kind == 1) return g / (1.f + __expf(-g)) * u;
  if (kind == 2) return fmaxf(g, 0.f) * u;
  const float k = 0.7978845608028654f * (g + 0.044715f * g * g * g);
  return 0.5f * g * (1.f + tanhf(k)) * u;
}

}  // namespace ft
