// SwiGLU and its gradient on bf16 values, the same rounding wherever they are formed: by the element-wise kernels or
// in the epilogue of the GEMM whose product they take.
#pragma once
#include <cuda_bf16.h>

namespace ss {

// silu(g) rounded to bf16, times u (the caller rounds the product)
__device__ __forceinline__ float swiglu_value(float g, float u) {
  const float s = __fdividef(g, 1.f + __expf(-g));
  return __bfloat162float(__float2bfloat16_rn(s)) * u;
}
// gradients of silu(g) * u for the gradient d of the product
__device__ __forceinline__ void swiglu_grad(float g, float u, float d, float& dg, float& du) {
  const float sig = __fdividef(1.f, 1.f + __expf(-g));
  du = d * __fmul_rn(g, sig);
  dg = __fmul_rn(__fmul_rn(d, u), __fmul_rn(sig, fmaf(g, 1.f - sig, 1.f)));
}

}  // namespace ss
