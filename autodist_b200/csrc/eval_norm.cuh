// Evaluation-mode batch-norm of one value, shared by the convolution's epilogue and the stand-alone pass (elementwise.cu): the
// library's order of operations, so that a fused layer gives the bits of convolution, normalisation, addition and ReLU run one by
// one over bf16 tensors.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace adb200 {

// Channel c: (mean, 1 / standard deviation, gamma, beta).
__device__ __forceinline__ float4 eval_norm_of(const float* mean, const float* var, const float* gamma, const float* beta, float eps, int c) {
  return make_float4(mean[c], rsqrtf(var[c] + eps), gamma[c], beta[c]);
}
__device__ __forceinline__ float eval_norm(float x, const float4& n) { return fmaf(n.z * (x - n.x), n.y, n.w); }
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16(x)); }

}  // namespace adb200
