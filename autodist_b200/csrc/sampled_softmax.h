// Host-side interface of the sampled-softmax kernels (see sampled_softmax.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace adb200 {

// logits: [N, 1 + K] fp32; ids: [K + N] (sampled classes, then the rows' own) and corrections: [K + N] are written for the passes behind.
// dot: [N], bf16 or fp32. inv_log_v: 1 / log(V + 1).
void sampled_logits(const __nv_bfloat16* raw, const void* dot, bool dot_bf16, const float* bias, const int64_t* neg, const int64_t* targets, int N, int K,
                    long long V, float inv_log_v, float num_sampled, float2* corrections, int* ids, float* logits, int* error, cudaStream_t st);
int sampled_grad_chunks(int N, int K);
// part: [sampled_grad_chunks(N, K), K]; dadj: [K + N]; grad: gradient of the mean loss (device scalar); ddot as dot
void sampled_grad(const float* logp, const int* ids, const float* grad, int N, int K, float* part, __nv_bfloat16* draw, void* ddot, bool dot_bf16, float* dadj,
                  cudaStream_t st);
// dbias[ids[i]] += the sum of dadj over all places of that id, in a fixed order. sums, firsts: [sampled_bias_chunks(n), n]
constexpr int kSampledScanMost = 24576;
int sampled_bias_chunks(int n);
void sampled_bias_grad(const int* ids, const float* dadj, float* sums, int* firsts, float* dbias, int n, cudaStream_t st);

}  // namespace adb200
