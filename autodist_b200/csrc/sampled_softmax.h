// Host-side interface of the sampled-softmax kernels (see sampled_softmax.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace adb200 {

// What both passes share. K and P are multiples of 8; every buffer starts on a 16-byte boundary.
struct SampledSoftmax {
  int N, K, P;                       // rows, sampled classes, width of out and true_w
  const __nv_bfloat16* out;          // [N, P]
  const __nv_bfloat16* true_w;       // [N, P]
  float* adj;                        // [K + N] correction of every sampled class, then of every row's own class
  int* ids;                          // [K + N] their ids
  float* lse;                        // [N]
  float* true_logit;                 // [N]
};

void sampled_softmax_fwd(const SampledSoftmax& s, const __nv_bfloat16* raw, const float* bias, const int64_t* neg, const int64_t* targets, long long V,
                         float inv_log_v, float num_sampled, float* loss, int* error, cudaStream_t st);
int sampled_softmax_chunks(int N, int K);
// part: [sampled_softmax_chunks(N, K), K]; dadj: [K + N]; grad: gradient of the mean loss (device scalar)
void sampled_softmax_bwd(const SampledSoftmax& s, const __nv_bfloat16* raw, const float* grad, float* part, __nv_bfloat16* draw, __nv_bfloat16* d_out,
                         __nv_bfloat16* d_true_w, float* dadj, cudaStream_t st);
// dbias[ids[i]] += dadj[i]
void sampled_softmax_bias_grad(const int* ids, const float* dadj, float* dbias, int n, cudaStream_t st);

}  // namespace adb200
