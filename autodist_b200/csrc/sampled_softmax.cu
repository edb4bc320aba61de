// Sampled softmax with a shared set of negatives (sm_100a): cross-entropy of the true class against K sampled classes, forward
// and backward, over the bf16 products that the GEMM leaves.
//
//   logit[n][k] = raw[n][k] + bias[neg[k]] - log(S P(neg[k])), -1e9 where neg[k] is the row's own class (accidental hits)
//   true[n]     = out[n] . true_w[n] + bias[target[n]] - log(S P(target[n]))
//   loss[n]     = log(exp(true[n]) + sum_k exp(logit[n][k])) - true[n],      P(i) = log((i + 2) / (i + 1)) / log(V + 1)
//
// Bound by the bytes of raw (read once forward, read once and written once backward): the logits are never stored in fp32, the
// corrections are formed once per class and read for four rows at a time. 2560 rows x 8192 classes, device time: the library's
// chain of casts, additions, comparison, mask, concatenation, log-softmax, its gradient and the sorted bias gradients 790 us,
// these kernels 4 + 23 forward, 27 + 7 + 2 backward.
//
// The reference uses tf.nn.sampled_softmax_loss (examples/lm1b/language_model.py:104-121).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "pdl.cuh"
#include "sampled_softmax.h"
#include "tcgen05_common.cuh"

namespace adb200 {
namespace {

using tc::load8_bf16;
using tc::store8_bf16;
using tc::unpack8_bf16;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// adj = bias - log(expected count) of every negative and every target; ids as 32 bits. An id outside the vocabulary reads nothing
// and is reported.
__global__ void sampled_prep_kernel(const float* __restrict__ bias, const int64_t* __restrict__ neg, const int64_t* __restrict__ targets, int K,
                                    int N, long long V, float inv_log_v, float num_sampled, float* __restrict__ adj, int* __restrict__ ids,
                                    int* __restrict__ error) {
  pdl_sync();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= K + N) return;
  const long long id = i < K ? neg[i] : targets[i - K];
  if ((unsigned long long)id >= (unsigned long long)V) {
    atomicExch(error, 71);
    adj[i] = 0.f;
    ids[i] = i < K ? -1 : -2;
    return;
  }
  const float f = (float)id;
  adj[i] = bias[id] - logf(num_sampled * (logf((f + 2.0f) / (f + 1.0f)) * inv_log_v));
  ids[i] = (int)id;
}

constexpr int kRows = 4;           // rows per block of the forward kernel

__global__ void __launch_bounds__(256) sampled_fwd_kernel(const __nv_bfloat16* __restrict__ raw, const float* __restrict__ adj, const int* __restrict__ ids,
                                                          const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ true_w,
                                                          float* __restrict__ lse, float* __restrict__ true_logit, float* __restrict__ loss, int N,
                                                          int K, int P) {
  pdl_sync();
  __shared__ float sm[8][kRows], ss[8][kRows];
  const int r0 = blockIdx.x * kRows, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int t[kRows];
  float m[kRows], s[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    t[r] = r0 + r < N ? ids[K + r0 + r] : -2;
    m[r] = -FLT_MAX;
    s[r] = 0.f;
  }
  for (int c = threadIdx.x * 8; c < K; c += 256 * 8) {
    uint4 q[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) q[r] = r0 + r < N ? *reinterpret_cast<const uint4*>(raw + (long long)(r0 + r) * K + c) : make_uint4(0, 0, 0, 0);
    const float4 a0 = *reinterpret_cast<const float4*>(adj + c), a1 = *reinterpret_cast<const float4*>(adj + c + 4);
    const int4 i0 = *reinterpret_cast<const int4*>(ids + c), i1 = *reinterpret_cast<const int4*>(ids + c + 4);
    const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const int id[8] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w};
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      float v[8];
      unpack8_bf16(q[r], v);
      float mx = m[r];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = id[j] == t[r] ? -1e9f : v[j] + a[j];
        mx = fmaxf(mx, v[j]);
      }
      s[r] *= expf(m[r] - mx);
      m[r] = mx;
#pragma unroll
      for (int j = 0; j < 8; ++j) s[r] += expf(v[j] - mx);
    }
  }
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float mo = __shfl_xor_sync(0xffffffffu, m[r], o), so = __shfl_xor_sync(0xffffffffu, s[r], o);
      const float mx = fmaxf(m[r], mo);
      s[r] = s[r] * expf(m[r] - mx) + so * expf(mo - mx);
      m[r] = mx;
    }
    if (lane == 0) { sm[w][r] = m[r]; ss[w][r] = s[r]; }
  }
  __syncthreads();
  const int row = r0 + w;
  if (w >= kRows || row >= N) return;
  float d = 0.f;                                             // warp w finishes row w
  for (int c = lane * 8; c < P; c += 256) {
    float x[8], y[8];
    load8_bf16(out + (long long)row * P + c, x);
    load8_bf16(true_w + (long long)row * P + c, y);
#pragma unroll
    for (int j = 0; j < 8; ++j) d = fmaf(x[j], y[j], d);
  }
  const float tl = warp_sum(d) + adj[K + row];
  float mx = tl;
#pragma unroll
  for (int i = 0; i < 8; ++i) mx = fmaxf(mx, sm[i][w]);
  float sum = expf(tl - mx);
#pragma unroll
  for (int i = 0; i < 8; ++i) sum += ss[i][w] * expf(sm[i][w] - mx);
  if (lane == 0) {
    const float l = mx + logf(sum);
    lse[row] = l;
    true_logit[row] = tl;
    loss[row] = l - tl;
  }
}

// draw[n][k] = softmax * scale and its column sums over a chunk of rows: a thread owns 8 columns and walks rows, four in flight; a
// block covers 256 columns, its eight row lanes meet in shared memory. scale = (gradient of the mean loss) / N.
__global__ void __launch_bounds__(256) sampled_bwd_kernel(const __nv_bfloat16* __restrict__ raw, const float* __restrict__ adj, const int* __restrict__ ids,
                                                          const float* __restrict__ lse, const float* __restrict__ grad, __nv_bfloat16* __restrict__ draw,
                                                          float* __restrict__ part, int N, int K, int rows_per_block) {
  pdl_sync();
  __shared__ float sums[8][256 + 8];
  const int c = (blockIdx.x * 32 + (threadIdx.x & 31)) * 8, rl = threadIdx.x >> 5;
  const int n0 = blockIdx.y * rows_per_block, n1 = min(N, n0 + rows_per_block);
  const float scale = *grad / N;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (c < K) {
    const float4 a0 = *reinterpret_cast<const float4*>(adj + c), a1 = *reinterpret_cast<const float4*>(adj + c + 4);
    const int4 i0 = *reinterpret_cast<const int4*>(ids + c), i1 = *reinterpret_cast<const int4*>(ids + c + 4);
    const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const int id[8] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w};
    for (int n = n0 + rl; n < n1; n += 32) {
      uint4 q[4];
      float l[4];
      int t[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = n + 8 * u;
        if (r >= n1) continue;
        q[u] = *reinterpret_cast<const uint4*>(raw + (long long)r * K + c);
        l[u] = lse[r];
        t[u] = ids[K + r];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = n + 8 * u;
        if (r >= n1) continue;
        float v[8];
        unpack8_bf16(q[u], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = id[j] == t[u] ? 0.f : expf(v[j] + a[j] - l[u]) * scale;
          acc[j] += v[j];
        }
        store8_bf16(draw + (long long)r * K + c, v);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) sums[rl][(threadIdx.x & 31) * 8 + j] = acc[j];
  __syncthreads();
  const int col = blockIdx.x * 256 + threadIdx.x;
  if (col < K) {
    float x = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) x += sums[i][threadIdx.x];
    part[(long long)blockIdx.y * K + col] = x;
  }
}

// dadj[k] = sum of the chunks' partials; gradients through the true class, one warp per row: d = (softmax - 1) * scale,
// d_out = d true_w, d_true_w = d out, dadj[K + n] = d.
__global__ void sampled_bwd_rows_kernel(const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ true_w, const float* __restrict__ lse,
                                        const float* __restrict__ true_logit, const float* __restrict__ grad, const float* __restrict__ part,
                                        __nv_bfloat16* __restrict__ d_out, __nv_bfloat16* __restrict__ d_true_w, float* __restrict__ dadj, int N,
                                        int K, int P, int chunks) {
  pdl_sync();
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid < K) {
    float s = 0.f;
    for (int y = 0; y < chunks; ++y) s += part[(long long)y * K + tid];
    dadj[tid] = s;
  }
  const int row = (int)(tid >> 5), lane = threadIdx.x & 31;
  if (row >= N) return;
  const float d = (expf(true_logit[row] - lse[row]) - 1.0f) * (*grad / N);
  if (lane == 0) dadj[K + row] = d;
  for (int c = lane * 8; c < P; c += 256) {
    float x[8], y[8];
    load8_bf16(out + (long long)row * P + c, x);
    load8_bf16(true_w + (long long)row * P + c, y);
#pragma unroll
    for (int j = 0; j < 8; ++j) { x[j] *= d; y[j] *= d; }
    store8_bf16(d_out + (long long)row * P + c, y);
    store8_bf16(d_true_w + (long long)row * P + c, x);
  }
}

__global__ void sampled_bias_grad_kernel(const int* __restrict__ ids, const float* __restrict__ dadj, float* __restrict__ dbias, int n) {
  pdl_sync();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && ids[i] >= 0) atomicAdd(dbias + ids[i], dadj[i]);
}

}  // namespace

void sampled_softmax_fwd(const SampledSoftmax& s, const __nv_bfloat16* raw, const float* bias, const int64_t* neg, const int64_t* targets, long long V,
                         float inv_log_v, float num_sampled, float* loss, int* error, cudaStream_t st) {
  launch_pdl(sampled_prep_kernel, dim3((s.K + s.N + 255) / 256), dim3(256), 0, st, bias, neg, targets, s.K, s.N, V, inv_log_v, num_sampled, s.adj, s.ids, error);
  launch_pdl(sampled_fwd_kernel, dim3((s.N + kRows - 1) / kRows), dim3(256), 0, st, raw, s.adj, s.ids, s.out, s.true_w, s.lse, s.true_logit, loss, s.N, s.K, s.P);
}

// Chunks of rows of the backward kernel: about four blocks per SM, at least 32 rows each.
int sampled_softmax_chunks(int N, int K) {
  const int cols = (K + 255) / 256, want = (148 * 4 + cols - 1) / cols, most = (N + 31) / 32;
  return want < most ? (want < 1 ? 1 : want) : (most < 1 ? 1 : most);
}
void sampled_softmax_bwd(const SampledSoftmax& s, const __nv_bfloat16* raw, const float* grad, float* part, __nv_bfloat16* draw, __nv_bfloat16* d_out,
                         __nv_bfloat16* d_true_w, float* dadj, cudaStream_t st) {
  const int chunks = sampled_softmax_chunks(s.N, s.K), rpb = (s.N + chunks - 1) / chunks;
  launch_pdl(sampled_bwd_kernel, dim3((s.K + 255) / 256, chunks), dim3(256), 0, st, raw, s.adj, s.ids, s.lse, grad, draw, part, s.N, s.K, rpb);
  const long long threads = (long long)s.N * 32 > s.K ? (long long)s.N * 32 : s.K;
  launch_pdl(sampled_bwd_rows_kernel, dim3((int)((threads + 255) / 256)), dim3(256), 0, st, s.out, s.true_w, s.lse, s.true_logit, grad, part, d_out, d_true_w, dadj,
             s.N, s.K, s.P, chunks);
}
void sampled_softmax_bias_grad(const int* ids, const float* dadj, float* dbias, int n, cudaStream_t st) {
  if (n > 0) launch_pdl(sampled_bias_grad_kernel, dim3((n + 255) / 256), dim3(256), 0, st, ids, dadj, dbias, n);
}

}  // namespace adb200
