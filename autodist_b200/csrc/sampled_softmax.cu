// Sampled softmax with a shared set of negatives (sm_100a): the logits of the true class and of K sampled classes from the bf16 products
// that the GEMM leaves, and what their softmax's gradient means for the products and the bias.
//
//   logit[n][1 + k] = (raw[n][k] + bias[neg[k]]) - log(S P(neg[k])), -1e9 where neg[k] is the row's own class (accidental hits)
//   logit[n][0]     = (dot[n] + bias[target[n]]) - log(S P(target[n])),       P(i) = log((i + 2) / (i + 1)) / log(V + 1)
//
// The log-softmax between the two is the library's: how it adds up a row decides the last bit of every probability, and with it which way
// a gradient is rounded to bf16. Twenty recurrent steps behind it turn such an ulp into 4e-4 of the gradients' norm; with the logits
// formed operation by operation as the composite expression forms them, and its log-softmax, training repeats the composite's bits.
// Bound by bytes: logits written, read and written by the log-softmax, read once more, the products read once and their gradient written
// once. 2560 rows x 8192 classes, device time: the composite's casts, additions, comparison, mask, concatenation, log-softmax, gradients
// and sorted bias gradients 790 us; here 32 for the logits, 65 for the library's log-softmax, 30 + 30 for the gradients. (One pass of
// kernels that also added up the rows took 61 in all, and did not repeat the composite's bits.)
//
// The reference uses tf.nn.sampled_softmax_loss (examples/lm1b/language_model.py:104-121).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pdl.cuh"
#include "sampled_softmax.h"
#include "sm_count.h"

namespace adb200 {
namespace {

// (bias, log of the expected count) of every negative and every target; ids as 32 bits. An id outside the vocabulary reads nothing
// and is reported. The library divides by a number known to the host by multiplying with its reciprocal,
// rounded from 64 bits; so does inv_log_v.
__global__ void sampled_prep_kernel(const float* __restrict__ bias, const int64_t* __restrict__ neg, const int64_t* __restrict__ targets, int K,
                                    int N, long long V, float inv_log_v, float num_sampled, float2* __restrict__ corrections, int* __restrict__ ids,
                                    int* __restrict__ error) {
  pdl_sync();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= K + N) return;
  const long long id = i < K ? neg[i] : targets[i - K];
  if ((unsigned long long)id >= (unsigned long long)V) {
    *const_cast<volatile int*>(error) = 71;                    // a plain store: the word may lie in host memory
    corrections[i] = make_float2(0.f, 0.f);
    ids[i] = i < K ? -1 : -2;
    return;
  }
  const float f = (float)id;
  // from 2^20 on the quotient's distance from 1 has few digits, from 2^24 on none; smaller ids keep it, and with it their results
  const float step = f < 1048576.0f ? logf(__fdiv_rn(f + 2.0f, f + 1.0f)) : log1pf(__fdiv_rn(1.0f, f + 1.0f));
  corrections[i] = make_float2(bias[id], logf(__fmul_rn(__fmul_rn(step, inv_log_v), num_sampled)));
  ids[i] = (int)id;
}

// A thread owns four columns 256 apart, so that every access of a warp is one run of memory although rows of 1 + K floats start anywhere,
// and walks rows four at a time; the columns' corrections stay in registers.
constexpr int kCols = 4;
__global__ void __launch_bounds__(256) sampled_logits_kernel(const __nv_bfloat16* __restrict__ raw, const void* __restrict__ dot, int dot_bf16,
                                                             const float2* __restrict__ corrections, const int* __restrict__ ids, float* __restrict__ logits,
                                                             int N, int K, int rows_per_block) {
  pdl_sync();
  const int c0 = blockIdx.x * 256 * kCols + threadIdx.x;
  const int n0 = blockIdx.y * rows_per_block, n1 = min(N, n0 + rows_per_block);
  float2 a[kCols];
  int id[kCols];
#pragma unroll
  for (int j = 0; j < kCols; ++j) {
    const int c = c0 + 256 * j;
    a[j] = c < K ? corrections[c] : make_float2(0.f, 0.f);
    id[j] = c < K ? ids[c] : -1;
  }
  if (blockIdx.x == 0)
    for (int n = n0 + threadIdx.x; n < n1; n += 256) {
      const float d = dot_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(dot)[n]) : static_cast<const float*>(dot)[n];
      const float2 t = corrections[K + n];
      logits[(long long)n * (K + 1)] = (d + t.x) - t.y;
    }
  for (int n = n0; n < n1; n += 4) {
    __nv_bfloat16 v[4][kCols];
    int own[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (n + u >= n1) continue;
      own[u] = ids[K + n + u];
#pragma unroll
      for (int j = 0; j < kCols; ++j)
        if (c0 + 256 * j < K) v[u][j] = raw[(long long)(n + u) * K + c0 + 256 * j];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (n + u >= n1) continue;
#pragma unroll
      for (int j = 0; j < kCols; ++j)
        if (c0 + 256 * j < K)
          logits[(long long)(n + u) * (K + 1) + 1 + c0 + 256 * j] = id[j] == own[u] ? -1e9f : (__bfloat162float(v[u][j]) + a[j].x) - a[j].y;
    }
  }
}

// The log-softmax's gradient for a loss that is the mean of -logp[n][0]: s = -grad / N arrives at the first column of a row, so a logit gets
// (s or 0) - exp(logp) s. draw is that in bf16 (0 for accidental hits, whose logit is a constant: exp gives 0 there), part its column
// sums over a chunk of rows, ddot and dadj[K + n] the first column's. A thread owns two neighbouring columns and walks rows four at a time.
__global__ void __launch_bounds__(256) sampled_grad_kernel(const float* __restrict__ logp, const int* __restrict__ ids, const float* __restrict__ grad,
                                                           __nv_bfloat16* __restrict__ draw, void* __restrict__ ddot, int dot_bf16, float* __restrict__ part,
                                                           float* __restrict__ dadj, int N, int K, int rows_per_block) {
  pdl_sync();
  const int c = (blockIdx.x * 256 + threadIdx.x) * 2;
  const int n0 = blockIdx.y * rows_per_block, n1 = min(N, n0 + rows_per_block);
  const float s = -(*grad / (float)N);
  if (blockIdx.x == 0)
    for (int n = n0 + threadIdx.x; n < n1; n += 256) {
      const float d = s - expf(logp[(long long)n * (K + 1)]) * s;
      dadj[K + n] = d;
      if (dot_bf16) static_cast<__nv_bfloat16*>(ddot)[n] = __float2bfloat16(d);
      else static_cast<float*>(ddot)[n] = d;
    }
  if (c >= K) return;                                          // K is a multiple of 8
  const int i0 = ids[c], i1 = ids[c + 1];
  float acc0 = 0.f, acc1 = 0.f;
  for (int n = n0; n < n1; n += 4) {
    float x[4], y[4];
    int own[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (n + u >= n1) continue;
      const float* row = logp + (long long)(n + u) * (K + 1) + 1 + c;
      x[u] = row[0];
      y[u] = row[1];
      own[u] = ids[K + n + u];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (n + u >= n1) continue;
      const float p = i0 == own[u] ? 0.f : 0.f - expf(x[u]) * s, q = i1 == own[u] ? 0.f : 0.f - expf(y[u]) * s;
      acc0 += p;
      acc1 += q;
      *reinterpret_cast<__nv_bfloat162*>(draw + (long long)(n + u) * K + c) = __floats2bfloat162_rn(p, q);
    }
  }
  *reinterpret_cast<float2*>(part + (long long)blockIdx.y * K + c) = make_float2(acc0, acc1);
}

// dadj[k] = sum of the chunks' partials.
__global__ void sampled_sums_kernel(const float* __restrict__ part, float* __restrict__ dadj, int K, int chunks) {
  pdl_sync();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  float s = 0.f;
#pragma unroll 8
  for (int y = 0; y < chunks; ++y) s += part[(long long)y * K + k];
  dadj[k] = s;
}

// Bias gradients: dbias[id] += the sum of dadj over the places of id, in an order that the ids alone decide, so that a step repeats its
// bits. A thread per place compares its id with a chunk of all places, read from shared memory as broadcasts, and keeps the sum and the
// first match; behind the chunks the first place of every id adds its sums. 10752 places of a Zipf vocabulary: 30 us; the library's
// sorted accumulation 118 (a warp per place, reading the ids itself: 38; with a load behind every match 46). The work is quadratic
// in the places: 16384 67 us (sorted 148), 24576 103 (173), 32768 270 (216), so longer lists are left to the library.
constexpr int kTile = 128;
__global__ void __launch_bounds__(kTile) sampled_bias_scan_kernel(const int* __restrict__ ids, const float* __restrict__ dadj, float* __restrict__ sums,
                                                                  int* __restrict__ firsts, int n, int tiles_per_chunk) {
  pdl_sync();
  __shared__ int4 tile_id[kTile / 4];
  __shared__ float4 tile_val[kTile / 4];
  const int i = blockIdx.x * kTile + threadIdx.x;
  const int id = i < n ? ids[i] : -3;                          // no place has the id -3; what is added up for negative ones is not used
  const int j0 = blockIdx.y * tiles_per_chunk * kTile, j1 = min(n, j0 + tiles_per_chunk * kTile);
  float s0 = 0.f, s1 = 0.f;
  int first = 0x7fffffff;
  int next_id = j0 + threadIdx.x < j1 ? ids[j0 + threadIdx.x] : -4;
  float next_val = j0 + threadIdx.x < j1 ? dadj[j0 + threadIdx.x] : 0.f;
  for (int j = j0; j < j1; j += kTile) {
    __syncthreads();
    reinterpret_cast<int*>(tile_id)[threadIdx.x] = next_id;
    reinterpret_cast<float*>(tile_val)[threadIdx.x] = next_val;
    __syncthreads();
    const int at = j + kTile + threadIdx.x;
    next_id = at < j1 ? ids[at] : -4;
    next_val = at < j1 ? dadj[at] : 0.f;
    int m = -1;                                                // first match of this tile
#pragma unroll
    for (int t = kTile / 4 - 1; t >= 0; --t) {
      const int4 q = tile_id[t];
      const float4 w = tile_val[t];
      if (q.w == id) { s1 += w.w; m = 4 * t + 3; }
      if (q.z == id) { s0 += w.z; m = 4 * t + 2; }
      if (q.y == id) { s1 += w.y; m = 4 * t + 1; }
      if (q.x == id) { s0 += w.x; m = 4 * t; }
    }
    if (m >= 0 && first == 0x7fffffff) first = j + m;
  }
  if (i < n) {
    sums[(long long)blockIdx.y * n + i] = s0 + s1;
    firsts[(long long)blockIdx.y * n + i] = first;
  }
}
__global__ void sampled_bias_add_kernel(const int* __restrict__ ids, const float* __restrict__ sums, const int* __restrict__ firsts, float* __restrict__ dbias,
                                        int n, int chunks) {
  pdl_sync();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || ids[i] < 0) return;
  float s = 0.f;
  int first = 0x7fffffff;
#pragma unroll 8
  for (int c = 0; c < chunks; ++c) {
    s += sums[(long long)c * n + i];
    first = min(first, firsts[(long long)c * n + i]);
  }
  if (first == i) dbias[ids[i]] += s;
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }
// Rows per block, so that a grid of `cols` blocks across comes to about eight blocks per SM, and at least 16 rows.
int rows_per_block(int N, int cols, int blocks) {
  const int want = ceil_div(blocks, cols), rows = ceil_div(N, want < 1 ? 1 : want);
  return ceil_div(rows < 16 ? 16 : rows, 4) * 4;
}
int grad_rows(int N, int K) { return rows_per_block(N, ceil_div(K, 512), 8 * sm_count()); }

}  // namespace

void sampled_logits(const __nv_bfloat16* raw, const void* dot, bool dot_bf16, const float* bias, const int64_t* neg, const int64_t* targets, int N, int K,
                    long long V, float inv_log_v, float num_sampled, float2* corrections, int* ids, float* logits, int* error, cudaStream_t st) {
  launch_pdl(sampled_prep_kernel, dim3(ceil_div(K + N, 256)), dim3(256), 0, st, bias, neg, targets, K, N, V, inv_log_v, num_sampled, corrections, ids, error);
  const int cols = ceil_div(K, 256 * kCols), rows = rows_per_block(N, cols, 8 * sm_count());
  launch_pdl(sampled_logits_kernel, dim3(cols, ceil_div(N, rows)), dim3(256), 0, st, raw, dot, (int)dot_bf16, corrections, ids, logits, N, K, rows);
}

int sampled_grad_chunks(int N, int K) { return ceil_div(N, grad_rows(N, K)); }
void sampled_grad(const float* logp, const int* ids, const float* grad, int N, int K, float* part, __nv_bfloat16* draw, void* ddot, bool dot_bf16, float* dadj,
                  cudaStream_t st) {
  launch_pdl(sampled_grad_kernel, dim3(ceil_div(K, 512), sampled_grad_chunks(N, K)), dim3(256), 0, st, logp, ids, grad, draw, ddot, (int)dot_bf16, part, dadj, N, K,
             grad_rows(N, K));
  launch_pdl(sampled_sums_kernel, dim3(ceil_div(K, 128)), dim3(128), 0, st, part, dadj, K, sampled_grad_chunks(N, K));
}
// Chunks of places: about 16 warps per SM, at least two tiles each.
int sampled_bias_chunks(int n) {
  const int want = ceil_div(4 * sm_count(), ceil_div(n, kTile)), most = ceil_div(n, 2 * kTile);
  return ceil_div(ceil_div(n, kTile), ceil_div(ceil_div(n, kTile), want < most ? want : most));
}
void sampled_bias_grad(const int* ids, const float* dadj, float* sums, int* firsts, float* dbias, int n, cudaStream_t st) {
  if (n <= 0) return;
  const int tiles = ceil_div(n, kTile), chunks = sampled_bias_chunks(n);
  launch_pdl(sampled_bias_scan_kernel, dim3(tiles, chunks), dim3(kTile), 0, st, ids, dadj, sums, firsts, n, ceil_div(tiles, chunks));
  launch_pdl(sampled_bias_add_kernel, dim3(ceil_div(n, 128)), dim3(128), 0, st, ids, sums, firsts, dbias, n, chunks);
}

}  // namespace adb200
