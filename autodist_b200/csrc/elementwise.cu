// Bandwidth-bound kernels of the transformer / optimizer path, written for sm_100a (HBM3e-bound: 16-byte
// vector accesses, one pass over the data, reductions in registers + warp shuffles, statistics in fp32).
//
//   layernorm (+ residual add + dropout) forward / backward, embedding sum + layernorm, masked softmax (+dropout)
//   forward / backward, log-softmax cross-entropy forward+backward in one pass, row gather / scatter-add,
//   column sums (bias gradients), fused Adam / SGD-momentum / Adagrad updates that also emit the bf16 compute copy.
//
// In the reference all of these are TensorFlow library ops (LayerNormalization, softmax, sparse CE, ResourceApply*:
// examples/benchmark/utils/modeling/layers/transformer.py:133-164, masked_softmax.py:37-56,
// autodist/kernel/common/op_info.py:24-68).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "elementwise.h"
#include "eval_norm.cuh"
#include "pdl.cuh"
#include "sm_count.h"

namespace adb200 {
namespace {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Counter-based dropout mask: the same (seed, index) gives the same decision in forward and backward. One 64-bit
// hash decides four neighbouring elements (16 bits each), so a vector of eight costs two hashes.
__device__ __forceinline__ uint64_t mix(uint64_t seed, uint64_t idx) {
  uint64_t x = seed + idx * 0x9E3779B97F4A7C15ull;
  x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27; x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  return x;
}
// Scales (0 or 1 / keep probability) of the eight elements starting at `base` (a multiple of 8).
__device__ __forceinline__ void keep_scale8(uint64_t seed, uint64_t base, uint32_t thresh16, float inv_keep, float* out) {
  const uint64_t h0 = mix(seed, base >> 2), h1 = mix(seed, (base >> 2) + 1);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    out[j] = (((uint32_t)(h0 >> (16 * j)) & 0xFFFFu) >= thresh16) ? inv_keep : 0.0f;
    out[4 + j] = (((uint32_t)(h1 >> (16 * j)) & 0xFFFFu) >= thresh16) ? inv_keep : 0.0f;
  }
}
__device__ __forceinline__ uint64_t step_seed(uint64_t seed, const long long* step) {
  return seed + (step ? (uint64_t)(*step) * 0x100000001B3ull : 0ull);
}

__device__ __forceinline__ void load8(const bf16* p, float* v) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 f = __bfloat1622float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void unpack8(const uint4& u, float* v) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 f = __bfloat1622float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void store8(bf16* p, const float* v) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}

// ------------------------------------------------------------------------------------------------ LayerNorm
// One warp per row, NV vectors of eight columns per lane (vector k of lane l: columns 256 k + 8 l ...), H a multiple of 8, at most
// 1024. Both kernels are bound by the instructions they issue, not by memory: with a block of H / 8 threads per row every thread
// paid the reductions, divisions, addresses and barriers for eight elements, 52 instructions an element in the forward pass.
// 4096 x 1024 with dropout, a block per row -> a warp per row, inputs in L2 / in HBM: forward 9.4 -> 7.5 / 11.4 -> 11.3 us, backward
// with its column sums 15.6 -> 13.0 / 19.9 -> 14.3; 4096 x 768 without dropout: 8.2 -> 5.2 / 9.2 -> 6.1 and 13.4 -> 9.5 / 14.6 -> 9.4.
//
// Dropout decisions of a row: hash number i of the tensor (mix above) decides elements 4 i ... 4 i + 3. The hashed counter
// seed + i * kGolden walks on by additions.
constexpr uint64_t kGolden = 0x9E3779B97F4A7C15ull;
__device__ __forceinline__ uint64_t mix_counter(uint64_t x) {
  x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27; x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  return x;
}
// v[0..8) *= 0 or inv_keep; `x`: the counter of the first four. thresh_hi: the 16-bit threshold in the upper half of a word.
__device__ __forceinline__ void drop8(float* v, uint64_t x, uint32_t thresh_hi, float inv_keep) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint64_t m = mix_counter(x + (h ? kGolden : 0ull));
    const uint32_t lo = (uint32_t)m, hi = (uint32_t)(m >> 32);
    float* w = v + 4 * h;
    w[0] *= (lo << 16) >= thresh_hi ? inv_keep : 0.f;
    w[1] *= (lo & 0xffff0000u) >= thresh_hi ? inv_keep : 0.f;
    w[2] *= (hi << 16) >= thresh_hi ? inv_keep : 0.f;
    w[3] *= (hi & 0xffff0000u) >= thresh_hi ? inv_keep : 0.f;
  }
}
struct LnDrop {
  uint32_t thresh_hi;
  float inv_keep;
  __device__ __forceinline__ explicit LnDrop(float p) {
    const uint32_t t = (uint32_t)(p * 65536.0f);
    thresh_hi = t < 65536u ? t << 16 : 0u;
    inv_keep = t < 65536u ? 1.0f / (1.0f - p) : 0.f;       // a threshold past 16 bits keeps nothing
  }
};

constexpr int kLnWarps = 4;              // warps (rows) per block

// z = dropout(x) + residual is written back (it is what the backward pass needs), y = LN(z) * gamma + beta.
// EARLY: gamma and beta are requested with the row, in 16 NV registers more, instead of behind the reductions. For few rows, where one
// more latency counts and the registers do not: us, a block per row / late / early: 4 x 608 2.2 / 2.6 / 2.3,
// 302 x 816 with dropout 2.9 / 3.5 / 2.9, 512 x 128 with dropout 2.3 / 2.3 / 2.1, 1184 x 1024 3.6 / 3.7 / 3.5; beyond two blocks per SM late ones.
template <int NV, bool EARLY>
__global__ void __launch_bounds__(32 * kLnWarps) ln_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res, const float* __restrict__ gamma,
                              const float* __restrict__ beta, bf16* __restrict__ z, bf16* __restrict__ y,
                              float* __restrict__ mean, float* __restrict__ rstd, int rows, int H, float eps,
                              float p_drop, uint64_t seed, const long long* step) {
  pdl_sync();
  const int lane = threadIdx.x & 31;
  const LnDrop drop(p_drop);
  const uint64_t sd = step_seed(seed, step);
  const float inv_h = 1.0f / H;
  for (int row = blockIdx.x * kLnWarps + (threadIdx.x >> 5); row < rows; row += gridDim.x * kLnWarps) {
    const long long off = (long long)row * H + lane * 8;
    uint4 xq[NV], rq[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      xq[k] = rq[k] = make_uint4(0, 0, 0, 0);
      if (lane * 8 + 256 * k < H) {
        xq[k] = *reinterpret_cast<const uint4*>(x + off + 256 * k);
        if (res) rq[k] = *reinterpret_cast<const uint4*>(res + off + 256 * k);
      }
    }
    float4 gq[EARLY ? NV : 1][2], bq[EARLY ? NV : 1][2];
    if (EARLY) {
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (lane * 8 + 256 * k < H) {
          const float4* gp = reinterpret_cast<const float4*>(gamma + lane * 8 + 256 * k);
          const float4* bp = reinterpret_cast<const float4*>(beta + lane * 8 + 256 * k);
          gq[k][0] = gp[0]; gq[k][1] = gp[1]; bq[k][0] = bp[0]; bq[k][1] = bp[1];
        }
    }
    const uint64_t counter = sd + (uint64_t)(off >> 2) * kGolden;
    float v[NV][8];
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      float r[8];
      unpack8(xq[k], v[k]);
      unpack8(rq[k], r);
      if (p_drop > 0.f) drop8(v[k], counter + 64ull * k * kGolden, drop.thresh_hi, drop.inv_keep);
#pragma unroll
      for (int j = 0; j < 8; ++j) { v[k][j] += r[j]; s += v[k][j]; }       // columns that do not exist hold zeros
    }
    const float mu = warp_sum(s) * inv_h;
    float q = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (lane * 8 + 256 * k < H) {
#pragma unroll
        for (int j = 0; j < 8; ++j) { const float dd = v[k][j] - mu; q += dd * dd; }
      }
    const float rs = rsqrtf(warp_sum(q) * inv_h + eps);
    if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (lane * 8 + 256 * k < H) {
        if (z) store8(z + off + 256 * k, v[k]);
        const float4* gp = reinterpret_cast<const float4*>(gamma + lane * 8 + 256 * k);
        const float4* bp = reinterpret_cast<const float4*>(beta + lane * 8 + 256 * k);
        constexpr int have = EARLY ? 1 : 0;
        const float4 g0 = EARLY ? gq[k * have][0] : gp[0], g1 = EARLY ? gq[k * have][1] : gp[1];
        const float4 b0 = EARLY ? bq[k * have][0] : bp[0], b1 = EARLY ? bq[k * have][1] : bp[1];
        const float gg[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (v[k][j] - mu) * rs * gg[j] + bb[j];
        store8(y + off + 256 * k, o);
      }
  }
}

// dz = rstd * (g*dy - mean(g*dy) - xhat * mean(g*dy*xhat)); dx = dz * dropout mask (only written when p_drop > 0).
// `dz_add` (optional) is added to dz before it is stored: the gradient arriving over the residual connection.
// A warp walks rows with the next row's vectors requested before the current one is reduced; its per-column sums (dgamma, dbeta
// and, when asked, the sum of what it writes to dx - the bias gradient of the linear layer in front of the residual) stay in
// registers, are added up over the block's warps in shared memory and then into part[k][slot][H], k = 0 (dgamma), 1 (dbeta), 2
// (sum of the output), slot = block % kLnSlots. `part` must be zero on entry; the reduction kernel that follows clears what it
// reads, so the buffer is zero again afterwards.
constexpr int kLnSlots = 16;
constexpr int ln_bwd_resident(int nv) { return nv <= 2 ? 4 : (nv == 3 ? 3 : 2); }     // blocks per SM whose registers hold 24 * nv sums per thread (four bytes of 1024 columns are spilled)

template <int NV>
__global__ void __launch_bounds__(32 * kLnWarps, ln_bwd_resident(NV))
ln_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ z, const float* __restrict__ mean,
                              const float* __restrict__ rstd, const float* __restrict__ gamma, const bf16* __restrict__ dz_add,
                              bf16* __restrict__ dz, bf16* __restrict__ dx, float* __restrict__ part, int rows, int H, float p_drop,
                              uint64_t seed, const long long* step, int want_out_sum) {
  pdl_sync();
  __shared__ float red[kLnWarps][256 * NV];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const LnDrop drop(p_drop);
  const uint64_t sd = step_seed(seed, step);
  const float inv_h = 1.0f / H;
  float ag[NV][8], ab[NV][8], ax[NV][8];
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j) ag[k][j] = ab[k][j] = ax[k][j] = 0.f;
  int row = blockIdx.x * kLnWarps + wib;
  const int step_rows = gridDim.x * kLnWarps;
  uint4 dq[NV], zq[NV];
  float mu = 0.f, rs = 0.f;
  auto request = [&](int r) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      dq[k] = zq[k] = make_uint4(0, 0, 0, 0);
      if (r < rows && lane * 8 + 256 * k < H) {
        dq[k] = *reinterpret_cast<const uint4*>(dy + (long long)r * H + lane * 8 + 256 * k);
        zq[k] = *reinterpret_cast<const uint4*>(z + (long long)r * H + lane * 8 + 256 * k);
      }
    }
    if (r < rows) { mu = mean[r]; rs = rstd[r]; }
  };
  request(row);
  for (; row < rows; row += step_rows) {
    const long long off = (long long)row * H + lane * 8;
    float xh[NV][8], g[NV][8];
    float s1 = 0.f, s2 = 0.f;
    const float rs_now = rs;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      float gam[8], d[8];
      if (lane * 8 + 256 * k < H) {
        const float4* gp = reinterpret_cast<const float4*>(gamma + lane * 8 + 256 * k);
        const float4 g0 = gp[0], g1 = gp[1];
        gam[0] = g0.x; gam[1] = g0.y; gam[2] = g0.z; gam[3] = g0.w; gam[4] = g1.x; gam[5] = g1.y; gam[6] = g1.z; gam[7] = g1.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) gam[j] = 0.f;
      }
      unpack8(dq[k], d);
      unpack8(zq[k], xh[k]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        xh[k][j] = (xh[k][j] - mu) * rs;
        ag[k][j] += d[j] * xh[k][j];
        ab[k][j] += d[j];
        g[k][j] = d[j] * gam[j];
        s1 += g[k][j];
        s2 += g[k][j] * xh[k][j];
      }
    }
    request(row + step_rows);                     // consumed in the next iteration
    s1 = warp_sum(s1) * inv_h;
    s2 = warp_sum(s2) * inv_h;
    const uint64_t counter = sd + (uint64_t)(off >> 2) * kGolden;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      if (lane * 8 + 256 * k >= H) continue;
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rs_now * (g[k][j] - s1 - xh[k][j] * s2);
      if (dz_add) {
        float add[8];
        load8(dz_add + off + 256 * k, add);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += add[j];
      }
      store8(dz + off + 256 * k, o);
      if (p_drop > 0.f && dx) {
        drop8(o, counter + 64ull * k * kGolden, drop.thresh_hi, drop.inv_keep);
        store8(dx + off + 256 * k, o);
      }
      if (want_out_sum) {
#pragma unroll
        for (int j = 0; j < 8; ++j) ax[k][j] += __bfloat162float(__float2bfloat16(o[j]));     // what the next kernel reads
      }
    }
  }
  // The blocks add their sums into kLnSlots shared rows (vector reductions, a few dozen blocks per address) instead of
  // writing one row each: the follow-up kernel then reads 16 rows per output instead of hundreds.
  auto flush = [&](const float (&a)[NV][8], int which) {
    if (which > 0) __syncthreads();               // the sums before have been read
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      float4* at = reinterpret_cast<float4*>(&red[wib][256 * k]);      // halves of a vector 128 columns apart: no bank conflicts
      at[lane] = make_float4(a[k][0], a[k][1], a[k][2], a[k][3]);
      at[32 + lane] = make_float4(a[k][4], a[k][5], a[k][6], a[k][7]);
    }
    __syncthreads();
    float* out = part + ((long long)which * kLnSlots + blockIdx.x % kLnSlots) * H;
    for (int i = threadIdx.x; i < 64 * NV; i += 32 * kLnWarps) {
      const int col = 256 * (i >> 6) + (i & 31) * 8 + ((i >> 5) & 1) * 4;
      if (col >= H) continue;
      float4 t = reinterpret_cast<const float4*>(red[0])[i];
#pragma unroll
      for (int w = 1; w < kLnWarps; ++w) {
        const float4 u = reinterpret_cast<const float4*>(red[w])[i];
        t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
      }
      atomicAdd(reinterpret_cast<float4*>(out + col), t);
    }
  };
  flush(ag, 0);
  flush(ab, 1);
  if (want_out_sum) flush(ax, 2);
}

// Up to three column sums over partials laid out [k][parts][H] in one launch: blockIdx.y = k, out = outs[k]. The partials are
// cleared as they are read (the producer adds into them again next time).
__global__ void colsum3_f32_kernel(float* __restrict__ part, float* __restrict__ out0, float* __restrict__ out1,
                                   float* __restrict__ out2, int parts, int H, int accumulate) {
  pdl_sync();
  __shared__ float sm[8][33];
  float* src = part + (long long)blockIdx.y * parts * H;
  float* out = blockIdx.y == 0 ? out0 : (blockIdx.y == 1 ? out1 : out2);
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
  float a = 0.f;
  if (c < H)
    for (int r = w; r < parts; r += 8) { a += src[(long long)r * H + c]; src[(long long)r * H + c] = 0.f; }
  sm[w][threadIdx.x & 31] = a;
  __syncthreads();
  if (w == 0 && c < H) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += sm[i][threadIdx.x];
    out[c] = accumulate ? out[c] + t : t;
  }
}

// out[c] (+)= sum over `parts` rows of part[r][c]. A block covers 32 columns; its 8 warps split the partial rows.
__global__ void colsum_f32_kernel(const float* __restrict__ part, float* __restrict__ out, int parts, int H, int accumulate) {
  pdl_sync();
  __shared__ float sm[8][33];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
  float a = 0.f;
  if (c < H)
    for (int r = w; r < parts; r += 8) a += part[(long long)r * H + c];
  sm[w][threadIdx.x & 31] = a;
  __syncthreads();
  if (w == 0 && c < H) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += sm[i][threadIdx.x];
    out[c] = accumulate ? out[c] + t : t;
  }
}

// Two reductions in one launch (layernorm's dgamma and dbeta): blockIdx.y picks the pair.
__global__ void colsum2_f32_kernel(const float* __restrict__ part_a, float* __restrict__ out_a, const float* __restrict__ part_b,
                                   float* __restrict__ out_b, int parts, int H, int accumulate) {
  pdl_sync();
  __shared__ float sm[8][33];
  const float* part = blockIdx.y ? part_b : part_a;
  float* out = blockIdx.y ? out_b : out_a;
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
  float a = 0.f;
  if (c < H)
    for (int r = w; r < parts; r += 8) a += part[(long long)r * H + c];
  sm[w][threadIdx.x & 31] = a;
  __syncthreads();
  if (w == 0 && c < H) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += sm[i][threadIdx.x];
    out[c] = accumulate ? out[c] + t : t;
  }
}

// ------------------------------------------------------------------------------------------------ embeddings
// z[row] = word[ids[row]] + pos[row % S] + type[tt[row]]  (bf16 tables), then the layernorm kernel runs on z.
__global__ void embed_sum_kernel(const bf16* __restrict__ word, const bf16* __restrict__ pos, const bf16* __restrict__ type,
                                 const int64_t* __restrict__ ids, const int64_t* __restrict__ tt, bf16* __restrict__ z,
                                 int rows, int S, int H, long long V, long long types, int* __restrict__ error) {
  pdl_sync();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= rows) return;
  long long w = ids[warp], t = tt ? tt[warp] : 0;
  if ((unsigned long long)w >= (unsigned long long)V || (unsigned long long)t >= (unsigned long long)types) {
    // ids outside the tables read row 0 instead of foreign memory; the step is reported as failed
    if (lane == 0 && error != nullptr) atomicExch(error, 21);
    w = 0; t = 0;
  }
  const int s = warp % S;
  for (int vec = lane; vec < H / 8; vec += 32) {
    float a[8], b[8], c[8];
    load8(word + w * H + vec * 8, a);
    load8(pos + (long long)s * H + vec * 8, b);
    load8(type + t * H + vec * 8, c);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] += b[j] + c[j];
    store8(z + (long long)warp * H + vec * 8, a);
  }
}

// dst[idx[r]] += src[r] (fp32 destination, bf16 source rows): dense embedding gradient by vector atomics.
__global__ void scatter_add_rows_kernel(float* __restrict__ dst, const int64_t* __restrict__ idx, const bf16* __restrict__ src,
                                        int rows, int H, float scale) {
  pdl_sync();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= rows) return;
  const long long r = idx[warp];
  for (int vec = lane; vec < H / 8; vec += 32) {
    float a[8];
    load8(src + (long long)warp * H + vec * 8, a);
    float* d = dst + r * H + vec * 8;
    atomicAdd(reinterpret_cast<float4*>(d), make_float4(a[0] * scale, a[1] * scale, a[2] * scale, a[3] * scale));
    atomicAdd(reinterpret_cast<float4*>(d + 4), make_float4(a[4] * scale, a[5] * scale, a[6] * scale, a[7] * scale));
  }
}

// scatter_add_rows_kernel with fp32 source rows: one thread per four columns (vector atomics when the rows are 16-byte aligned). Replaces the
// sort-based embedding gradient of the library: 16384 rows of 192 took 16 radix-sort passes and a dozen helpers, 0.3 ms.
__global__ void scatter_add_rows_f32_kernel(float* __restrict__ dst, const int64_t* __restrict__ idx, const float* __restrict__ src,
                                            long long total, int h4, int H, int vec) {
  pdl_sync();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const long long row = t / h4;
  const int c = (int)(t % h4) * 4;
  const float* a = src + row * H + c;
  float* d = dst + idx[row] * (long long)H + c;
  if (vec) {
    atomicAdd(reinterpret_cast<float4*>(d), *reinterpret_cast<const float4*>(a));
  } else {
    for (int j = 0; j < 4 && c + j < H; ++j) atomicAdd(d + j, a[j]);
  }
}

// Lookups of (user, item) pairs in two fp32 tables of rows [mf | h columns]: gmf = product of the first mf columns (fp32), x = [user's
// h, item's h] as bf16, what the first layer of the other branch reads. The first columns are kept for the backward pass. Four columns
// per thread. An id outside its table reads zeros and is reported by a plain store (the word may lie in host memory).
__global__ void pair_lookup_kernel(const float* __restrict__ ut, const float* __restrict__ it, const int64_t* __restrict__ users, const int64_t* __restrict__ items,
                                   float* __restrict__ gmf, bf16* __restrict__ x, float* __restrict__ kept, long long total, int mf4, int h4,
                                   long long nu, long long ni, int* __restrict__ error) {
  pdl_sync();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int w4 = mf4 + h4;
  const long long r = t / w4;
  const int c = (int)(t % w4);
  const long long u = users[r], i = items[r];
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
  if ((unsigned long long)u < (unsigned long long)nu) a = reinterpret_cast<const float4*>(ut)[u * w4 + c];
  else *const_cast<volatile int*>(error) = 72;
  if ((unsigned long long)i < (unsigned long long)ni) b = reinterpret_cast<const float4*>(it)[i * w4 + c];
  else *const_cast<volatile int*>(error) = 72;
  if (c < mf4) {
    reinterpret_cast<float4*>(gmf)[r * mf4 + c] = make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w);
    if (kept != nullptr) {
      reinterpret_cast<float4*>(kept)[r * 2 * mf4 + c] = a;
      reinterpret_cast<float4*>(kept)[(r * 2 + 1) * mf4 + c] = b;
    }
    return;
  }
  const int j = c - mf4;
  auto put = [&](long long at, const float4& v) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    reinterpret_cast<uint2*>(x)[at] = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
  };
  put(r * 2 * h4 + j, a);
  put((r * 2 + 1) * h4 + j, b);
}

// Its gradient: dgmf times the other row's columns, and dx, added into the tables' fp32 gradients (vector reductions, any order).
__global__ void pair_lookup_bwd_kernel(const float* __restrict__ dgmf, long long ld, const bf16* __restrict__ dx, const float* __restrict__ kept,
                                       const int64_t* __restrict__ users, const int64_t* __restrict__ items, float* __restrict__ gu,
                                       float* __restrict__ gi, long long total, int mf4, int h4, long long nu, long long ni) {
  pdl_sync();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int w4 = mf4 + h4;
  const long long r = t / w4;
  const int c = (int)(t % w4);
  const long long u = users[r], i = items[r];
  float4 a, b;
  if (c < mf4) {
    const float4 d = *reinterpret_cast<const float4*>(dgmf + r * ld + 4 * c);
    const float4 ku = reinterpret_cast<const float4*>(kept)[r * 2 * mf4 + c], ki = reinterpret_cast<const float4*>(kept)[(r * 2 + 1) * mf4 + c];
    a = make_float4(d.x * ki.x, d.y * ki.y, d.z * ki.z, d.w * ki.w);
    b = make_float4(d.x * ku.x, d.y * ku.y, d.z * ku.z, d.w * ku.w);
  } else {
    auto get = [&](long long at) {
      const uint2 q = reinterpret_cast<const uint2*>(dx)[at];
      return make_float4(__uint_as_float(q.x << 16), __uint_as_float(q.x & 0xffff0000u), __uint_as_float(q.y << 16), __uint_as_float(q.y & 0xffff0000u));
    };
    a = get(r * 2 * h4 + c - mf4);
    b = get((r * 2 + 1) * h4 + c - mf4);
  }
  if ((unsigned long long)u < (unsigned long long)nu) atomicAdd(reinterpret_cast<float4*>(gu) + u * w4 + c, a);
  if ((unsigned long long)i < (unsigned long long)ni) atomicAdd(reinterpret_cast<float4*>(gi) + i * w4 + c, b);
}

// Binary cross-entropy with logits: part[block] = sum over the block's elements of max(x, 0) - x y + log(1 + exp(-|x|)). An infinite x gives
// what the library's (1 - y) x - min(x, 0) + log(..) gives, which cancels for finite ones.
constexpr int kBcePerBlock = 16384;
__global__ void __launch_bounds__(1024) bce_logits_kernel(const float* __restrict__ x, const float* __restrict__ y, float* __restrict__ part, long long n,
                                                          float scale) {
  pdl_sync();
  __shared__ float sm[32];
  const long long n0 = (long long)blockIdx.x * kBcePerBlock, n1 = n0 + kBcePerBlock < n ? n0 + kBcePerBlock : n;
  float s = 0.f;
#pragma unroll 4
  for (long long i = n0 + threadIdx.x; i < n1; i += 1024) {
    const float v = x[i], t = y[i];              // both computed and one taken: a branch keeps the next loads waiting (16384 logits 6 us more)
    const float plain = (fmaxf(v, 0.f) - v * t) + log1pf(expf(-fabsf(v))), far = (1.0f - t) * v - fminf(v, 0.f);
    s += isinf(v) ? far : plain;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = warp_sum(sm[threadIdx.x]);
    if (threadIdx.x == 0) part[blockIdx.x] = s * scale;
  }
}
__global__ void bce_logits_bwd_kernel(const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ grad, float* __restrict__ dx,
                                      long long n, float scale) {
  pdl_sync();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dx[i] = (1.0f / (1.0f + expf(-x[i])) - y[i]) * (*grad * scale);
}

// out[k][c] = sum over rows r = k + j*stride (j < count) of x[r][c]: position-embedding gradient (k = position).
__global__ void strided_rowsum_kernel(const bf16* __restrict__ x, float* __restrict__ out, int keys, int stride, int count, int H) {
  pdl_sync();
  const int k = blockIdx.y;
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= H || k >= keys) return;
  float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int j = 0; j < count; ++j) {
    float v[8];
    load8(x + ((long long)k + (long long)j * stride) * H + c, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] += v[i];
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) out[(long long)k * H + c + i] = a[i];
}

// part[y][k][c] = sum over row chunk y of the rows with key[row]==k of x[row][c]   (keys small: token-type gradient).
// With key == nullptr every row has key 0: plain column sums (bias gradients). A block covers 64 columns (8 vectors)
// with 32 row lanes per vector; the lanes' sums meet in shared memory.
__global__ void keyed_colsum_kernel(const bf16* __restrict__ x, const int64_t* __restrict__ key, float* __restrict__ part,
                                    int rows, int H, int keys, int rows_per_block) {
  pdl_sync();
  __shared__ float sm[32][65];
  const int vec = threadIdx.x & 7, rl = threadIdx.x >> 3;
  const int c = blockIdx.x * 64 + vec * 8;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  for (int k = 0; k < keys; ++k) {
    float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (c < H && key == nullptr) {
      for (int r = r0 + rl; r < r1; r += 128) {                // four rows in flight
        uint4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = r + 32 * u < r1 ? *reinterpret_cast<const uint4*>(x + (long long)(r + 32 * u) * H + c) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float v[8];
          unpack8(q[u], v);
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] += v[i];
        }
      }
    } else if (c < H)
      for (int r = r0 + rl; r < r1; r += 32) {
        if (key[r] != k) continue;
        float v[8];
        load8(x + (long long)r * H + c, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] += v[i];
      }
#pragma unroll
    for (int i = 0; i < 8; ++i) sm[rl][vec * 8 + i] = a[i];
    __syncthreads();
    if (threadIdx.x < 64 && blockIdx.x * 64 + threadIdx.x < H) {
      float t = 0.f;
#pragma unroll 8
      for (int i = 0; i < 32; ++i) t += sm[i][threadIdx.x];
      part[((long long)blockIdx.y * keys + k) * H + blockIdx.x * 64 + threadIdx.x] = t;
    }
    __syncthreads();
  }
}

// out[r] = src[idx[r]] (bf16 rows)
__global__ void gather_rows_kernel(const bf16* __restrict__ src, const int64_t* __restrict__ idx, bf16* __restrict__ out, int rows, int H) {
  pdl_sync();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= rows) return;
  const long long r = idx[warp];
  for (int vec = lane; vec < H / 8; vec += 32)
    *reinterpret_cast<uint4*>(out + (long long)warp * H + vec * 8) = *reinterpret_cast<const uint4*>(src + r * H + vec * 8);
}

// Row gather from an fp32 table with the bf16 cast fused (sampled-softmax / embedding lookups of master weights).
__global__ void gather_rows_f32_kernel(const float* __restrict__ src, const int64_t* __restrict__ idx, bf16* __restrict__ out, int rows, int H) {
  pdl_sync();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= rows) return;
  const long long r = idx[warp];
  for (int vec = lane; vec < H / 8; vec += 32) {
    const float4 a = *reinterpret_cast<const float4*>(src + r * H + vec * 8);
    const float4 b = *reinterpret_cast<const float4*>(src + r * H + vec * 8 + 4);
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    store8(out + (long long)warp * H + vec * 8, v);
  }
}

// dst[idx[r]] += src[r] for bf16 rows whose indices are unique (MLM positions of one sequence never repeat)
__global__ void scatter_add_rows_bf16_kernel(bf16* __restrict__ dst, const int64_t* __restrict__ idx, const bf16* __restrict__ src, int rows, int H) {
  pdl_sync();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= rows) return;
  const long long r = idx[warp];
  for (int vec = lane; vec < H / 8; vec += 32) {
    float a[8], b[8];
    load8(src + (long long)warp * H + vec * 8, a);
    load8(dst + r * H + vec * 8, b);
#pragma unroll
    for (int j = 0; j < 8; ++j) b[j] += a[j];
    store8(dst + r * H + vec * 8, b);
  }
}

// ------------------------------------------------------------------------------------------------ softmax
// Rows of length S (<= 1024, multiple of 8) of a [B, heads, S, S] tensor; one warp per row. p = softmax(scale*x + mask[b]);
// writes p (needed by the backward pass) and, when dropout is on, p_drop = dropout(p) for the P.V product.
template <int TPR> __device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = TPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int TPR> __device__ __forceinline__ float group_max(float v) {
#pragma unroll
  for (int o = TPR / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// TPR threads per row, VPT 8-element vectors per thread: S = 8 * TPR * VPT. (S = 128 -> 16 threads, two rows per warp.)
template <int TPR, int VPT>
__global__ void softmax_fwd_kernel(const bf16* __restrict__ x, const float* __restrict__ mask, bf16* __restrict__ p,
                                   bf16* __restrict__ p_drop, long long rows, int S, int rows_per_batch, float scale,
                                   float pd, uint64_t seed, const long long* step) {
  pdl_sync();
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = gt / TPR;
  const int t = (int)(gt % TPR);
  const bool live = row < rows;
  const long long rr = live ? row : rows - 1;
  const int b = (int)(rr / rows_per_batch);
  float v[VPT][8];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int col = (t + TPR * i) * 8;
    load8(x + rr * S + col, v[i]);
    float mk[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (mask) {
      const float4 m0 = *reinterpret_cast<const float4*>(mask + (long long)b * S + col);
      const float4 m1 = *reinterpret_cast<const float4*>(mask + (long long)b * S + col + 4);
      mk[0] = m0.x; mk[1] = m0.y; mk[2] = m0.z; mk[3] = m0.w; mk[4] = m1.x; mk[5] = m1.y; mk[6] = m1.z; mk[7] = m1.w;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) { v[i][j] = v[i][j] * scale + mk[j]; mx = fmaxf(mx, v[i][j]); }
  }
  mx = group_max<TPR>(mx);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) { v[i][j] = __expf(v[i][j] - mx); s += v[i][j]; }
  const float inv = 1.0f / group_sum<TPR>(s);
  if (!live) return;
  const uint32_t thresh = (uint32_t)(pd * 65536.0f);
  const float inv_keep = pd > 0.f ? 1.0f / (1.0f - pd) : 1.0f;
  const uint64_t sd = step_seed(seed, step);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const long long off = row * S + (t + TPR * i) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[i][j] *= inv;
    store8(p + off, v[i]);
    if (pd > 0.f && p_drop) {
      float ks[8];
      keep_scale8(sd, (uint64_t)off, thresh, inv_keep, ks);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] *= ks[j];
      store8(p_drop + off, v[i]);
    }
  }
}

// ds = scale * p * (dp' - sum(dp' * p)) with dp' = dp * dropout mask; written over dp.
template <int TPR, int VPT>
__global__ void softmax_bwd_kernel(bf16* __restrict__ dp, const bf16* __restrict__ p, long long rows, int S, float scale,
                                   float pd, uint64_t seed, const long long* step) {
  pdl_sync();
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = gt / TPR;
  const int t = (int)(gt % TPR);
  const bool live = row < rows;
  const long long rr = live ? row : rows - 1;
  const uint32_t thresh = (uint32_t)(pd * 65536.0f);
  const float inv_keep = pd > 0.f ? 1.0f / (1.0f - pd) : 1.0f;
  const uint64_t sd = step_seed(seed, step);
  float d[VPT][8], pr[VPT][8];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const long long off = rr * S + (t + TPR * i) * 8;
    load8(dp + off, d[i]);
    load8(p + off, pr[i]);
    if (pd > 0.f) {
      float ks[8];
      keep_scale8(sd, (uint64_t)off, thresh, inv_keep, ks);
#pragma unroll
      for (int j = 0; j < 8; ++j) d[i][j] *= ks[j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s += d[i][j] * pr[i][j];
  }
  s = group_sum<TPR>(s);
  if (!live) return;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) d[i][j] = scale * pr[i][j] * (d[i][j] - s);
    store8(dp + row * S + (t + TPR * i) * 8, d[i]);
  }
}

// ------------------------------------------------------------------------------------------------ cross-entropy
// One block per row of logits [rows, ld] (first V columns valid). loss_sum += w * (lse - x[label]); the logits are
// overwritten by d loss / d logits = w / denom * (softmax - onehot) (zero in the padding columns). denom is read
// from device memory (sum of weights, computed by weight_sum_kernel) so that the whole step stays on the device.
__global__ void weight_sum_kernel(const float* __restrict__ w, int n, float* __restrict__ out, float eps) {
  pdl_sync();
  float a = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) a += w[i];
  a = warp_sum(a);
  __shared__ float s[32];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < (blockDim.x >> 5); ++i) t += s[i];
    *out = t + eps;
  }
}

__global__ void xent_kernel(bf16* __restrict__ logits, const int64_t* __restrict__ labels, const float* __restrict__ weights,
                            const float* __restrict__ denom, float* __restrict__ loss_sum, int V, int ld, float loss_scale) {
  pdl_sync();
  const int row = blockIdx.x;
  bf16* x = logits + (long long)row * ld;
  __shared__ float red[32];
  __shared__ float bc;
  float mx = -INFINITY;
  for (int c = threadIdx.x; c < V; c += blockDim.x) mx = fmaxf(mx, __bfloat162float(x[c]));
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) { float m = red[0]; for (int i = 1; i < (blockDim.x >> 5); ++i) m = fmaxf(m, red[i]); bc = m; }
  __syncthreads();
  mx = bc;
  float s = 0.f;
  for (int c = threadIdx.x; c < V; c += blockDim.x) s += __expf(__bfloat162float(x[c]) - mx);
  s = warp_sum(s);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) { float t = 0.f; for (int i = 0; i < (blockDim.x >> 5); ++i) t += red[i]; bc = t; }
  __syncthreads();
  const float sum = bc;
  const float w = weights ? weights[row] : 1.0f;
  const float dn = *denom;
  const long long label = labels[row];
  if (threadIdx.x == 0) atomicAdd(loss_sum, loss_scale * w * (logf(sum) + mx - __bfloat162float(x[label])) / dn);
  const float g = loss_scale * w / dn;
  const float inv = 1.0f / sum;
  for (int c = threadIdx.x; c < ld; c += blockDim.x) {
    float v = 0.f;
    if (c < V) v = g * (__expf(__bfloat162float(x[c]) - mx) * inv - (c == label ? 1.0f : 0.0f));
    x[c] = __float2bfloat16(v);
  }
}

// Image with at most 8 channels (any strides) -> bf16 [N, Hp, Wp, 8]: pixels at (pad, pad), zeros in the halo and the spare channels.
template <typename T>
__global__ void pad_image8_kernel(const T* __restrict__ x, long long sn, long long sc, long long sh, long long sw, int C, int H, int W,
                                  bf16* __restrict__ xp, int Hp, int Wp, int pad, long long total) {
  pdl_sync();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int wp = (int)(i % Wp), hp = (int)((i / Wp) % Hp);
  const long long n = i / ((long long)Wp * Hp);
  const int h = hp - pad, w = wp - pad;
  float v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] = 0.f;
  if (h >= 0 && h < H && w >= 0 && w < W) {
    const T* src = x + n * sn + h * sh + w * sw;
#pragma unroll
    for (int c = 0; c < 8; ++c) if (c < C) v[c] = (float)src[c * sc];
  }
  uint32_t o[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    __nv_bfloat162 hh = __floats2bfloat162_rn(v[2 * c], v[2 * c + 1]);
    o[c] = *reinterpret_cast<uint32_t*>(&hh);
  }
  *reinterpret_cast<uint4*>(xp + i * 8) = make_uint4(o[0], o[1], o[2], o[3]);
}

__global__ void relu_bwd_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ y, uint4* __restrict__ dx, long long n8) {
  pdl_sync();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  uint4 d = dy[i];
  const uint4 yy = y[i];
  uint32_t* dw = reinterpret_cast<uint32_t*>(&d);
  const uint32_t* yw = reinterpret_cast<const uint32_t*>(&yy);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    // a bf16 is positive when it is neither zero nor has its sign bit set
    const uint32_t lo = yw[k] & 0xFFFFu, hi = yw[k] >> 16;
    const uint32_t keep_lo = (lo != 0u && lo < 0x8000u) ? 0xFFFFu : 0u;
    const uint32_t keep_hi = (hi != 0u && hi < 0x8000u) ? 0xFFFF0000u : 0u;
    dw[k] &= (keep_lo | keep_hi);
  }
  dx[i] = d;
}

__global__ void tanh_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ y, bf16* __restrict__ dx, long long n) {
  pdl_sync();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { float t = __bfloat162float(y[i]); dx[i] = __float2bfloat16(__bfloat162float(dy[i]) * (1.0f - t * t)); }
}

__global__ void gelu_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ u, bf16* __restrict__ dx, long long n) {
  pdl_sync();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float x = __bfloat162float(u[i]);
  const float k = 0.7978845608028654f;
  const float t = tanhf(k * (x + 0.044715f * x * x * x));
  const float d = 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * k * (1.0f + 3.0f * 0.044715f * x * x);
  dx[i] = __float2bfloat16(__bfloat162float(dy[i]) * d);
}

__global__ void add_bf16_kernel(const bf16* __restrict__ a, const bf16* __restrict__ b, bf16* __restrict__ out, long long n8) {
  pdl_sync();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  float x[8], y[8];
  load8(a + i * 8, x);
  load8(b + i * 8, y);
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] += y[j];
  store8(out + i * 8, x);
}

// ------------------------------------------------------------------------------------------------ optimizers
// Flat multi-tensor updates over [n] fp32 master weights; each also writes the bf16 copy the next forward reads.
// lr and the step counter live in device memory so that a captured CUDA graph follows schedules.
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                            bf16* __restrict__ p16, long long n, const float* __restrict__ lr_ptr, float b1, float b2, float eps,
                            float wd, int decoupled, const long long* __restrict__ step_ptr, float grad_scale) {
  pdl_sync();
  const float lr = *lr_ptr;
  const float t = (float)(*step_ptr);
  const float c1 = 1.0f - powf(b1, t), c2 = 1.0f - powf(b2, t);
  const float inv_c1 = 1.0f / c1, inv_c2 = 1.0f / c2;
  const long long nvec = n / 4;
  const long long stride = (long long)gridDim.x * blockDim.x;
  // two independent 16-byte groups per iteration keep eight loads in flight per thread
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nvec; q += 2 * stride) {
    float4 P[2], G[2], M[2], V[2];
    bool live[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long i = (q + u * stride) * 4;
      live[u] = (q + u * stride) < nvec;
      if (live[u]) {
        P[u] = *reinterpret_cast<const float4*>(p + i);
        G[u] = __ldcs(reinterpret_cast<const float4*>(g + i));
        M[u] = *reinterpret_cast<const float4*>(m + i);
        V[u] = *reinterpret_cast<const float4*>(v + i);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (!live[u]) continue;
      const long long i = (q + u * stride) * 4;
      float pp[4] = {P[u].x, P[u].y, P[u].z, P[u].w}, gg[4] = {G[u].x, G[u].y, G[u].z, G[u].w};
      float mm[4] = {M[u].x, M[u].y, M[u].z, M[u].w}, vv[4] = {V[u].x, V[u].y, V[u].z, V[u].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float gr = gg[j] * grad_scale;
        if (wd != 0.f) { if (decoupled) pp[j] *= 1.0f - lr * wd; else gr += wd * pp[j]; }
        mm[j] = b1 * mm[j] + (1.0f - b1) * gr;
        vv[j] = b2 * vv[j] + (1.0f - b2) * gr * gr;
        pp[j] -= lr * (mm[j] * inv_c1) / (sqrtf(vv[j] * inv_c2) + eps);
      }
      *reinterpret_cast<float4*>(p + i) = make_float4(pp[0], pp[1], pp[2], pp[3]);
      *reinterpret_cast<float4*>(m + i) = make_float4(mm[0], mm[1], mm[2], mm[3]);
      *reinterpret_cast<float4*>(v + i) = make_float4(vv[0], vv[1], vv[2], vv[3]);
      if (p16) {
        __nv_bfloat162 lo = __floats2bfloat162_rn(pp[0], pp[1]), hi = __floats2bfloat162_rn(pp[2], pp[3]);
        *reinterpret_cast<uint2*>(p16 + i) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
      }
    }
  }
  // tail (n not a multiple of 4)
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const long long i = nvec * 4 + threadIdx.x;
    float gr = g[i] * grad_scale, pp = p[i];
    if (wd != 0.f) { if (decoupled) pp *= 1.0f - lr * wd; else gr += wd * pp; }
    const float mm = b1 * m[i] + (1.0f - b1) * gr, vv = b2 * v[i] + (1.0f - b2) * gr * gr;
    pp -= lr * (mm * inv_c1) / (sqrtf(vv * inv_c2) + eps);
    p[i] = pp; m[i] = mm; v[i] = vv;
    if (p16) p16[i] = __float2bfloat16(pp);
  }
}

// One element of the updates with at most one state per weight: `p` and the state `s` in place. The roundings are spelled out, so that every
// kernel gives a weight the same bits.
struct SgdRule {
  float momentum, dampening, wd, grad_scale;
  int nesterov;
  const long long* step_ptr;
  __device__ __forceinline__ bool state() const { return momentum != 0.f; }
  __device__ __forceinline__ bool first() const { return state() && *step_ptr <= 1; }       // the state starts as the first gradient
  __device__ __forceinline__ void operator()(float& p, float g, float& s, float lr, bool first_step) const {
    float gr = fmaf(g, grad_scale, wd * p);
    if (momentum != 0.f) {
      s = first_step ? gr : fmaf(1.0f - dampening, gr, momentum * s);
      gr = nesterov ? fmaf(momentum, s, gr) : s;
    }
    p = fmaf(-lr, gr, p);
  }
};
struct AdagradRule {
  float eps, wd, grad_scale;
  __device__ __forceinline__ bool state() const { return true; }
  __device__ __forceinline__ bool first() const { return false; }
  __device__ __forceinline__ void operator()(float& p, float g, float& s, float lr, bool) const {
    const float gr = fmaf(g, grad_scale, wd * p);
    s = fmaf(gr, gr, s);
    p = p - lr * gr / (sqrtf(s) + eps);
  }
};

// HBM-bound: 22 bytes per weight (with a state). In groups (every buffer on a 16-byte boundary, 8 for the bf16 copy) a thread has two 16-byte
// groups of each buffer in flight, as in adam_kernel: 138 M weights of VGG-16 with momentum 820 us -> 502 in four launches, 0.92 of
// the copy rate. One weight per thread for other bases, and for few weights, where a thread's chain of eight roots and divisions
// counts. us, momentum and Adagrad, one per thread / in groups: 4096 1.7, 1.8 / 2.0, 3.5; 524288 2.9, 3.7 / 3.3, 4.9; 1048576 5.1, 5.8 / 3.6, 5.4;
// 4194304 17.8, 18.5 / 9.1, 15.2.
constexpr long long kFlatGroupsLeast = 1 << 20;
template <class Rule>
__device__ __forceinline__ void flat_one(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ s, bf16* __restrict__ p16, long long i,
                                         float lr, const Rule& rule, bool state, bool first) {
  float pp = p[i], ss = state && !first ? s[i] : 0.f;
  rule(pp, g[i], ss, lr, first);
  p[i] = pp;
  if (state) s[i] = ss;
  if (p16) p16[i] = __float2bfloat16(pp);
}
template <class Rule>
__global__ void flat_update_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ s, bf16* __restrict__ p16,
                                   long long n, const float* __restrict__ lr_ptr, const Rule rule) {
  pdl_sync();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) flat_one(p, g, s, p16, i, *lr_ptr, rule, rule.state(), rule.first());
}
template <class Rule>
__global__ void __launch_bounds__(256, 4) flat_update_groups_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ s, bf16* __restrict__ p16,
                                          long long n, const float* __restrict__ lr_ptr, const Rule rule) {
  pdl_sync();
  const float lr = *lr_ptr;
  const bool state = rule.state(), first = rule.first();
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const long long nvec = n / 4;
  constexpr int U = 2;
  for (long long q = tid; q < nvec; q += U * stride) {
    float4 P[U], G[U], S[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long k = q + u * stride;
      S[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < nvec) {
        P[u] = reinterpret_cast<const float4*>(p)[k];
        G[u] = __ldcs(reinterpret_cast<const float4*>(g) + k);
        if (state && !first) S[u] = reinterpret_cast<const float4*>(s)[k];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long k = q + u * stride;
      if (k >= nvec) continue;
      rule(P[u].x, G[u].x, S[u].x, lr, first);
      rule(P[u].y, G[u].y, S[u].y, lr, first);
      rule(P[u].z, G[u].z, S[u].z, lr, first);
      rule(P[u].w, G[u].w, S[u].w, lr, first);
      reinterpret_cast<float4*>(p)[k] = P[u];
      if (state) reinterpret_cast<float4*>(s)[k] = S[u];
      if (p16) {
        __nv_bfloat162 lo = __floats2bfloat162_rn(P[u].x, P[u].y), hi = __floats2bfloat162_rn(P[u].z, P[u].w);
        reinterpret_cast<uint2*>(p16)[k] = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
      }
    }
  }
  if (tid < n - nvec * 4) flat_one(p, g, s, p16, nvec * 4 + tid, lr, rule, state, first);
}

// Row-sparse updates: only the rows that received a gradient are touched (rows must be unique, i.e. a coalesced
// gradient). kind 0 = SGD, 1 = lazy Adam (moments of untouched rows do not decay), 2 = Adagrad. One warp per row.
__global__ void sparse_rows_update_kernel(float* __restrict__ p, float* __restrict__ s1, float* __restrict__ s2,
                                          bf16* __restrict__ p16, const int64_t* __restrict__ rows, const float* __restrict__ g,
                                          int n, int H, long long V, int kind, const float* __restrict__ lr_ptr, float b1, float b2,
                                          float eps, const long long* __restrict__ step_ptr, float grad_scale) {
  pdl_sync();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n) return;
  const long long r = rows[warp];
  if (r < 0 || r >= V) return;                       // out-of-range ids are ignored, never written
  const float lr = *lr_ptr;
  float inv_c1 = 1.f, inv_c2 = 1.f;
  if (kind == 1) {
    const float t = (float)(*step_ptr);
    inv_c1 = 1.0f / (1.0f - powf(b1, t));
    inv_c2 = 1.0f / (1.0f - powf(b2, t));
  }
  for (int c = lane; c < H; c += 32) {
    const long long i = r * H + c;
    const float gr = g[(long long)warp * H + c] * grad_scale;
    float np;
    if (kind == 0) {
      np = p[i] - lr * gr;
    } else if (kind == 1) {
      const float m = b1 * s1[i] + (1.0f - b1) * gr, v = b2 * s2[i] + (1.0f - b2) * gr * gr;
      s1[i] = m;
      s2[i] = v;
      np = p[i] - lr * (m * inv_c1) / (sqrtf(v * inv_c2) + eps);
    } else {
      const float a = s1[i] + gr * gr;
      s1[i] = a;
      np = p[i] - lr * gr / (sqrtf(a) + eps);
    }
    p[i] = np;
    if (p16) p16[i] = __float2bfloat16(np);
  }
}

// Owner-side update of a row-sharded table: only rows whose flag was raised by the scatter-add of this step are touched.
// Their gradient row (already the mean over replicas) is applied, written back as bf16, cleared, and the flag is lowered, so
// that update and clearing cost what the touched rows cost, not what the shard costs. kind as in sparse_rows_update_kernel.
//
// Lane l of a warp reads the flags of four neighbouring rows, the groups of a warp's lanes lie a grid apart: ids are Zipf-distributed,
// the first rows of a table are nearly all touched and have to be spread over the warps. The warp then walks its touched rows
// together, 16 bytes of every buffer per lane (`vec`: rows start on 16-byte boundaries). 793471 rows of 512, 10 k of them touched,
// Adagrad: one flag per warp and iteration with 4-byte accesses 157 us, so 21 (58 with the loads of one
// 16-byte group at a time: the stores to `g` keep the compiler from moving them together).
template <int KIND>
__global__ void flagged_rows_update_kernel(float* __restrict__ p, float* __restrict__ s1, float* __restrict__ s2, bf16* __restrict__ p16,
                                           float* __restrict__ g, uint8_t* __restrict__ flags, long long rows, int H,
                                           const float* __restrict__ lr_ptr, float b1, float b2, float eps,
                                           const long long* __restrict__ step_ptr, int vec) {
  pdl_sync();
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  const float lr = *lr_ptr;
  float inv_c1 = 1.f, inv_c2 = 1.f;
  if (KIND == 1) {
    const float t = (float)(*step_ptr);
    inv_c1 = 1.0f / (1.0f - powf(b1, t));
    inv_c2 = 1.0f / (1.0f - powf(b2, t));
  }
  auto apply = [&](float& w, float gr, float& a, float& b) {
    if (KIND == 0) {
      w = w - lr * gr;
    } else if (KIND == 1) {
      a = b1 * a + (1.0f - b1) * gr;
      b = b2 * b + (1.0f - b2) * gr * gr;
      w = w - lr * (a * inv_c1) / (sqrtf(b * inv_c2) + eps);
    } else {
      a = a + gr * gr;
      w = w - lr * gr / (sqrtf(a) + eps);
    }
  };
  const long long groups = (rows + 3) / 4;
  const bool words = (reinterpret_cast<uintptr_t>(flags) & 3) == 0;
  for (long long base = 0; base < groups; base += 32 * nwarp) {
    const long long mine = base + lane * nwarp + warp0;                // this lane's group of four rows
    uint32_t f = 0;
    if (mine < groups) {
      if (words && mine * 4 + 4 <= rows) {
        f = *reinterpret_cast<const uint32_t*>(flags + mine * 4);
        if (f != 0) *reinterpret_cast<uint32_t*>(flags + mine * 4) = 0u;
      } else {
        for (int k = 0; k < 4 && mine * 4 + k < rows; ++k) {
          f |= (uint32_t)flags[mine * 4 + k] << (8 * k);
          flags[mine * 4 + k] = 0;
        }
      }
    }
    unsigned pending = __ballot_sync(0xffffffffu, f != 0);
    while (pending != 0) {
      const int src = __ffs(pending) - 1;
      pending &= pending - 1;
      const uint32_t ff = __shfl_sync(0xffffffffu, f, src);
      const long long first = (base + src * nwarp + warp0) * 4;
      for (int k = 0; k < 4; ++k) {
        if (((ff >> (8 * k)) & 0xffu) == 0) continue;
        const long long off = (first + k) * H;
        if (vec) {
          for (int c0 = lane * 4; c0 < H; c0 += 512) {                  // four groups of every buffer in flight
            float4 G[4], P[4], A[4], B[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int c = c0 + 128 * u;
              if (c >= H) continue;
              G[u] = *reinterpret_cast<const float4*>(g + off + c);
              P[u] = *reinterpret_cast<const float4*>(p + off + c);
              A[u] = B[u] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (KIND != 0) A[u] = *reinterpret_cast<const float4*>(s1 + off + c);
              if (KIND == 1) B[u] = *reinterpret_cast<const float4*>(s2 + off + c);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int c = c0 + 128 * u;
              if (c >= H) continue;
              apply(P[u].x, G[u].x, A[u].x, B[u].x); apply(P[u].y, G[u].y, A[u].y, B[u].y);
              apply(P[u].z, G[u].z, A[u].z, B[u].z); apply(P[u].w, G[u].w, A[u].w, B[u].w);
              *reinterpret_cast<float4*>(g + off + c) = make_float4(0.f, 0.f, 0.f, 0.f);
              *reinterpret_cast<float4*>(p + off + c) = P[u];
              if (KIND != 0) *reinterpret_cast<float4*>(s1 + off + c) = A[u];
              if (KIND == 1) *reinterpret_cast<float4*>(s2 + off + c) = B[u];
              if (p16) {
                __nv_bfloat162 lo = __floats2bfloat162_rn(P[u].x, P[u].y), hi = __floats2bfloat162_rn(P[u].z, P[u].w);
                *reinterpret_cast<uint2*>(p16 + off + c) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
              }
            }
          }
        } else {
          for (int c = lane; c < H; c += 32) {
            const long long i = off + c;
            const float gr = g[i];
            g[i] = 0.f;
            float w = p[i], a = KIND != 0 ? s1[i] : 0.f, b = KIND == 1 ? s2[i] : 0.f;
            apply(w, gr, a, b);
            p[i] = w;
            if (KIND != 0) s1[i] = a;
            if (KIND == 1) s2[i] = b;
            if (p16) p16[i] = __float2bfloat16(w);
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ LSTM cell (K17)
// gates [B, 4S] in the order i, j, f, o (fp32); c = sigmoid(f + fb) * c_prev + sigmoid(i) * tanh(j); h = sigmoid(o) * tanh(c)
__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + __expf(-x)); }

__global__ void lstm_cell_fwd_kernel(const float* __restrict__ gates, const float* __restrict__ c_prev, float* __restrict__ c,
                                     bf16* __restrict__ h, int B, int S, float forget_bias) {
  pdl_sync();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)B * S) return;
  const int b = (int)(idx / S), s = (int)(idx % S);
  const float* g = gates + (long long)b * 4 * S;
  const float i = g[s], j = g[S + s], f = g[2 * S + s], o = g[3 * S + s];
  const float cn = sigmoidf_(f + forget_bias) * c_prev[idx] + sigmoidf_(i) * tanhf(j);
  c[idx] = cn;
  h[idx] = __float2bfloat16(sigmoidf_(o) * tanhf(cn));
}

__global__ void lstm_cell_bwd_kernel(const float* __restrict__ gates, const float* __restrict__ c_prev, const float* __restrict__ c,
                                     const float* __restrict__ dh, const float* __restrict__ dc_next, float* __restrict__ dgates,
                                     float* __restrict__ dc_prev, int B, int S, float forget_bias) {
  pdl_sync();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)B * S) return;
  const int b = (int)(idx / S), s = (int)(idx % S);
  const float* g = gates + (long long)b * 4 * S;
  float* dg = dgates + (long long)b * 4 * S;
  const float si = sigmoidf_(g[s]), tj = tanhf(g[S + s]), sf = sigmoidf_(g[2 * S + s] + forget_bias), so = sigmoidf_(g[3 * S + s]);
  const float tc = tanhf(c[idx]);
  const float d_h = dh[idx];
  const float dct = (dc_next ? dc_next[idx] : 0.f) + d_h * so * (1.0f - tc * tc);
  dg[s] = dct * tj * si * (1.0f - si);
  dg[S + s] = dct * si * (1.0f - tj * tj);
  dg[2 * S + s] = dct * c_prev[idx] * sf * (1.0f - sf);
  dg[3 * S + s] = d_h * tc * so * (1.0f - so);
  dc_prev[idx] = dct * sf;
}

// The cell of a whole-sequence layer: gates, dh and dgates are bf16 (what the products around it write and read), four columns per
// thread with 8- and 16-byte accesses, S a multiple of 4. dc_next may be null (the last step); it may alias dc_prev.
__device__ __forceinline__ void load4b(const bf16* p, float* v) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void store4b(bf16* p, const float* v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
}
__global__ void lstm_seq_fwd_kernel(const bf16* __restrict__ gates, const float* __restrict__ c_prev, float* __restrict__ c, bf16* __restrict__ h,
                                    int B, int S, float forget_bias) {
  pdl_sync();
  const int s4 = S / 4;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)B * s4) return;
  const long long b = t / s4;
  const int s = (int)(t % s4) * 4;
  const bf16* g = gates + b * 4 * S + s;
  const long long at = b * S + s;
  float i[4], j[4], f[4], o[4], hv[4];
  load4b(g, i); load4b(g + S, j); load4b(g + 2 * S, f); load4b(g + 3 * S, o);
  const float4 cp = *reinterpret_cast<const float4*>(c_prev + at);
  float cn[4] = {cp.x, cp.y, cp.z, cp.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    cn[e] = sigmoidf_(f[e] + forget_bias) * cn[e] + sigmoidf_(i[e]) * tanhf(j[e]);
    hv[e] = sigmoidf_(o[e]) * tanhf(cn[e]);
  }
  *reinterpret_cast<float4*>(c + at) = make_float4(cn[0], cn[1], cn[2], cn[3]);
  store4b(h + at, hv);
}
__global__ void lstm_seq_bwd_kernel(const bf16* __restrict__ gates, const float* __restrict__ c_prev, const float* __restrict__ c,
                                    const bf16* __restrict__ dh, const float* dc_next, bf16* __restrict__ dgates, float* dc_prev, int B, int S,
                                    float forget_bias) {
  pdl_sync();
  const int s4 = S / 4;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)B * s4) return;
  const long long b = t / s4;
  const int s = (int)(t % s4) * 4;
  const bf16* g = gates + b * 4 * S + s;
  bf16* dg = dgates + b * 4 * S + s;
  const long long at = b * S + s;
  float i[4], j[4], f[4], o[4], d[4], dc[4] = {0, 0, 0, 0};
  load4b(g, i); load4b(g + S, j); load4b(g + 2 * S, f); load4b(g + 3 * S, o); load4b(dh + at, d);
  const float4 cp4 = *reinterpret_cast<const float4*>(c_prev + at), c4 = *reinterpret_cast<const float4*>(c + at);
  if (dc_next != nullptr) { const float4 n4 = *reinterpret_cast<const float4*>(dc_next + at); dc[0] = n4.x; dc[1] = n4.y; dc[2] = n4.z; dc[3] = n4.w; }
  const float cp[4] = {cp4.x, cp4.y, cp4.z, cp4.w}, cc[4] = {c4.x, c4.y, c4.z, c4.w};
  float di[4], dj[4], df[4], dv[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float si = sigmoidf_(i[e]), tj = tanhf(j[e]), sf = sigmoidf_(f[e] + forget_bias), so = sigmoidf_(o[e]), tc = tanhf(cc[e]);
    const float dct = dc[e] + d[e] * so * (1.0f - tc * tc);
    di[e] = dct * tj * si * (1.0f - si);
    dj[e] = dct * si * (1.0f - tj * tj);
    df[e] = dct * cp[e] * sf * (1.0f - sf);
    dv[e] = d[e] * tc * so * (1.0f - so);
    dc[e] = dct * sf;
  }
  store4b(dg, di); store4b(dg + S, dj); store4b(dg + 2 * S, df); store4b(dg + 3 * S, dv);
  *reinterpret_cast<float4*>(dc_prev + at) = make_float4(dc[0], dc[1], dc[2], dc[3]);
}

// ------------------------------------------------------------------------------------------------ global-norm clip (K19)
// acc += weight * sum(x^2); later x *= min(1, max_norm / (sqrt(acc) + 1e-6)). The norm never visits the host.
__global__ void sumsq_kernel(const float* __restrict__ x, long long n, float* __restrict__ acc, float weight) {
  pdl_sync();
  float a = 0.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) a += x[i] * x[i];
  a = warp_sum(a);
  __shared__ float sm[32];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < (blockDim.x >> 5); ++i) t += sm[i];
    atomicAdd(acc, t * weight);
  }
}
__global__ void clip_scale_kernel(float* __restrict__ x, long long n, const float* __restrict__ acc, float max_norm) {
  pdl_sync();
  const float norm = sqrtf(*acc);
  if (norm <= max_norm) return;
  const float sc = max_norm / (norm + 1e-6f);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) x[i] *= sc;
}

// ------------------------------------------------------------------------------------------------ convolution as GEMM (K10)
// Channels-last activations x [N, H, W, C] (C a multiple of 8). im2col lays the receptive fields out as the rows of the
// GEMM operand cols [N*Ho*Wo, KH*KW*C] (tap-major, channel-minor, matching a weight reshaped to [Cout, KH, KW, C]);
// col2im is its adjoint in gather form: every input pixel sums the taps that read it, so no atomics are needed.
__global__ void im2col_kernel(const bf16* __restrict__ x, bf16* __restrict__ cols, int N, int H, int W, int C, int KH, int KW,
                              int stride, int pad, int Ho, int Wo) {
  pdl_sync();
  const int c8 = C / 8;
  const long long total = (long long)N * Ho * Wo * KH * KW * c8;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int cv = (int)(idx % c8);
  long long r = idx / c8;
  const int tap = (int)(r % (KH * KW));
  r /= (KH * KW);
  const int wo = (int)(r % Wo), ho = (int)((r / Wo) % Ho), n = (int)(r / ((long long)Wo * Ho));
  const int hi = ho * stride - pad + tap / KW, wi = wo * stride - pad + tap % KW;
  uint4 v = make_uint4(0, 0, 0, 0);
  if (hi >= 0 && hi < H && wi >= 0 && wi < W)
    v = *reinterpret_cast<const uint4*>(x + (((long long)n * H + hi) * W + wi) * C + cv * 8);
  *reinterpret_cast<uint4*>(cols + idx * 8) = v;
}

__global__ void col2im_kernel(const bf16* __restrict__ dcols, bf16* __restrict__ dx, int N, int H, int W, int C, int KH, int KW,
                              int stride, int pad, int Ho, int Wo) {
  pdl_sync();
  const int c8 = C / 8;
  const long long total = (long long)N * H * W * c8;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int cv = (int)(idx % c8);
  long long r = idx / c8;
  const int wi = (int)(r % W), hi = (int)((r / W) % H), n = (int)(r / ((long long)W * H));
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int kh = 0; kh < KH; ++kh) {
    const int hn = hi + pad - kh;
    if (hn < 0 || hn % stride) continue;
    const int ho = hn / stride;
    if (ho >= Ho) continue;
    for (int kw = 0; kw < KW; ++kw) {
      const int wn = wi + pad - kw;
      if (wn < 0 || wn % stride) continue;
      const int wo = wn / stride;
      if (wo >= Wo) continue;
      float v[8];
      load8(dcols + ((((long long)n * Ho + ho) * Wo + wo) * (KH * KW) + kh * KW + kw) * C + cv * 8, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += v[j];
    }
  }
  store8(dx + idx * 8, acc);
}

// ------------------------------------------------------------------------------------------------ batch-norm (K14), pooling (K15)
// Channels-last activations seen as a matrix [rows = N*H*W, C] (C a multiple of 8).
// Statistics: part[y][0][c] = sum x, part[y][1][c] = sum x^2 over row chunk y (then colsum_f32 over the chunks).
// Each thread keeps four independent 16-byte loads in flight.
__global__ void bn_stats_kernel(const bf16* __restrict__ x, float* __restrict__ part, int rows, int C, int rows_per_block) {
  pdl_sync();
  __shared__ float s1[32][65], s2[32][65];
  const int vec = threadIdx.x & 7, rl = threadIdx.x >> 3;
  const int c = blockIdx.x * 64 + vec * 8;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float a[8] = {0, 0, 0, 0, 0, 0, 0, 0}, b[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (c < C)
    for (int r = r0 + rl; r < r1; r += 128) {
      float v[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int rr = r + 32 * u;
        if (rr < r1) {
          load8(x + (long long)rr * C + c, v[u]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) v[u][i] = 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < 8; ++i) { a[i] += v[u][i]; b[i] += v[u][i] * v[u][i]; }
    }
#pragma unroll
  for (int i = 0; i < 8; ++i) { s1[rl][vec * 8 + i] = a[i]; s2[rl][vec * 8 + i] = b[i]; }
  __syncthreads();
  if (threadIdx.x < 64 && blockIdx.x * 64 + threadIdx.x < C) {
    float t1 = 0.f, t2 = 0.f;
    for (int i = 0; i < 32; ++i) { t1 += s1[i][threadIdx.x]; t2 += s2[i][threadIdx.x]; }
    part[((long long)blockIdx.y * 2 + 0) * C + blockIdx.x * 64 + threadIdx.x] = t1;
    part[((long long)blockIdx.y * 2 + 1) * C + blockIdx.x * 64 + threadIdx.x] = t2;
  }
}

// Bias gradient of a convolution (+ ReLU backward): dx = dy masked by y > 0 (when y is given), part[chunk][c] = sum of dx over
// the chunk's rows. Channels-last matrix [rows, C]; 64 channels per block column, four 16-byte loads in flight per thread.
__global__ void relu_bwd_colsum_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ y, bf16* __restrict__ dx, float* __restrict__ part,
                                       int rows, int C, int rows_per_block) {
  pdl_sync();
  __shared__ float s1[32][65];
  const int vec = threadIdx.x & 7, rl = threadIdx.x >> 3;
  const int c = blockIdx.x * 64 + vec * 8;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (c < C)
    for (int r = r0 + rl; r < r1; r += 128) {
      float v[4][8], m[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int rr = r + 32 * u;
        if (rr < r1) {
          load8(dy + (long long)rr * C + c, v[u]);
          if (y != nullptr) load8(y + (long long)rr * C + c, m[u]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) { v[u][i] = 0.f; m[u][i] = 1.f; }
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int rr = r + 32 * u;
        if (y != nullptr) {
#pragma unroll
          for (int i = 0; i < 8; ++i) v[u][i] = m[u][i] > 0.f ? v[u][i] : 0.f;
          if (rr < r1) store8(dx + (long long)rr * C + c, v[u]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] += v[u][i];
      }
    }
#pragma unroll
  for (int i = 0; i < 8; ++i) s1[rl][vec * 8 + i] = a[i];
  __syncthreads();
  if (threadIdx.x < 64 && blockIdx.x * 64 + threadIdx.x < C) {
    float t1 = 0.f;
    for (int i = 0; i < 32; ++i) t1 += s1[i][threadIdx.x];
    part[(long long)blockIdx.y * C + blockIdx.x * 64 + threadIdx.x] = t1;
  }
}

// Row-walking layout of the batch-norm passes: a thread keeps one group of 8 channels (its coefficients stay in registers, so a
// row costs nothing but its own 16-byte loads and stores) and walks rows, kBnUnroll of them in flight; consecutive threads
// hold consecutive channel groups, so a block reads whole rows. grid.y covers C > 2048.
constexpr int kBnThreads = 256;
constexpr int kBnUnroll = 4;

struct BnWalk {
  int c;                 // first channel of this thread
  long long row, step;   // first row, rows between two rows of this thread
  bool live;
};
__device__ __forceinline__ BnWalk bn_walk(int C, int blocks) {
  const int c8 = C / 8, tpr = c8 < kBnThreads ? c8 : kBnThreads, rpb = kBnThreads / tpr;
  const int rl = threadIdx.x / tpr, g = blockIdx.y * kBnThreads + threadIdx.x % tpr;
  return {g * 8, (long long)blockIdx.x * rpb + rl, (long long)blocks * rpb, rl < rpb && g < c8};
}
__device__ __forceinline__ void load_f8(const float* p, float* v) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) != 0) {          // parameters may start anywhere in their storage
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = p[j];
    return;
  }
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// y = relu?(x * scale + shift (+ res)) with scale / shift derived from the per-channel sums (sum x, sum x^2); the last block of each
// grid column records mean / rstd and folds the batch statistics into the running ones - one launch for the whole
// normalisation. `keep` (with relu) receives one byte per 8 channels, bit j: y_j > 0, which is all the backward passes need of y:
// they read 1/16 of the bytes.
__global__ void __launch_bounds__(kBnThreads, 3) bn_apply_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res, bf16* __restrict__ y,
                                uint8_t* __restrict__ keep, long long rows, int C, int relu, const float* __restrict__ sums,
                                const float* __restrict__ gamma, const float* __restrict__ beta, float inv_rows, float eps,
                                float* __restrict__ mean, float* __restrict__ rstd, float* __restrict__ run_mean, float* __restrict__ run_var,
                                long long* __restrict__ batches, float momentum, float unbias) {
  pdl_sync();
  const BnWalk w = bn_walk(C, gridDim.x - 1);
  if (!w.live) return;
  const int c = w.c;
  long long row = w.row;
  if (blockIdx.x == gridDim.x - 1) {
    // The statistics have a block of their own: in the block of the first rows their loads and stores came on top of its rows.
    if (blockIdx.y == 0 && threadIdx.x == 0 && batches != nullptr) *batches += 1;
    if (threadIdx.x >= (C / 8 < kBnThreads ? C / 8 : kBnThreads)) return;
    float s1[8], s2[8], rm[8], rv[8];
    load_f8(sums + c, s1); load_f8(sums + C + c, s2);
    if (run_mean != nullptr) { load_f8(run_mean + c, rm); load_f8(run_var + c, rv); }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float mu = s1[j] * inv_rows;
      const float var = fmaxf(s2[j] * inv_rows - mu * mu, 0.f);
      mean[c + j] = mu;
      rstd[c + j] = rsqrtf(var + eps);
      if (run_mean != nullptr) {
        run_mean[c + j] = (1.0f - momentum) * rm[j] + momentum * mu;
        run_var[c + j] = (1.0f - momentum) * rv[j] + momentum * var * unbias;
      }
    }
    return;
  }
  // the first rows are requested before the coefficients, so that their latency hides under them
  uint4 xq[kBnUnroll], rq[kBnUnroll];
#pragma unroll
  for (int u = 0; u < kBnUnroll; ++u) {
    const long long r = row + u * w.step;
    xq[u] = rq[u] = make_uint4(0, 0, 0, 0);
    if (r < rows) {
      xq[u] = *reinterpret_cast<const uint4*>(x + r * C + c);
      if (res != nullptr) rq[u] = *reinterpret_cast<const uint4*>(res + r * C + c);
    }
  }
  float sc[8], sh[8];
  {
    float s1[8], s2[8], ga[8], be[8];
    load_f8(sums + c, s1); load_f8(sums + C + c, s2); load_f8(gamma + c, ga); load_f8(beta + c, be);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float mu = s1[j] * inv_rows;
      const float var = fmaxf(s2[j] * inv_rows - mu * mu, 0.f);
      sc[j] = ga[j] * rsqrtf(var + eps);
      sh[j] = be[j] - mu * sc[j];
    }
  }
  while (row < rows) {
#pragma unroll
    for (int u = 0; u < kBnUnroll; ++u) {
      const long long r = row + u * w.step;
      if (r >= rows) break;
      float v[8], rv[8];
      unpack8(xq[u], v);
      unpack8(rq[u], rv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float o = fmaf(v[j], sc[j], sh[j]) + rv[j];
        v[j] = relu ? fmaxf(o, 0.f) : o;
      }
      uint4 q;
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
      *reinterpret_cast<uint4*>(y + r * C + c) = q;
      if (keep != nullptr) {
        const uint32_t wd[4] = {q.x, q.y, q.z, q.w};
        uint32_t bits = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)                       // y >= 0 here: positive means any bit below the sign
          bits |= ((wd[j] & 0x7fffu) != 0 ? 1u : 0u) << (2 * j) | ((wd[j] & 0x7fff0000u) != 0 ? 2u : 0u) << (2 * j);
        keep[(r * C + c) >> 3] = (uint8_t)bits;
      }
    }
    row += kBnUnroll * w.step;
#pragma unroll
    for (int u = 0; u < kBnUnroll; ++u) {
      const long long r = row + u * w.step;
      if (r < rows) {
        xq[u] = *reinterpret_cast<const uint4*>(x + r * C + c);
        if (res != nullptr) rq[u] = *reinterpret_cast<const uint4*>(res + r * C + c);
      }
    }
  }
}

// Evaluation mode: y = relu?(batch_norm(x) + res) from the running statistics, one pass (the library takes three kernels: the
// inverse deviation, the normalisation and the ReLU), rounding where those round. HBM-bound, in the row-walking layout.
__global__ void __launch_bounds__(kBnThreads, 2) bn_eval_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res, bf16* __restrict__ y,
                                                                long long rows, int C, int relu, const float* __restrict__ gamma,
                                                                const float* __restrict__ beta, const float* __restrict__ mean,
                                                                const float* __restrict__ var, float eps) {
  pdl_sync();
  const BnWalk w = bn_walk(C, gridDim.x);
  if (!w.live) return;
  float4 n[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) n[j] = eval_norm_of(mean, var, gamma, beta, eps, w.c + j);
  for (long long row = w.row; row < rows; row += kBnUnroll * w.step) {
    uint4 xq[kBnUnroll], rq[kBnUnroll];
#pragma unroll
    for (int u = 0; u < kBnUnroll; ++u) {
      const long long r = row + u * w.step;
      rq[u] = make_uint4(0, 0, 0, 0);
      if (r < rows) {
        xq[u] = *reinterpret_cast<const uint4*>(x + r * C + w.c);
        if (res != nullptr) rq[u] = *reinterpret_cast<const uint4*>(res + r * C + w.c);
      }
    }
#pragma unroll
    for (int u = 0; u < kBnUnroll; ++u) {
      const long long r = row + u * w.step;
      if (r >= rows) break;
      float v[8], rv[8];
      unpack8(xq[u], v);
      unpack8(rq[u], rv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = eval_norm(v[j], n[j]);
        if (res != nullptr) v[j] = round_bf16(v[j]) + rv[j];
        v[j] = relu && v[j] < 0.f ? 0.f : v[j];              // a NaN stays a NaN
      }
      store8(y + r * C + w.c, v);
    }
  }
}

// Small tensors are bound by the latencies that follow one another: 16 x 128 channels at 14 x 14 took 6.9 us (forward 4.8) with the
// slots added up by 64 threads one after the other and the running statistics in the block of the first rows, and take 5.2
// (3.6) now; 64 x 64 x 112 x 112 42.6 us (0.76 of the copy rate).
//
// Backward statistics and coefficients in one launch. Each block adds its sums over a chunk of rows into one of kBnSlots
// shared rows of partials: part[y % kBnSlots][0][c] += sum dy', part[..][1][c] += sum dy' * xhat, dy' = dy masked by the
// ReLU (the forward pass's `keep` bytes, see bn_apply_kernel). The last block of a 64-channel group to finish (a ticket counter per group) adds the slots up, clears them
// and its counter, and writes what the second pass needs:
//   dx = gamma * rstd * (dy' - dbeta / M - xhat * dgamma / M) = A * dy' + B * x + K per channel; coef = [A (C), B (C), K (C)]
// together with sums = [dbeta (C), dgamma (C)], which are also added into dbeta_acc / dgamma_acc (the parameters'
// gradient buffers) when those are given. `counters` ([C / 64]) and `part` ([kBnSlots, 2, C]) must be zero on entry and
// are zero again on exit. Four blocks per SM leave 64 registers a thread, of which 8 bytes are spilled.
constexpr int kBnSlots = 16;
constexpr int kBnCounterFloats = 256;          // ticket counters in front of the slots: one per 64 channels, C <= 16384

__global__ void __launch_bounds__(256, 4) bn_bwd_stats_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const uint8_t* __restrict__ keep,
                                    const float* __restrict__ mean, const float* __restrict__ rstd, const float* __restrict__ gamma,
                                    unsigned int* __restrict__ counters, float* __restrict__ part, float* __restrict__ sums,
                                    float* __restrict__ coef, float* __restrict__ dgamma_acc, float* __restrict__ dbeta_acc,
                                    int rows, int C, int rows_per_block, int relu, float inv_rows) {
  pdl_sync();
  __shared__ float s1[32][65], s2[32][65];
  __shared__ int s_last;
  const int vec = threadIdx.x & 7, rl = threadIdx.x >> 3;
  const int c = blockIdx.x * 64 + vec * 8;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  // a = sum dy', b = sum dy' * x; sum dy' * xhat = rstd * (b - mean * a) is formed once per block from the totals
  float a[8] = {0, 0, 0, 0, 0, 0, 0, 0}, b[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (c < C) {
    for (int r = r0 + rl; r < r1; r += 128) {
      uint4 dq[4], xq[4];
      uint32_t kq[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int rr = r + 32 * u;
        dq[u] = xq[u] = make_uint4(0, 0, 0, 0);
        kq[u] = 0xffu;
        if (rr < r1) {
          dq[u] = *reinterpret_cast<const uint4*>(dy + (long long)rr * C + c);
          xq[u] = *reinterpret_cast<const uint4*>(x + (long long)rr * C + c);
          if (relu) kq[u] = keep[((long long)rr * C + c) >> 3];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float d[8], xv[8];
        unpack8(dq[u], d);
        unpack8(xq[u], xv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float g = (kq[u] >> i) & 1u ? d[i] : 0.f;
          a[i] += g;
          b[i] = fmaf(g, xv[i], b[i]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) { s1[rl][vec * 8 + i] = a[i]; s2[rl][vec * 8 + i] = b[i]; }
  __syncthreads();
  const int cc = blockIdx.x * 64 + threadIdx.x;              // the channel thread < 64 owns from here on
  if (threadIdx.x < 64 && cc < C) {
    float t1 = 0.f, t2 = 0.f;
    for (int i = 0; i < 32; ++i) { t1 += s1[i][threadIdx.x]; t2 += s2[i][threadIdx.x]; }
    t2 = rstd[cc] * (t2 - mean[cc] * t1);
    atomicAdd(&part[((long long)(blockIdx.y % kBnSlots) * 2 + 0) * C + cc], t1);
    atomicAdd(&part[((long long)(blockIdx.y % kBnSlots) * 2 + 1) * C + cc], t2);
    __threadfence();                                         // the sums are visible before the ticket is taken
  }
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&counters[blockIdx.x], 1u) == gridDim.y - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // All loads of a thread are requested before its first store: behind the stores that clear the slots they ran one after the other
  // (the compiler cannot tell them apart), 16 latencies for every call.
  const int slots = gridDim.y < kBnSlots ? gridDim.y : kBnSlots;
  const int ch = threadIdx.x & 63, grp = threadIdx.x >> 6, cl = blockIdx.x * 64 + ch;
  const bool mine = threadIdx.x < 64 && cl < C;
  float v0[kBnSlots / 4], v1[kBnSlots / 4];
  float rsd = 0.f, ga = 0.f, mu = 0.f, old_b = 0.f, old_g = 0.f;
#pragma unroll
  for (int u = 0; u < kBnSlots / 4; ++u) {
    const int r = grp + 4 * u;
    v0[u] = v1[u] = 0.f;
    if (cl < C && r < slots) {                               // written by atomics in L2: read there, not through L1
      v0[u] = __ldcg(&part[((long long)r * 2 + 0) * C + cl]);
      v1[u] = __ldcg(&part[((long long)r * 2 + 1) * C + cl]);
    }
  }
  if (mine) {
    rsd = rstd[cl]; ga = gamma[cl]; mu = mean[cl];
    if (dbeta_acc != nullptr) old_b = dbeta_acc[cl];
    if (dgamma_acc != nullptr) old_g = dgamma_acc[cl];
  }
  float t0 = 0.f, t1 = 0.f;
#pragma unroll
  for (int u = 0; u < kBnSlots / 4; ++u) {
    const int r = grp + 4 * u;
    t0 += v0[u];
    t1 += v1[u];
    if (cl < C && r < slots) {
      part[((long long)r * 2 + 0) * C + cl] = 0.f;
      part[((long long)r * 2 + 1) * C + cl] = 0.f;
    }
  }
  s1[grp][ch] = t0;
  s2[grp][ch] = t1;
  __syncthreads();
  if (mine) {
    const float s0 = (s1[0][ch] + s1[1][ch]) + (s1[2][ch] + s1[3][ch]), sx = (s2[0][ch] + s2[1][ch]) + (s2[2][ch] + s2[3][ch]);
    sums[cl] = s0;
    sums[C + cl] = sx;
    if (dbeta_acc != nullptr) dbeta_acc[cl] = old_b + s0;
    if (dgamma_acc != nullptr) dgamma_acc[cl] = old_g + sx;
    const float gr = ga * rsd;
    const float k0 = s0 * inv_rows, k1 = sx * inv_rows;
    const float bx = -gr * rsd * k1;
    coef[cl] = gr;
    coef[C + cl] = bx;
    coef[2 * C + cl] = -bx * mu - gr * k0;
  }
  if (threadIdx.x == 0) counters[blockIdx.x] = 0u;
}

// ADD: another gradient of x, read from rows `add_ld` apart, is added. Two blocks per SM: 24 coefficients and four rows of two or
// three tensors per thread take 104 to 121 registers; at three blocks per SM the compiler spilled 224 bytes.
template <bool ADD>
__global__ void __launch_bounds__(kBnThreads, 2) bn_bwd_apply_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                                    const uint8_t* __restrict__ keep, const float* __restrict__ coef, const bf16* __restrict__ add,
                                    long long add_ld, bf16* __restrict__ dx, bf16* __restrict__ dres, long long rows, int C, int relu) {
  constexpr int U = kBnUnroll;
  pdl_sync();
  const BnWalk w = bn_walk(C, gridDim.x);
  if (!w.live) return;
  const int c = w.c;
  float ca[8], cb[8], ck[8];
  load_f8(coef + c, ca); load_f8(coef + C + c, cb); load_f8(coef + 2 * C + c, ck);
  for (long long row = w.row; row < rows; row += U * w.step) {
    uint4 dq[U], xq[U], aq[ADD ? U : 1];
    uint32_t kq[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long r = row + u * w.step;
      kq[u] = 0xffu;
      if (r < rows) {
        dq[u] = *reinterpret_cast<const uint4*>(dy + r * C + c);
        xq[u] = *reinterpret_cast<const uint4*>(x + r * C + c);
        if (relu) kq[u] = keep[(r * C + c) >> 3];
        if (ADD) aq[u] = *reinterpret_cast<const uint4*>(add + r * add_ld + c);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long r = row + u * w.step;
      if (r >= rows) break;
      float d[8], xv[8], gm[8];
      unpack8(dq[u], d);
      unpack8(xq[u], xv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float g = (kq[u] >> j) & 1u ? d[j] : 0.f;
        gm[j] = g;
        d[j] = fmaf(ca[j], g, fmaf(cb[j], xv[j], ck[j]));
      }
      if (ADD) {                                            // the gradient x received from its other consumer
        unpack8(aq[u], xv);
#pragma unroll
        for (int j = 0; j < 8; ++j) d[j] += xv[j];
      }
      store8(dx + r * C + c, d);
      if (dres != nullptr) store8(dres + r * C + c, gm);    // gradient of the residual branch: dy masked by the ReLU
    }
  }
}

// Max pooling over [N, H, W, C] windows (k x k, stride, pad). The forward pass records, per output element, which
// window position held the first maximum (kh * k + kw, 255 = empty window); the backward pass routes the gradient
// with that code, so ties (common after a ReLU) go to exactly one input as in the library.
//
// A thread per group of 8 channels of a pixel. Its place is divided out in 32 bits where the count fits: 64-bit divisions by runtime
// values used to cost more than the loads. KT / ST: window and stride as compile-time constants for the common poolings (3 x 3 and
// 2 x 2, stride 2), whose window is then requested at once; 0 = from the arguments. 64 x 112 x 112 x 64, 3 x 3, cold
// caches: forward 61 -> 41 us, backward 102 -> 41; the five 2 x 2 layers of VGG-16, 32 images: 174 -> 118 and
// 260 -> 123 (0.8 of the copy rate in the largest).
struct PoolAt { int n, h, w, cv; bool live; };        // image, pixel row, pixel column, group of 8 channels
template <typename U>
__device__ __forceinline__ PoolAt pool_split(U t, int rows, int cols, int c8) {
  const U p = t / (U)c8, q = p / (U)cols, n = q / (U)rows;
  return {(int)n, (int)(q - n * rows), (int)(p - q * cols), (int)(t - p * c8), true};
}
__device__ __forceinline__ PoolAt pool_at(int images, int rows, int cols, int c8) {
  const unsigned long long total = (unsigned long long)images * rows * cols * c8, t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return {0, 0, 0, 0, false};
  return total <= 0xffffffffull ? pool_split<unsigned>((unsigned)t, rows, cols, c8) : pool_split<unsigned long long>(t, rows, cols, c8);
}

// All ones in the halves where a > b as bf16 (false for NaN).
__device__ __forceinline__ uint32_t gt2_mask(uint32_t a, uint32_t b) {
  return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
}

// Maxima and positions are kept as pairs of 16-bit halves: a comparison and two selections by mask for two channels of a tap, where
// fp32 took five instructions per channel (3 x 3 at the size above: 55 -> 41 us). A window's first tap is taken as it is, whatever its value.
template <int KT, int ST>
__global__ void maxpool_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, uint8_t* __restrict__ code, int N, int H, int W,
                                   int C, int k_arg, int stride_arg, int pad, int Ho, int Wo) {
  pdl_sync();
  const int k = KT > 0 ? KT : k_arg, stride = ST > 0 ? ST : stride_arg;
  const int c8 = C / 8;
  const PoolAt o = pool_at(N, Ho, Wo, c8);
  if (!o.live) return;
  uint32_t m[4] = {0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u}, pos[4] = {0x00ff00ffu, 0x00ff00ffu, 0x00ff00ffu, 0x00ff00ffu};
  bool first = true;
  auto take = [&](const uint4& q, int kh, int kw) {
    const uint32_t t = (uint32_t)(kh * k + kw) * 0x10001u, v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t more = first ? 0xffffffffu : gt2_mask(v[j], m[j]);
      m[j] = (v[j] & more) | (m[j] & ~more);
      pos[j] = (t & more) | (pos[j] & ~more);
    }
    first = false;
  };
  const int h0 = o.h * stride - pad, w0 = o.w * stride - pad;
  auto inside = [&](int kh, int kw) { return h0 + kh >= 0 && h0 + kh < H && w0 + kw >= 0 && w0 + kw < W; };
  auto at = [&](int kh, int kw) { return *reinterpret_cast<const uint4*>(x + (((long long)o.n * H + h0 + kh) * W + w0 + kw) * C + o.cv * 8); };
  if constexpr (KT > 0) {
    uint4 q[KT * KT];
#pragma unroll
    for (int i = 0; i < KT * KT; ++i)
      if (inside(i / KT, i % KT)) q[i] = at(i / KT, i % KT);
#pragma unroll
    for (int i = 0; i < KT * KT; ++i)
      if (inside(i / KT, i % KT)) take(q[i], i / KT, i % KT);
  } else {
    for (int kh = 0; kh < k; ++kh)
      for (int kw = 0; kw < k; ++kw)
        if (inside(kh, kw)) take(at(kh, kw), kh, kw);
  }
  const long long out = (((long long)o.n * Ho + o.h) * Wo + o.w) * C + o.cv * 8;
  *reinterpret_cast<uint4*>(y + out) = make_uint4(m[0], m[1], m[2], m[3]);
  *reinterpret_cast<uint2*>(code + out) = make_uint2(__byte_perm(pos[0], pos[1], 0x6420), __byte_perm(pos[2], pos[3], 0x6420));
}

// acc += dv where the window's code names tap t.
__device__ __forceinline__ void pool_route(float* acc, const uint4& dv, const uint2& code, uint32_t t) {
  float d[8];
  unpack8(dv, d);
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if ((((j < 4 ? code.x : code.y) >> (8 * (j & 3))) & 0xffu) == t) acc[j] += d[j];
}

// Any window: a thread per input pixel, which looks at every window that covers it.
__global__ void maxpool_bwd_kernel(const uint8_t* __restrict__ code, const bf16* __restrict__ dy, bf16* __restrict__ dx, int N, int H,
                                   int W, int C, int k, int stride, int pad, int Ho, int Wo) {
  pdl_sync();
  const int c8 = C / 8;
  const PoolAt i = pool_at(N, H, W, c8);
  if (!i.live) return;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int kh = 0; kh < k; ++kh) {
    const int hn = i.h + pad - kh;
    if (hn < 0 || hn % stride) continue;
    const int ho = hn / stride;
    if (ho >= Ho) continue;
    for (int kw = 0; kw < k; ++kw) {
      const int wn = i.w + pad - kw;
      if (wn < 0 || wn % stride) continue;
      const int wo = wn / stride;
      if (wo >= Wo) continue;
      const long long o = ((((long long)i.n * Ho + ho) * Wo + wo) * C) + i.cv * 8;
      pool_route(acc, *reinterpret_cast<const uint4*>(dy + o), *reinterpret_cast<const uint2*>(code + o), (uint32_t)(kh * k + kw));
    }
  }
  store8(dx + (((long long)i.n * H + i.h) * W + i.w) * C + i.cv * 8, acc);
}

// 3 x 3 (PAD 0 or 1) and 2 x 2 (PAD 0) windows of stride 2: a thread per block of 2 x 2 input pixels, which lie in the windows of two
// rows and two columns (2 x 2: one): every window is read four times (once) instead of nine (four).
template <int KT, int PAD>
__global__ void maxpool_bwd2_kernel(const uint8_t* __restrict__ code, const bf16* __restrict__ dy, bf16* __restrict__ dx, int N, int H, int W,
                                    int C, int Ho, int Wo) {
  pdl_sync();
  constexpr int R = KT == 2 ? 1 : 2;                       // window rows and columns a block lies in
  const int c8 = C / 8;
  const PoolAt i = pool_at(N, (H + 1) / 2, (W + 1) / 2, c8);
  if (!i.live) return;
  const int h0 = KT == 2 ? i.h : i.h - 1 + PAD, w0 = KT == 2 ? i.w : i.w - 1 + PAD;      // first of them
  uint4 dv[R][R];
  uint2 cd[R][R];
#pragma unroll
  for (int a = 0; a < R; ++a)
#pragma unroll
    for (int b = 0; b < R; ++b) {
      dv[a][b] = make_uint4(0, 0, 0, 0);
      cd[a][b] = make_uint2(0xffffffffu, 0xffffffffu);     // no window: names no tap
      if (h0 + a >= 0 && h0 + a < Ho && w0 + b >= 0 && w0 + b < Wo) {
        const long long o = (((long long)i.n * Ho + h0 + a) * Wo + w0 + b) * C + i.cv * 8;
        dv[a][b] = *reinterpret_cast<const uint4*>(dy + o);
        cd[a][b] = *reinterpret_cast<const uint2*>(code + o);
      }
    }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int hi = 2 * i.h + u, wi = 2 * i.w + v;
      if (hi >= H || wi >= W) continue;
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int a = R - 1; a >= 0; --a)                     // taps in ascending order
#pragma unroll
        for (int b = R - 1; b >= 0; --b) {
          const int kh = u + PAD - 2 * (KT == 2 ? a : a - 1 + PAD), kw = v + PAD - 2 * (KT == 2 ? b : b - 1 + PAD);
          if (kh >= 0 && kh < KT && kw >= 0 && kw < KT) pool_route(acc, dv[a][b], cd[a][b], (uint32_t)(kh * KT + kw));
        }
      store8(dx + (((long long)i.n * H + hi) * W + wi) * C + i.cv * 8, acc);
    }
}

// ------------------------------------------------------------------------------------------------ PowerSGD (K8)
// Rank-r (r <= 4) factors of an fp32 matrix M [m, n]; all three kernels are bandwidth-bound passes over M.
//   psgd_p : M += err (in place); P[i, :] = M[i, :] . Q          one warp per row
//   psgd_q : Qn[j, :] = sum_i M[i, j] * P[i, :]                  blocks own 32 columns, their warps split the rows
//   psgd_d : err = M - P Q^T;  M = P Q^T                          elementwise
constexpr int PSGD_MAXR = 4;

__global__ void psgd_p_kernel(float* __restrict__ M, const float* __restrict__ err, const float* __restrict__ Q, float* __restrict__ P,
                              int m, int n, int r) {
  pdl_sync();
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= m) return;
  float acc[PSGD_MAXR] = {0.f, 0.f, 0.f, 0.f};
  for (int j = lane; j < n; j += 32) {
    const long long idx = (long long)row * n + j;
    float v = M[idx];
    if (err) { v += err[idx]; M[idx] = v; }
    for (int k = 0; k < r; ++k) acc[k] += v * Q[(long long)j * r + k];
  }
  for (int k = 0; k < r; ++k) {
    const float t = warp_sum(acc[k]);
    if (lane == 0) P[(long long)row * r + k] = t;
  }
}

__global__ void psgd_q_kernel(const float* __restrict__ M, const float* __restrict__ P, float* __restrict__ Qn, int m, int n, int r) {
  pdl_sync();
  __shared__ float sm[8][32][PSGD_MAXR];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane;
  float acc[PSGD_MAXR] = {0.f, 0.f, 0.f, 0.f};
  if (col < n)
    for (int i = w; i < m; i += 8) {
      const float v = M[(long long)i * n + col];
      for (int k = 0; k < r; ++k) acc[k] += v * P[(long long)i * r + k];
    }
  for (int k = 0; k < PSGD_MAXR; ++k) sm[w][lane][k] = acc[k];
  __syncthreads();
  if (w == 0 && col < n)
    for (int k = 0; k < r; ++k) {
      float t = 0.f;
      for (int i = 0; i < 8; ++i) t += sm[i][lane][k];
      Qn[(long long)col * r + k] = t;
    }
}

__global__ void psgd_d_kernel(float* __restrict__ M, float* __restrict__ err, const float* __restrict__ P, const float* __restrict__ Q,
                              int m, int n, int r) {
  pdl_sync();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)m * n) return;
  const int i = (int)(idx / n), j = (int)(idx % n);
  float a = 0.f;
  for (int k = 0; k < r; ++k) a += P[(long long)i * r + k] * Q[(long long)j * r + k];
  err[idx] = M[idx] - a;
  M[idx] = a;
}

// ---- PowerSGD over all matrices of a step at once ------------------------------------------------------------------------------
// Each gradient matrix i is M_i = grad[off_i : off_i + m_i * n_i] seen as [m_i, n_i]; its factors live at P[p_off_i] ([m_i, r]) and
// Q[q_off_i] ([n_i, r]) in two flat buffers that are all-reduced as one message each. The three passes run once per step for all
// matrices (a table lookup finds the matrix of a row / column block / element) instead of three launches per variable.
struct PsgdTable {
  const long long* off;         // [nmat] start of M_i in the flat gradient / residual buffers
  const int* m;                 // [nmat]
  const int* n;                 // [nmat]
  const long long* p_off;       // [nmat]
  const long long* q_off;       // [nmat]
  const long long* row_prefix;  // [nmat + 1] rows before matrix i
  const long long* blk_prefix;  // [nmat + 1] 32-column blocks before matrix i
  const long long* elem_prefix; // [nmat + 1] elements before matrix i
  int nmat;
};

__device__ __forceinline__ int psgd_find(const long long* prefix, int nmat, long long x) {
  int lo = 0, hi = nmat - 1;                      // last i with prefix[i] <= x
  while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (prefix[mid] <= x) lo = mid; else hi = mid - 1; }
  return lo;
}

// M += err (written back), P = M Q: one warp per matrix row.
__global__ void psgd_p_batched_kernel(float* __restrict__ grad, const float* __restrict__ err, const float* __restrict__ Q,
                                      float* __restrict__ P, PsgdTable t, int r, long long rows) {
  pdl_sync();
  const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int i = psgd_find(t.row_prefix, t.nmat, row);
  const int n = t.n[i];
  const long long local = row - t.row_prefix[i];
  float* M = grad + t.off[i] + local * n;
  const float* e = err + t.off[i] + local * n;
  const float* q = Q + t.q_off[i];
  float acc[PSGD_MAXR] = {0.f, 0.f, 0.f, 0.f};
  for (int j = lane; j < n; j += 32) {
    const float v = M[j] + e[j];
    M[j] = v;
    for (int k = 0; k < r; ++k) acc[k] += v * q[(long long)j * r + k];
  }
  for (int k = 0; k < r; ++k) {
    const float s = warp_sum(acc[k]);
    if (lane == 0) P[t.p_off[i] + local * r + k] = s;
  }
}

// Modified Gram-Schmidt on the columns of every P_i (one block per matrix), as orthogonalize_ of the Python compressor.
__global__ void psgd_orth_batched_kernel(float* __restrict__ P, PsgdTable t, int r) {
  pdl_sync();
  __shared__ float red[32];
  __shared__ float bcast;
  const int i = blockIdx.x;
  const int m = t.m[i];
  float* p = P + t.p_off[i];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto block_sum = [&](float v) {
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) { float s = 0.f; for (int x = 0; x < nw; ++x) s += red[x]; bcast = s; }
    __syncthreads();
    return bcast;
  };
  for (int k = 0; k < r; ++k) {
    float a = 0.f;
    for (int row = threadIdx.x; row < m; row += blockDim.x) { const float v = p[(long long)row * r + k]; a += v * v; }
    const float inv = 1.0f / (sqrtf(block_sum(a)) + 1e-8f);
    for (int row = threadIdx.x; row < m; row += blockDim.x) p[(long long)row * r + k] *= inv;
    __syncthreads();
    for (int j = k + 1; j < r; ++j) {
      float d = 0.f;
      for (int row = threadIdx.x; row < m; row += blockDim.x) d += p[(long long)row * r + k] * p[(long long)row * r + j];
      const float dot = block_sum(d);
      for (int row = threadIdx.x; row < m; row += blockDim.x) p[(long long)row * r + j] -= dot * p[(long long)row * r + k];
      __syncthreads();
    }
  }
}

// Q = M^T P: one block (8 warps) per 32 columns of one matrix.
__global__ void psgd_q_batched_kernel(const float* __restrict__ grad, const float* __restrict__ P, float* __restrict__ Q, PsgdTable t, int r) {
  pdl_sync();
  __shared__ float sm[8][32][PSGD_MAXR];
  const int i = psgd_find(t.blk_prefix, t.nmat, blockIdx.x);
  const int m = t.m[i], n = t.n[i];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col = (int)(blockIdx.x - t.blk_prefix[i]) * 32 + lane;
  const float* M = grad + t.off[i];
  const float* p = P + t.p_off[i];
  float acc[PSGD_MAXR] = {0.f, 0.f, 0.f, 0.f};
  if (col < n)
    for (int row = w; row < m; row += 8) {
      const float v = M[(long long)row * n + col];
      for (int k = 0; k < r; ++k) acc[k] += v * p[(long long)row * r + k];
    }
  for (int k = 0; k < PSGD_MAXR; ++k) sm[w][lane][k] = acc[k];
  __syncthreads();
  if (w == 0 && col < n)
    for (int k = 0; k < r; ++k) {
      float s = 0.f;
      for (int x = 0; x < 8; ++x) s += sm[x][lane][k];
      Q[t.q_off[i] + (long long)col * r + k] = s;
    }
}

// err = M - P Q^T; M = P Q^T: one thread per element of all matrices.
__global__ void psgd_d_batched_kernel(float* __restrict__ grad, float* __restrict__ err, const float* __restrict__ P, const float* __restrict__ Q,
                                      PsgdTable t, int r, long long total) {
  pdl_sync();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int i = psgd_find(t.elem_prefix, t.nmat, idx);
  const long long local = idx - t.elem_prefix[i];
  const int n = t.n[i];
  const long long row = local / n, col = local % n;
  float a = 0.f;
  for (int k = 0; k < r; ++k) a += P[t.p_off[i] + row * r + k] * Q[t.q_off[i] + col * r + k];
  const long long g = t.off[i] + local;
  err[g] = grad[g] - a;
  grad[g] = a;
}

__global__ void cast_f32_bf16_kernel(const float* __restrict__ x, bf16* __restrict__ y, long long n) {
  pdl_sync();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16(x[i]);
}

// The feed of a step: a handful of small tensors, one launch instead of one copy each. A step of the tiny BERT (seven tensors) took
// 391 us with copies and takes 360, one of NeuMF (three) 439 and 415.
//
// A block copies kCopyBlockBytes (16 KB), 64 bytes per thread, all requested before the first is stored, in the widest words that source
// and destination share. A source that shares none with its destination (a slice of bytes or of 16-bit values) is read in aligned words
// that are shifted together. 64 MB, us, and the library (byte by byte it was 120 at every offset but 0):
// offset 0 19.5 (22.2), 8 20.0 (22.5), 4 20.6 (22.5), 1 or 2 26.2 (44.5).
template <typename W>
__device__ __forceinline__ void copy_words(const char* src, char* dst, long long b0, long long b1) {
  constexpr int U = kCopyBlockBytes / 256 / (int)sizeof(W);
  W v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long at = b0 + (threadIdx.x + 256 * u) * (int)sizeof(W);
    if (at + (int)sizeof(W) <= b1) v[u] = *reinterpret_cast<const W*>(src + at);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long at = b0 + (threadIdx.x + 256 * u) * (int)sizeof(W);
    if (at + (int)sizeof(W) <= b1) *reinterpret_cast<W*>(dst + at) = v[u];
  }
}
__global__ void __launch_bounds__(256) copy_list_kernel(const CopyList c) {
  pdl_sync();
  int i = 0;
  while (i + 1 < c.n && (int)blockIdx.x >= c.first[i + 1]) ++i;
  const long long b0 = (long long)(blockIdx.x - c.first[i]) * kCopyBlockBytes, b1 = min(c.bytes[i], b0 + kCopyBlockBytes);
  const char* src = reinterpret_cast<const char*>(c.src[i]);
  char* dst = reinterpret_cast<char*>(c.dst[i]);
  const unsigned from = (unsigned)(reinterpret_cast<uintptr_t>(src) & 15), to = (unsigned)(reinterpret_cast<uintptr_t>(dst) & 15), both = from | to;
  long long done = b0;
  if ((both & 15) == 0) {
    copy_words<uint4>(src, dst, b0, b1);
    done = b0 + ((b1 - b0) & ~15LL);
  } else if ((both & 7) == 0) {
    copy_words<uint2>(src, dst, b0, b1);
    done = b0 + ((b1 - b0) & ~7LL);
  } else if ((both & 3) == 0) {
    copy_words<uint32_t>(src, dst, b0, b1);
    done = b0 + ((b1 - b0) & ~3LL);
  } else if ((to & 3) == 0) {
    // word t of the destination lies in the words t and t + 1 of the source from `low` on; both lie inside [b0, b1) for t in [1, words)
    const unsigned shift = (from & 3) * 8;
    const uint32_t* low = reinterpret_cast<const uint32_t*>(src + b0 - (from & 3));
    const int words = (int)((b1 - b0 - (4 - (int)(from & 3))) / 4);       // whole words of the source behind the first, cut, one
    if (words > 1) {
      if (threadIdx.x < 4) dst[b0 + threadIdx.x] = src[b0 + threadIdx.x];
      constexpr int U = kCopyBlockBytes / 256 / 4;
      uint32_t v[U], w[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = 1 + threadIdx.x + 256 * u;
        if (t < words) { v[u] = low[t]; w[u] = low[t + 1]; }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = 1 + threadIdx.x + 256 * u;
        if (t < words) *reinterpret_cast<uint32_t*>(dst + b0 + 4 * t) = __funnelshift_r(v[u], w[u], shift);
      }
      done = b0 + 4LL * words;
    }
  }
  for (long long at = done + threadIdx.x; at < b1; at += 256) dst[at] = src[at];
}

__global__ void increment_kernel(long long* c) {
  pdl_sync(); *c += 1; }

inline int blocks_for(long long n, int per) { return (int)((n + per - 1) / per); }

}  // namespace

// ---------------------------------------------------------------------------------------------- launchers
void ln_fwd(const bf16* x, const bf16* res, const float* gamma, const float* beta, bf16* z, bf16* y, float* mean, float* rstd,
            int rows, int H, float eps, float p_drop, uint64_t seed, const long long* step, cudaStream_t st) {
  if (rows <= 0) return;
  const int blocks = blocks_for(rows, kLnWarps) < sm_count() * 8 ? blocks_for(rows, kLnWarps) : sm_count() * 8;
  auto pick = [&](auto early) {
    constexpr bool E = decltype(early)::value;
    return H <= 256 ? ln_fwd_kernel<1, E> : (H <= 512 ? ln_fwd_kernel<2, E> : (H <= 768 ? ln_fwd_kernel<3, E> : ln_fwd_kernel<4, E>));
  };
  auto kern = rows <= sm_count() * 2 * kLnWarps ? pick(std::true_type{}) : pick(std::false_type{});
  launch_pdl(kern, dim3(blocks), dim3(32 * kLnWarps), 0, st, x, res, gamma, beta, z, y, mean, rstd, rows, H, eps, p_drop, seed, step);
}
int ln_bwd_part_floats(int H) { return 3 * kLnSlots * H; }
// part: 3 * 16 * H floats, zero on entry and zero again on return. dsum (optional): column sums of the tensor the kernel hands to the layer in
// front of the residual connection (dx when the dropout copy is written, else dz).
void ln_bwd(const bf16* dy, const bf16* z, const float* mean, const float* rstd, const float* gamma, const bf16* dz_add, bf16* dz,
            bf16* dx, float* part, float* dgamma, float* dbeta, float* dsum, int rows, int H, float p_drop, uint64_t seed,
            const long long* step, int accumulate, cudaStream_t st) {
  // as many blocks as the SMs hold at once, so that a warp keeps several rows (a block's per-column sums are written once)
  const int most = sm_count() * ln_bwd_resident((H + 255) / 256), want = blocks_for(rows, kLnWarps);
  const int blocks = want < 1 ? 1 : (want < most ? want : most);
  auto kern = H <= 256 ? ln_bwd_kernel<1> : (H <= 512 ? ln_bwd_kernel<2> : (H <= 768 ? ln_bwd_kernel<3> : ln_bwd_kernel<4>));
  launch_pdl(kern, dim3(blocks), dim3(32 * kLnWarps), 0, st, dy, z, mean, rstd, gamma, dz_add, dz, dx, part, rows, H, p_drop, seed, step, dsum != nullptr);
  launch_pdl(colsum3_f32_kernel, dim3(dim3(blocks_for(H, 32), dsum != nullptr ? 3 : 2)), dim3(256), 0, st, part, dgamma, dbeta, dsum, kLnSlots, H, accumulate);
}
void embed_sum(const bf16* word, const bf16* pos, const bf16* type, const int64_t* ids, const int64_t* tt, bf16* z, int rows, int S,
               int H, long long V, long long types, int* error, cudaStream_t st) {
  launch_pdl(embed_sum_kernel, dim3(blocks_for(rows, 4)), dim3(128), 0, st, word, pos, type, ids, tt, z, rows, S, H, V, types, error);
}
void scatter_add_rows(float* dst, const int64_t* idx, const bf16* src, int rows, int H, float scale, cudaStream_t st) {
  launch_pdl(scatter_add_rows_kernel, dim3(blocks_for(rows, 4)), dim3(128), 0, st, dst, idx, src, rows, H, scale);
}
void scatter_add_rows_f32(float* dst, const int64_t* idx, const float* src, long long rows, int H, cudaStream_t st) {
  const int h4 = (H + 3) / 4;
  const int vec = H % 4 == 0 && ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15) == 0;
  if (rows > 0) launch_pdl(scatter_add_rows_f32_kernel, dim3(blocks_for(rows * h4, 256)), dim3(256), 0, st, dst, idx, src, rows * h4, h4, H, vec);
}
void pair_lookup(const float* ut, const float* it, const int64_t* users, const int64_t* items, float* gmf, bf16* x, float* kept, long long rows, int mf,
                 int h, long long nu, long long ni, int* error, cudaStream_t st) {
  const long long total = rows * ((mf + h) / 4);
  if (total > 0) launch_pdl(pair_lookup_kernel, dim3(blocks_for(total, 256)), dim3(256), 0, st, ut, it, users, items, gmf, x, kept, total, mf / 4, h / 4, nu, ni, error);
}
void pair_lookup_bwd(const float* dgmf, long long ld, const bf16* dx, const float* kept, const int64_t* users, const int64_t* items, float* gu, float* gi,
                     long long rows, int mf, int h, long long nu, long long ni, cudaStream_t st) {
  const long long total = rows * ((mf + h) / 4);
  if (total > 0) launch_pdl(pair_lookup_bwd_kernel, dim3(blocks_for(total, 256)), dim3(256), 0, st, dgmf, ld, dx, kept, users, items, gu, gi, total, mf / 4, h / 4, nu, ni);
}
int bce_logits_parts(long long n) { return blocks_for(n, kBcePerBlock); }
void bce_logits(const float* x, const float* y, float* part, long long n, float scale, cudaStream_t st) {
  launch_pdl(bce_logits_kernel, dim3(bce_logits_parts(n)), dim3(1024), 0, st, x, y, part, n, scale);
}
void bce_logits_bwd(const float* x, const float* y, const float* grad, float* dx, long long n, float scale, cudaStream_t st) {
  launch_pdl(bce_logits_bwd_kernel, dim3(blocks_for(n, 256)), dim3(256), 0, st, x, y, grad, dx, n, scale);
}
void copy_list(const CopyList& c, cudaStream_t st) {
  if (c.n > 0 && c.first[c.n] > 0) launch_pdl(copy_list_kernel, dim3(c.first[c.n]), dim3(256), 0, st, c);
}
void strided_rowsum(const bf16* x, float* out, int keys, int stride, int count, int H, cudaStream_t st) {
  dim3 grid(blocks_for(H / 8, 128), keys);
  launch_pdl(strided_rowsum_kernel, dim3(grid), dim3(128), 0, st, x, out, keys, stride, count, H);
}
// Chunks of rows: with 16 of them a narrow matrix of many rows (16384 x 64 to 256: bias gradients of a batch of pairs) ran in a few dozen
// blocks, 7.6 us; a chunk per 256 rows takes 3.2.
int colsum_parts(int rows) { return rows >= 4096 ? (rows / 256 < 64 ? rows / 256 : 64) : (rows >= 2048 ? 16 : (rows >= 256 ? 4 : 1)); }
void keyed_colsum(const bf16* x, const int64_t* key, float* part, float* out, int rows, int H, int keys, int accumulate, cudaStream_t st) {
  const int parts = colsum_parts(rows);
  const int rpb = (rows + parts - 1) / parts;
  dim3 grid(blocks_for(H, 64), parts);
  launch_pdl(keyed_colsum_kernel, dim3(grid), dim3(256), 0, st, x, key, part, rows, H, keys, rpb);
  launch_pdl(colsum_f32_kernel, dim3(blocks_for(keys * H, 32)), dim3(256), 0, st, part, out, parts, keys * H, accumulate);
}
void gather_rows(const bf16* src, const int64_t* idx, bf16* out, int rows, int H, cudaStream_t st) {
  launch_pdl(gather_rows_kernel, dim3(blocks_for(rows, 4)), dim3(128), 0, st, src, idx, out, rows, H);
}
void gather_rows_f32(const float* src, const int64_t* idx, bf16* out, int rows, int H, cudaStream_t st) {
  launch_pdl(gather_rows_f32_kernel, dim3(blocks_for(rows, 4)), dim3(128), 0, st, src, idx, out, rows, H);
}
void scatter_add_rows_bf16(bf16* dst, const int64_t* idx, const bf16* src, int rows, int H, cudaStream_t st) {
  launch_pdl(scatter_add_rows_bf16_kernel, dim3(blocks_for(rows, 4)), dim3(128), 0, st, dst, idx, src, rows, H);
}
#define ADB_SOFTMAX_DISPATCH(KERNEL, ...)                                                              \
  do {                                                                                                 \
    const int threads = S / 8;                                                                         \
    if (threads == 8) launch_pdl(KERNEL<8, 1>, dim3(blocks_for(rows * 8, 256)), dim3(256), 0, st, __VA_ARGS__);            \
    else if (threads == 16) launch_pdl(KERNEL<16, 1>, dim3(blocks_for(rows * 16, 256)), dim3(256), 0, st, __VA_ARGS__);    \
    else if (threads == 32) launch_pdl(KERNEL<32, 1>, dim3(blocks_for(rows * 32, 256)), dim3(256), 0, st, __VA_ARGS__);    \
    else if (threads == 64) launch_pdl(KERNEL<32, 2>, dim3(blocks_for(rows * 32, 256)), dim3(256), 0, st, __VA_ARGS__);    \
    else if (threads == 128) launch_pdl(KERNEL<32, 4>, dim3(blocks_for(rows * 32, 256)), dim3(256), 0, st, __VA_ARGS__);   \
  } while (0)
bool softmax_supported(int S) { return S == 64 || S == 128 || S == 256 || S == 512 || S == 1024; }
void softmax_fwd(const bf16* x, const float* mask, bf16* p, bf16* p_drop, long long rows, int S, int rows_per_batch, float scale,
                 float pd, uint64_t seed, const long long* step, cudaStream_t st) {
  ADB_SOFTMAX_DISPATCH(softmax_fwd_kernel, x, mask, p, p_drop, rows, S, rows_per_batch, scale, pd, seed, step);
}
void softmax_bwd(bf16* dp, const bf16* p, long long rows, int S, float scale, float pd, uint64_t seed, const long long* step,
                 cudaStream_t st) {
  ADB_SOFTMAX_DISPATCH(softmax_bwd_kernel, dp, p, rows, S, scale, pd, seed, step);
}
void weight_sum(const float* w, int n, float* out, float eps, cudaStream_t st) { launch_pdl(weight_sum_kernel, dim3(1), dim3(256), 0, st, w, n, out, eps); }
void xent(bf16* logits, const int64_t* labels, const float* weights, const float* denom, float* loss_sum, int rows, int V, int ld,
          float loss_scale, cudaStream_t st) {
  launch_pdl(xent_kernel, dim3(rows), dim3(V >= 4096 ? 1024 : 128), 0, st, logits, labels, weights, denom, loss_sum, V, ld, loss_scale);
}
void gelu_bwd(const bf16* dy, const bf16* u, bf16* dx, long long n, cudaStream_t st) {
  launch_pdl(gelu_bwd_kernel, dim3(blocks_for(n, 256)), dim3(256), 0, st, dy, u, dx, n);
}
void pad_image8(const void* x, int is_fp32, long long sn, long long sc, long long sh, long long sw, int N, int C, int H, int W, bf16* xp,
                int Hp, int Wp, int pad, cudaStream_t st) {
  const long long total = (long long)N * Hp * Wp;
  if (is_fp32) launch_pdl(pad_image8_kernel<float>, dim3(blocks_for(total, 256)), dim3(256), 0, st, reinterpret_cast<const float*>(x), sn, sc, sh, sw, C, H, W, xp, Hp, Wp, pad, total);
  else launch_pdl(pad_image8_kernel<bf16>, dim3(blocks_for(total, 256)), dim3(256), 0, st, reinterpret_cast<const bf16*>(x), sn, sc, sh, sw, C, H, W, xp, Hp, Wp, pad, total);
}
void relu_bwd(const bf16* dy, const bf16* y, bf16* dx, long long n, cudaStream_t st) {
  launch_pdl(relu_bwd_kernel, dim3(blocks_for(n / 8, 256)), dim3(256), 0, st, reinterpret_cast<const uint4*>(dy), reinterpret_cast<const uint4*>(y),
                                                          reinterpret_cast<uint4*>(dx), n / 8);
}
void tanh_bwd(const bf16* dy, const bf16* y, bf16* dx, long long n, cudaStream_t st) {
  launch_pdl(tanh_bwd_kernel, dim3(blocks_for(n, 256)), dim3(256), 0, st, dy, y, dx, n);
}
void add_bf16(const bf16* a, const bf16* b, bf16* out, long long n, cudaStream_t st) {
  launch_pdl(add_bf16_kernel, dim3(blocks_for(n / 8, 256)), dim3(256), 0, st, a, b, out, n / 8);
}
void adam_update(float* p, const float* g, float* m, float* v, bf16* p16, long long n, const float* lr, float b1, float b2,
                 float eps, float wd, int decoupled, const long long* step, float grad_scale, cudaStream_t st) {
  const long long groups = (n / 4 + 1) / 2 + 1;
  const int blocks = (int)((groups + 255) / 256 < sm_count() * 16 ? (groups + 255) / 256 : sm_count() * 16);
  launch_pdl(adam_kernel, dim3(blocks < 1 ? 1 : blocks), dim3(256), 0, st, p, g, m, v, p16, n, lr, b1, b2, eps, wd, decoupled, step, grad_scale);
}
template <class Rule>
void flat_update(float* p, const float* g, float* state, bf16* p16, long long n, const float* lr, const Rule& rule, cudaStream_t st) {
  if (n <= 0) return;
  const bool groups = n >= kFlatGroupsLeast && ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(state)) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(p16) & 7) == 0;
  if (groups) {
    const long long blocks = (n / 8 + 1 + 255) / 256, most = sm_count() * 16LL;
    launch_pdl(flat_update_groups_kernel<Rule>, dim3((unsigned)(blocks < most ? blocks : most)), dim3(256), 0, st, p, g, state, p16, n, lr, rule);
  } else {
    launch_pdl(flat_update_kernel<Rule>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, p, g, state, p16, n, lr, rule);
  }
}
void sgd_update(float* p, const float* g, float* mom, bf16* p16, long long n, const float* lr, float momentum, float dampening,
                float wd, int nesterov, const long long* step, float grad_scale, cudaStream_t st) {
  flat_update(p, g, momentum != 0.f ? mom : nullptr, p16, n, lr, SgdRule{momentum, dampening, wd, grad_scale, nesterov, step}, st);
}
void adagrad_update(float* p, const float* g, float* acc, bf16* p16, long long n, const float* lr, float eps, float wd,
                    float grad_scale, cudaStream_t st) {
  flat_update(p, g, acc, p16, n, lr, AdagradRule{eps, wd, grad_scale}, st);
}
void sparse_rows_update(float* p, float* s1, float* s2, bf16* p16, const int64_t* rows, const float* g, int n, int H, long long V,
                        int kind, const float* lr, float b1, float b2, float eps, const long long* step, float grad_scale,
                        cudaStream_t st) {
  if (n <= 0) return;
  launch_pdl(sparse_rows_update_kernel, dim3(blocks_for(n, 8)), dim3(256), 0, st, p, s1, s2, p16, rows, g, n, H, V, kind, lr, b1, b2, eps, step, grad_scale);
}
void flagged_rows_update(float* p, float* s1, float* s2, bf16* p16, float* g, uint8_t* flags, long long rows, int H, int kind,
                         const float* lr, float b1, float b2, float eps, const long long* step, cudaStream_t st) {
  if (rows <= 0) return;
  const uintptr_t at = reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(s1) | reinterpret_cast<uintptr_t>(s2);
  const int vec = H % 4 == 0 && (at & 15) == 0 && (reinterpret_cast<uintptr_t>(p16) & 7) == 0;
  long long blocks = (rows + 31) / 32;           // a lane per group of four rows: spread over as many warps as there are groups, up to eight blocks per SM, then up to 32 groups a warp
  if (blocks > sm_count() * 8) blocks = sm_count() * 8;
  auto kern = kind == 0 ? flagged_rows_update_kernel<0> : (kind == 1 ? flagged_rows_update_kernel<1> : flagged_rows_update_kernel<2>);
  launch_pdl(kern, dim3((int)blocks), dim3(256), 0, st, p, s1, s2, p16, g, flags, rows, H, lr, b1, b2, eps, step, vec);
}
void lstm_cell_fwd(const float* gates, const float* c_prev, float* c, bf16* h, int B, int S, float fb, cudaStream_t st) {
  launch_pdl(lstm_cell_fwd_kernel, dim3(blocks_for((long long)B * S, 256)), dim3(256), 0, st, gates, c_prev, c, h, B, S, fb);
}
void lstm_cell_bwd(const float* gates, const float* c_prev, const float* c, const float* dh, const float* dc_next, float* dgates,
                   float* dc_prev, int B, int S, float fb, cudaStream_t st) {
  launch_pdl(lstm_cell_bwd_kernel, dim3(blocks_for((long long)B * S, 256)), dim3(256), 0, st, gates, c_prev, c, dh, dc_next, dgates, dc_prev, B, S, fb);
}
void lstm_seq_fwd(const bf16* gates, const float* c_prev, float* c, bf16* h, int B, int S, float fb, cudaStream_t st) {
  launch_pdl(lstm_seq_fwd_kernel, dim3(blocks_for((long long)B * (S / 4), 128)), dim3(128), 0, st, gates, c_prev, c, h, B, S, fb);
}
void lstm_seq_bwd(const bf16* gates, const float* c_prev, const float* c, const bf16* dh, const float* dc_next, bf16* dgates, float* dc_prev, int B,
                  int S, float fb, cudaStream_t st) {
  launch_pdl(lstm_seq_bwd_kernel, dim3(blocks_for((long long)B * (S / 4), 128)), dim3(128), 0, st, gates, c_prev, c, dh, dc_next, dgates, dc_prev, B, S, fb);
}
void sumsq(const float* x, long long n, float* acc, float weight, cudaStream_t st) {
  const int blocks = (int)(n / 1024 + 1 < 592 ? n / 1024 + 1 : 592);
  launch_pdl(sumsq_kernel, dim3(blocks), dim3(256), 0, st, x, n, acc, weight);
}
void clip_scale(float* x, long long n, const float* acc, float max_norm, cudaStream_t st) {
  const int blocks = (int)(n / 1024 + 1 < 592 ? n / 1024 + 1 : 592);
  launch_pdl(clip_scale_kernel, dim3(blocks), dim3(256), 0, st, x, n, acc, max_norm);
}
// Row chunks per channel block: enough blocks to fill the SMs (~8 per SM) while each chunk keeps >= 128 rows.
int bn_bwd_part_floats(int C) { return kBnCounterFloats + kBnSlots * 2 * C; }
int bn_parts(int rows, int C) {
  const int cb = (C + 63) / 64;
  int parts = (592 + cb - 1) / cb;
  if (parts > rows / 128) parts = rows / 128;
  if (parts > 512) parts = 512;
  return parts < 1 ? 1 : parts;
}
// One wave of resident blocks (`per_sm` per SM) unless that leaves a thread fewer than kBnUnroll rows.
dim3 bn_grid(long long rows, int C, int per_sm) {
  const int c8 = C / 8, tpr = c8 < kBnThreads ? c8 : kBnThreads, rpb = kBnThreads / tpr, gy = (c8 + kBnThreads - 1) / kBnThreads;
  long long blocks = (rows + (long long)rpb * kBnUnroll - 1) / ((long long)rpb * kBnUnroll);
  const long long cap = (sm_count() * per_sm + gy - 1) / gy;
  if (blocks > cap) blocks = cap;
  return dim3((unsigned)(blocks < 1 ? 1 : blocks), (unsigned)gy);
}
// sums [2, C] = per-channel sum and sum of squares of x. part: [bn_parts, 2, C]
void bn_sums(const bf16* x, float* part, float* sums, int rows, int C, cudaStream_t st) {
  const int parts = bn_parts(rows, C), rpb = (rows + parts - 1) / parts;
  launch_pdl(bn_stats_kernel, dim3(dim3(blocks_for(C, 64), parts)), dim3(256), 0, st, x, part, rows, C, rpb);
  launch_pdl(colsum_f32_kernel, dim3(blocks_for(2 * C, 32)), dim3(256), 0, st, part, sums, parts, 2 * C, 0);
}
// part: [bn_parts, 2, C]; sums: [2, C]
// sums_given: `sums` already holds the per-channel sum and sum of squares (the convolution's epilogue produced them); the
// whole normalisation is then one launch.
// keep (optional, [rows, C / 8] bytes): which outputs are positive, for the backward pass of a fused ReLU
void bn_fwd(const bf16* x, const float* gamma, const float* beta, const bf16* res, bf16* y, uint8_t* keep, float* mean, float* rstd, float* part,
            float* sums, int rows, int C, float eps, int relu, int sums_given, float* run_mean, float* run_var, long long* batches,
            float momentum, cudaStream_t st) {
  const float unbias = rows > 1 ? (float)rows / (float)(rows - 1) : 1.0f;
  if (!sums_given) bn_sums(x, part, sums, rows, C, st);
  dim3 grid = bn_grid(rows, C, 3);
  if ((grid.x + 1) * grid.y <= sm_count() * 3 || grid.x == 1) grid.x += 1;      // the block of the statistics, within the same wave
  launch_pdl(bn_apply_kernel, grid, dim3(kBnThreads), 0, st, x, res, y, relu ? keep : nullptr, (long long)rows, C, relu, sums, gamma, beta,
             1.0f / rows, eps, mean, rstd, run_mean, run_var, batches, momentum, unbias);
}
void bn_eval(const bf16* x, const bf16* res, bf16* y, const float* gamma, const float* beta, const float* mean, const float* var, float eps,
             int rows, int C, int relu, cudaStream_t st) {
  launch_pdl(bn_eval_kernel, bn_grid(rows, C, 2), dim3(kBnThreads), 0, st, x, res, y, (long long)rows, C, relu, gamma, beta, mean, var, eps);
}
// part: [bn_bwd_part_floats], zero between calls; sums: [2, C]; coef: [3, C]
void bn_bwd(const bf16* dy, const bf16* x, const uint8_t* keep, const float* mean, const float* rstd, const float* gamma, bf16* dx, bf16* dres,
            float* part, float* sums, float* coef, int rows, int C, int relu, float* dgamma_acc, float* dbeta_acc, const bf16* add, long long add_ld,
            cudaStream_t st) {
  const int parts = bn_parts(rows, C), rpb = (rows + parts - 1) / parts;
  launch_pdl(bn_bwd_stats_kernel, dim3(dim3(blocks_for(C, 64), parts)), dim3(256), 0, st, dy, x, keep, mean, rstd, gamma, reinterpret_cast<unsigned int*>(part),
                                                                      part + kBnCounterFloats, sums, coef, dgamma_acc, dbeta_acc, rows, C, rpb,
                                                                      relu, 1.0f / rows);
  launch_pdl(add != nullptr ? bn_bwd_apply_kernel<true> : bn_bwd_apply_kernel<false>, bn_grid(rows, C, 2), dim3(kBnThreads), 0, st, dy, x, keep, coef, add, add_ld, dx, dres, (long long)rows, C, relu);
}
// dx = relu'(y) * dy (skipped when y is null) and out[c] (+)= column sums of dx. part: [bn_parts(rows, C), C] floats.
void relu_bwd_colsum(const bf16* dy, const bf16* y, bf16* dx, float* part, float* out, int rows, int C, int accumulate, cudaStream_t st) {
  const int parts = bn_parts(rows, C), rpb = (rows + parts - 1) / parts;
  launch_pdl(relu_bwd_colsum_kernel, dim3(dim3(blocks_for(C, 64), parts)), dim3(256), 0, st, dy, y, dx, part, rows, C, rpb);
  launch_pdl(colsum_f32_kernel, dim3(blocks_for(C, 32)), dim3(256), 0, st, part, out, parts, C, accumulate);
}
void maxpool_fwd(const bf16* x, bf16* y, uint8_t* code, int N, int H, int W, int C, int k, int stride, int pad, int Ho, int Wo,
                 cudaStream_t st) {
  if (N <= 0 || Ho <= 0 || Wo <= 0 || C < 8) return;
  const dim3 grid(blocks_for((long long)N * Ho * Wo * (C / 8), 256));
  auto kern = stride == 2 && k == 3 ? maxpool_fwd_kernel<3, 2> : (stride == 2 && k == 2 ? maxpool_fwd_kernel<2, 2> : maxpool_fwd_kernel<0, 0>);
  launch_pdl(kern, grid, dim3(256), 0, st, x, y, code, N, H, W, C, k, stride, pad, Ho, Wo);
}
void maxpool_bwd(const uint8_t* code, const bf16* dy, bf16* dx, int N, int H, int W, int C, int k, int stride, int pad, int Ho, int Wo,
                 cudaStream_t st) {
  if (N <= 0 || H <= 0 || W <= 0 || C < 8) return;
  if (stride == 2 && ((k == 3 && (pad == 0 || pad == 1)) || (k == 2 && pad == 0))) {
    const dim3 grid(blocks_for((long long)N * ((H + 1) / 2) * ((W + 1) / 2) * (C / 8), 256));
    auto kern = k == 2 ? maxpool_bwd2_kernel<2, 0> : (pad == 1 ? maxpool_bwd2_kernel<3, 1> : maxpool_bwd2_kernel<3, 0>);
    launch_pdl(kern, grid, dim3(256), 0, st, code, dy, dx, N, H, W, C, Ho, Wo);
    return;
  }
  const dim3 grid(blocks_for((long long)N * H * W * (C / 8), 256));
  launch_pdl(maxpool_bwd_kernel, grid, dim3(256), 0, st, code, dy, dx, N, H, W, C, k, stride, pad, Ho, Wo);
}
void im2col(const bf16* x, bf16* cols, int N, int H, int W, int C, int KH, int KW, int stride, int pad, int Ho, int Wo, cudaStream_t st) {
  const long long total = (long long)N * Ho * Wo * KH * KW * (C / 8);
  launch_pdl(im2col_kernel, dim3(blocks_for(total, 256)), dim3(256), 0, st, x, cols, N, H, W, C, KH, KW, stride, pad, Ho, Wo);
}
void col2im(const bf16* dcols, bf16* dx, int N, int H, int W, int C, int KH, int KW, int stride, int pad, int Ho, int Wo, cudaStream_t st) {
  const long long total = (long long)N * H * W * (C / 8);
  launch_pdl(col2im_kernel, dim3(blocks_for(total, 256)), dim3(256), 0, st, dcols, dx, N, H, W, C, KH, KW, stride, pad, Ho, Wo);
}
void psgd_p(float* M, const float* err, const float* Q, float* P, int m, int n, int r, cudaStream_t st) {
  launch_pdl(psgd_p_kernel, dim3(blocks_for(m, 4)), dim3(128), 0, st, M, err, Q, P, m, n, r);
}
void psgd_q(const float* M, const float* P, float* Qn, int m, int n, int r, cudaStream_t st) {
  launch_pdl(psgd_q_kernel, dim3(blocks_for(n, 32)), dim3(256), 0, st, M, P, Qn, m, n, r);
}
void psgd_d(float* M, float* err, const float* P, const float* Q, int m, int n, int r, cudaStream_t st) {
  launch_pdl(psgd_d_kernel, dim3(blocks_for((long long)m * n, 256)), dim3(256), 0, st, M, err, P, Q, m, n, r);
}
// tab: int64 [8 arrays] laid out by the caller as device pointers; phase 0 = P pass, 1 = orthogonalise, 2 = Q pass, 3 = decompress.
void psgd_batched(int phase, float* grad, float* err, float* P, float* Q, const long long* off, const int* m, const int* n,
                  const long long* p_off, const long long* q_off, const long long* row_prefix, const long long* blk_prefix,
                  const long long* elem_prefix, int nmat, int r, long long rows, long long blocks, long long elems, cudaStream_t st) {
  if (nmat <= 0) return;
  PsgdTable t{off, m, n, p_off, q_off, row_prefix, blk_prefix, elem_prefix, nmat};
  if (phase == 0) launch_pdl(psgd_p_batched_kernel, dim3(blocks_for(rows, 4)), dim3(128), 0, st, grad, err, Q, P, t, r, rows);
  else if (phase == 1) launch_pdl(psgd_orth_batched_kernel, dim3(nmat), dim3(256), 0, st, P, t, r);
  else if (phase == 2) launch_pdl(psgd_q_batched_kernel, dim3((unsigned)blocks), dim3(256), 0, st, grad, P, Q, t, r);
  else launch_pdl(psgd_d_batched_kernel, dim3(blocks_for(elems, 256)), dim3(256), 0, st, grad, err, P, Q, t, r, elems);
}
void cast_f32_bf16(const float* x, bf16* y, long long n, cudaStream_t st) {
  launch_pdl(cast_f32_bf16_kernel, dim3(blocks_for(n, 256)), dim3(256), 0, st, x, y, n);
}
void increment(long long* c, cudaStream_t st) { launch_pdl(increment_kernel, dim3(1), dim3(1), 0, st, c); }

}  // namespace adb200
