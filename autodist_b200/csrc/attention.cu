// Fused self-attention on tcgen05, forward and backward, for heads of 64 columns: the S x S scores, probabilities and their
// gradients live in tensor memory and registers only.
//
// Forward (one CTA per head and 128 queries, two CTAs per SM): S = Q K^T per tile of 128 keys, online softmax in registers (two
// threads per query row), dropout, P (bf16) through shared memory, O = P V per tile, rescaled and summed in registers in fp32.
// Writes the context and the log of the row sums.
//
// Backward: P is recomputed from the log sums, dP = dO V^T, dS = scale * P * (dP * keep - sum(dO * O)). One kernel, three roles:
//   BWD_ALL  S <= 128: a head is one tile; dQ, dK, dV of a head at once
//   BWD_KV   the CTA owns 128 keys and walks the query tiles: dV += (P keep)^T dO, dK += dS^T Q
//   BWD_Q    the CTA owns 128 queries and walks the key tiles: dQ += dS K
// For S > 128 the scores are recomputed by both roles; that is cheaper than summing dQ across CTAs: the products are a
// quarter of the time, and no fp32 gradient travels through memory. CTAs are persistent over heads / owned tiles, with the next
// tiles in flight (TMA) and the next scores multiplied while 16 warps work on the current ones (four threads per row).
//
// What bounds it: the elementwise part - exponential, dropout, conversions - about 20 instructions per score and pass. Without
// fusion the same scores made 11 passes through memory per layer as bf16. The dropout decisions are the ones of the
// softmax kernels (elementwise.cu): same counter-based function of (seed, step, offset in [B, heads, S, S]). Hashing costs as
// much as the rest of a pass, so the forward pass keeps the decisions as bits (1/16 of the scores' bf16 bytes).
//
// Per layer, 16 heads, dropout 0.1 (separate products and softmax kernels -> here): 32 x 128 tokens forward 37 -> 17 us, backward
// 52 -> 20; 6 x 512 tokens forward about 85 -> 36, backward about 140 -> 54 (60 with the next scores multiplied only once P and dS of
// the current ones were in shared memory, and one value per instruction). The backward pass took 124 us while it hashed the
// decisions again, read its row sums when it needed them and stored 32-byte pieces of the gradients directly.
//
// Every mbarrier wait is bounded: a role that gives up raises `abort`, which ends the waits of the others, and records a code.
#include "attention.h"
#include "gemm_epilogue.cuh"
#include "pdl.cuh"
#include "tcgen05_common.cuh"

namespace adb200 {
namespace {

using namespace tc;

constexpr int TILE = 128 * 64 * 2;        // 128 rows x 64 bf16, one 128-byte swizzle row each
constexpr int PTILE = 2 * TILE;           // 128 x 128 bf16 as two chunks of 64 columns

__device__ __forceinline__ void named_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// D[128, N] (+)= A B^T over 64 columns, both K-major tiles of 128-byte rows.
__device__ __forceinline__ void mma_nt64(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc) {
#pragma unroll
  for (int k = 0; k < 4; ++k) umma(d, make_desc(a + k * 32, 16, 1024), make_desc(b + k * 32, 16, 1024), idesc, k != 0);
}
// D[128, 64] (+)= P X over 128 rows of X: P [128, 128] K-major in two chunks, X [128, 64] with its columns contiguous (MN-major B).
__device__ __forceinline__ void mma_px(uint32_t d, uint32_t p, uint32_t x, uint32_t idesc, bool accumulate) {
#pragma unroll
  for (int k = 0; k < 8; ++k)
    umma(d, make_desc(p + (k >> 2) * TILE + (k & 3) * 32, 16, 1024), make_desc(x + k * 2048, TILE, 1024), idesc, (accumulate || k != 0) ? 1u : 0u);
}
// D[128, 64] (+)= P^T X over 128 rows: P's columns become the rows of D (MN-major A, chunks of 64 columns TILE bytes apart).
__device__ __forceinline__ void mma_ptx(uint32_t d, uint32_t p, uint32_t x, uint32_t idesc, bool accumulate) {
#pragma unroll
  for (int k = 0; k < 8; ++k)
    umma(d, make_desc(p + k * 2048, TILE, 1024), make_desc(x + k * 2048, TILE, 1024), idesc, (accumulate || k != 0) ? 1u : 0u);
}

constexpr float kLog2e = 1.4426950408889634f;
// 2^x on the special-function unit; the callers fold log2(e) into the factor and the offset of the scores.
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}

// The additive mask in base 2. Finite masks end at -65536: a key that far below another one has a weight of zero either way, and the
// lowest float, which would overflow here, keeps its place above minus infinity (a key that does not exist). Scores of a row
// whose keys all lie there are told apart to 2^-7.
__device__ __forceinline__ float mask_base2(float mask) { return mask > -INFINITY ? fmaxf(mask * kLog2e, -65536.f) : mask; }

// Decision bits of 32 consecutive scores whose first has offset `base` (a multiple of 4: one counter decides four neighbours, so with
// dropout the rows must be multiples of four long; the launchers check it). mix64 of consecutive counters, their products with the
// odd constant formed by additions.
__device__ __forceinline__ uint32_t keep_bits32(uint64_t seed, uint64_t base, uint32_t thresh16) {
  constexpr uint64_t kStep = 0x9E3779B97F4A7C15ull;
  const uint64_t x0 = seed + (base >> 2) * kStep;
  const uint32_t limit = thresh16 << 16;
  uint32_t bits = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    uint64_t x = x0 + (uint64_t)i * kStep;
    x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull;
    x ^= x >> 27; x *= 0x94D049BB133111EBull;
    x ^= x >> 31;
    const uint32_t lo = (uint32_t)x, hi = (uint32_t)(x >> 32);
    // a 16-bit field against the threshold: compared in the upper half of a word, where the lower half does not matter
    if ((lo << 16) >= limit) bits |= 1u << (4 * i);
    if (lo >= limit) bits |= 2u << (4 * i);
    if ((hi << 16) >= limit) bits |= 4u << (4 * i);
    if (hi >= limit) bits |= 8u << (4 * i);
  }
  return bits;
}

// 1 / keep probability. With probability 1 no score is kept: context and gradients are zero, and any finite factor will do.
__device__ __forceinline__ float inverse_keep(float drop_p) { return drop_p > 0.f && drop_p < 1.f ? 1.0f / (1.0f - drop_p) : 1.0f; }

// A wait of the elementwise warps, which meet in named barriers: a warp whose wait fails raises the abort flag and walks on
// without waiting, so that nobody is left behind at a barrier.
__device__ __forceinline__ void soft_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, bool& ok) {
  if (ok && !mbar_wait(bar, parity, abort_flag)) {
    ok = false;
    *abort_flag = 1;
  }
}

// Waits for copies that were requested on `bars[i]` but that nobody will consume any more (after an abort).
__device__ __forceinline__ void drain(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try(bar, parity) && clock64() - t0 < 20000000LL) {}
}

// ------------------------------------------------------------------------------------------------ forward
constexpr int FWD_SOFT = 256;                       // softmax threads: two per query row, 64 keys each
constexpr int FWD_THREADS = FWD_SOFT + 64;          // + TMA warp + MMA warp
constexpr int FWD_MAX_S = 1024;
constexpr int FWD_SMEM = TILE /*Q*/ + 2 * TILE /*K*/ + TILE /*V*/ + PTILE + FWD_MAX_S * 4 /*mask*/ + 4 * 128 * 4 /*row exchange*/ + 128 /*barriers*/ + 1024;

__global__ void __launch_bounds__(FWD_THREADS, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv,
                const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + TILE;
  uint8_t* sV = sK + 2 * TILE;
  uint8_t* sP = sV + TILE;
  float* s_mask = reinterpret_cast<float*>(sP + PTILE);
  float* s_red = s_mask + FWD_MAX_S;                 // [2][2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_red + 4 * 128);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 3, *v_full = bars + 5, *v_empty = bars + 6, *s_full = bars + 7, *p_full = bars + 8,
           *o_full = bars + 9;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 10; ++i) mbar_init(&bars[i], &bars[i] == p_full ? FWD_SOFT / 32 : 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(256) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tO = tmem + 128;
  pdl_sync();

  const int tiles = (p.S + 127) / 128;
  const int qt = blockIdx.x % tiles, h = (blockIdx.x / tiles) % p.heads, b = blockIdx.x / (tiles * p.heads);
  const int H = p.heads * 64;

  if (warp == 8) {
    if (elect_one()) {
      bool ok = true;
      int nk = 0, nv = 0;
      mbar_expect_tx(q_full, TILE);
      tma_load_4d(sQ, &mq, q_full, 0, qt * 128, h, b);
      for (int j = 0; j < tiles && ok; ++j) {
        ok = mbar_wait(&k_empty[j & 1], ((j >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(&k_full[j & 1], TILE);
        tma_load_4d(sK + (j & 1) * TILE, &mk, &k_full[j & 1], 0, j * 128, h, b);
        ++nk;
        ok = mbar_wait(v_empty, (j & 1) ^ 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(v_full, TILE);
        tma_load_4d(sV, &mv, v_full, 0, j * 128, h, b);
        ++nv;
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.error_flag) atomicExch(p.error_flag, 61);
      }
      if (*abort_flag) {
        drain(q_full, 0);
        for (int j = nk > 2 ? nk - 2 : 0; j < nk; ++j) drain(&k_full[j & 1], (j >> 1) & 1);
        if (nv > 0) drain(v_full, (nv - 1) & 1);
      }
    }
  } else if (warp == 9) {
    if (elect_one()) {
      const uint32_t id_s = make_idesc(128, false, false), id_o = make_idesc(64, false, true);
      const uint32_t aQ = smem_u32(sQ), aK = smem_u32(sK), aV = smem_u32(sV), aP = smem_u32(sP);
      bool ok = mbar_wait(q_full, 0, abort_flag) && mbar_wait(&k_full[0], 0, abort_flag);
      if (ok) {
        tc_fence_after();
        mma_nt64(tS, aQ, aK, id_s);
        umma_commit(s_full);
        umma_commit(&k_empty[0]);
      }
      for (int j = 0; j < tiles && ok; ++j) {
        ok = mbar_wait(p_full, j & 1, abort_flag);       // P(j) is in shared memory, S(j) and O(j - 1) have been read
        if (!ok) break;
        tc_fence_after();
        if (j + 1 < tiles) {
          ok = mbar_wait(&k_full[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          mma_nt64(tS, aQ, aK + ((j + 1) & 1) * TILE, id_s);
          umma_commit(s_full);
          umma_commit(&k_empty[(j + 1) & 1]);
        }
        ok = mbar_wait(v_full, j & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        mma_px(tO, aP, aV, id_o, false);
        umma_commit(o_full);
        umma_commit(v_empty);
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.error_flag) atomicExch(p.error_flag, 62);
      }
    }
  } else {
    const int q = warp & 3, hf = warp >> 2;
    const int r = q * 32 + lane;                           // row of the tile
    const int row = qt * 128 + r;                          // query
    for (int c = threadIdx.x; c < tiles * 128; c += FWD_SOFT)
      s_mask[c] = c < p.S ? (p.mask != nullptr ? mask_base2(p.mask[(long long)b * p.S + c]) : 0.f) : -INFINITY;
    const float scale2 = p.scale * kLog2e;                 // scores, maxima and exponents are kept in base 2
    const uint64_t scale2x = both(scale2);
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    const uint32_t thresh = (uint32_t)(p.drop_p * 65536.0f);
    const uint32_t some = thresh > 0xffffu ? 0u : 0xffffffffu;      // probability 1: no 16-bit field reaches the threshold
    const float inv_keep = inverse_keep(p.drop_p);
    const uint64_t sd = p.seed + (p.step ? (uint64_t)(*p.step) * 0x100000001B3ull : 0ull);
    const uint64_t row_off = (((uint64_t)b * p.heads + h) * p.S + row) * p.S;
    const long long keep_row = (((long long)b * p.heads + h) * p.S + row) * attn_keep_words(p.S);
    const uint32_t p_row = smem_u32(sP) + (uint32_t)hf * TILE + (uint32_t)r * 128u;
    const uint32_t swz = (uint32_t)(r & 7);
    float m = -INFINITY, l = 0.f, corr = 0.f;
    float o[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) o[i] = 0.f;
    bool ok = true;
    named_sync(1, FWD_SOFT);                               // the mask is in shared memory
    for (int j = 0; j < tiles; ++j) {
      soft_wait(s_full, j & 1, abort_flag, ok);
      tc_fence_after();
      // Most blocks of 64 keys carry one mask value (no padding among them): the maximum is then taken over the bare scores and the
      // exponent's argument is one fused multiply-add.
      const float* mk = s_mask + j * 128 + hf * 64;
      const float m0 = mk[0];
      const bool plain = __all_sync(0xffffffffu, mk[lane] == m0 && mk[32 + lane] == m0 && m0 > -INFINITY);
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float v[16];
        tmem_ld16(tS + lane_base + hf * 64 + c * 16, v);
        if (plain) {
#pragma unroll
          for (int i = 0; i < 16; i += 2) mx = max3(mx, v[i], v[i + 1]);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) mx = fmaxf(mx, fmaf(v[i], scale2, mk[c * 16 + i]));
        }
      }
      if (plain) mx = fmaf(mx, scale2, m0);
      float* red = s_red + (j & 1) * 256;
      red[hf * 128 + r] = mx;
      named_sync(1, FWD_SOFT);
      const float m_new = fmaxf(m, fmaxf(mx, red[(hf ^ 1) * 128 + r]));
      // Keys masked with minus infinity up to here: nothing to rescale, and the exponents are taken against 0 instead of the maximum
      // (a row without any key ends as 0 / 0).
      const float base = m_new > -INFINITY ? m_new : 0.f;
      const float corr_new = ex2(m - base);
      m = m_new;
      l *= corr_new;
      if (j > 0) {                                         // the context of the tiles before, in terms of their maximum
        soft_wait(o_full, (j - 1) & 1, abort_flag, ok);
        tc_fence_after();
        float v[32];
        tmem_ld32(tO + lane_base + hf * 32, v);
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = fmaf(o[i], corr, v[i]);
      }
      corr = corr_new;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int key = j * 128 + hf * 64 + c * 32;
        uint32_t bits = 0xffffffffu;
        if (p.drop_p > 0.f) {
          bits = keep_bits32(sd, row_off + (uint64_t)key, thresh) & some;
          if (row < p.S) p.keep[keep_row + (key >> 5)] = bits;
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float v[16];
          tmem_ld16(tS + lane_base + hf * 64 + c * 32 + e * 16, v);
          if (plain) {
            const uint64_t off = both(m0 - base);
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              const float2 arg = unpack_f32x2(fma2(pack_f32x2(v[i], v[i + 1]), scale2x, off));
              v[i] = ex2(arg.x);
              v[i + 1] = ex2(arg.y);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = ex2(fmaf(v[i], scale2, mk[c * 32 + e * 16 + i] - base));
          }
          uint64_t sum0 = 0, sum1 = 0;
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            sum0 = add2(sum0, pack_f32x2(v[i], v[i + 1]));
            sum1 = add2(sum1, pack_f32x2(v[i + 2], v[i + 3]));
          }
          const float2 sum = unpack_f32x2(add2(sum0, sum1));
          l += sum.x + sum.y;
          if (p.drop_p > 0.f) {                            // 1 / keep probability is applied to the context at the end
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = (bits >> (e * 16 + i)) & 1u ? v[i] : 0.f;
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
            st_shared_v4(p_row + (((uint32_t)(c * 4 + e * 2 + i) ^ swz) << 4), pack_bf16x2(v[8 * i], v[8 * i + 1]), pack_bf16x2(v[8 * i + 2], v[8 * i + 3]),
                         pack_bf16x2(v[8 * i + 4], v[8 * i + 5]), pack_bf16x2(v[8 * i + 6], v[8 * i + 7]));
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (elect_one()) mbar_arrive(p_full);
    }
    soft_wait(o_full, (tiles - 1) & 1, abort_flag, ok);
    tc_fence_after();
    s_red[((tiles & 1) * 2 + hf) * 128 + r] = l;           // the exchange buffer the last tile did not use
    named_sync(1, FWD_SOFT);
    l += s_red[((tiles & 1) * 2 + (hf ^ 1)) * 128 + r];
    const float inv = inv_keep / l;
    float out[32];
    tmem_ld32(tO + lane_base + hf * 32, out);
#pragma unroll
    for (int i = 0; i < 32; ++i) out[i] = fmaf(o[i], corr, out[i]) * inv;
    if (row < p.S) {
      __nv_bfloat16* dst = p.ctx + ((long long)b * p.S + row) * H + h * 64 + hf * 32;
#pragma unroll
      for (int i = 0; i < 4; ++i) store8_bf16(dst + 8 * i, out + 8 * i);
      if (hf == 0) p.lse[((long long)b * p.heads + h) * p.S + row] = m / kLog2e + __logf(l);
    }
    if (!ok && lane == 0 && p.error_flag) atomicExch(p.error_flag, 63);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------ backward
enum { BWD_ALL = 0, BWD_KV = 1, BWD_Q = 2 };
constexpr int BWD_SOFT = 512;                       // four threads per row, 32 keys each
constexpr int BWD_THREADS = BWD_SOFT + 64;
constexpr int BWD_SMEM = 4 * TILE /*owned, two items*/ + 4 * TILE /*walked, two iterations*/ + 2 * PTILE + 128 /*barriers*/ + 1024;

// delta[b][h][s] = sum over the head's 64 columns of dctx * ctx: eight lanes per head, 16-byte loads, one pass.
__global__ void __launch_bounds__(256) attn_delta_kernel(const AttnParams p, long long groups) {
  pdl_sync();
  const long long g = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3;      // (token, head)
  const int l8 = threadIdx.x & 7;
  float part = 0.f;
  if (g < groups) {
    float a[8], d[8];
    load8_bf16(p.ctx + g * 64 + l8 * 8, a);
    load8_bf16(p.dctx + g * 64 + l8 * 8, d);
#pragma unroll
    for (int x = 0; x < 8; ++x) part = fmaf(a[x], d[x], part);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (g < groups && l8 == 0) {
    const long long token = g / p.heads;
    p.delta[((token / p.S) * p.heads + g % p.heads) * p.S + token % p.S] = part;
  }
}

template <int MODE>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv,
                const __grid_constant__ CUtensorMap mdo, const __grid_constant__ AttnGradMaps grads, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sOwn = smem;                              // [2 items][2 tiles]: K, V (or Q, dO when queries are owned)
  uint8_t* sOth = sOwn + 4 * TILE;                   // [2 iterations][2 tiles]: Q, dO (or K, V)
  uint8_t* sP = sOth + 4 * TILE;
  uint8_t* sD = sP + PTILE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sD + PTILE);
  uint64_t *own_full = bars, *own_empty = bars + 2, *oth_full = bars + 4, *oth_empty = bars + 6, *s_full = bars + 8, *pd_full = bars + 9,
           *acc_done = bars + 10, *acc_free = bars + 11, *s_read = bars + 12;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 13; ++i) mbar_init(&bars[i], (&bars[i] == pd_full || &bars[i] == acc_free || &bars[i] == s_read) ? BWD_SOFT / 32 : 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 17) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tDP = tmem + 128, tAcc = tmem + 256;      // accumulators: dV | dK | dQ (KV, ALL), dQ (Q)
  pdl_sync();

  const int tiles = (p.S + 127) / 128;
  const int inner = MODE == BWD_ALL ? 1 : tiles;
  const int items = p.B * p.heads * (MODE == BWD_ALL ? 1 : tiles);
  // item -> owned tile, head, sequence; iteration it of the CTA -> its item number and inner step
  auto own_tile = [&](int item) { return MODE == BWD_ALL ? 0 : item % tiles; };
  auto head_of = [&](int item) { return (MODE == BWD_ALL ? item : item / tiles) % p.heads; };
  auto batch_of = [&](int item) { return (MODE == BWD_ALL ? item : item / tiles) / p.heads; };

  if (warp == 16) {
    if (elect_one()) {
      bool ok = true;
      int n_own = 0, n_oth = 0;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const int ot = own_tile(item), h = head_of(item), b = batch_of(item);
        const int os = n_own & 1;
        ok = mbar_wait(&own_empty[os], ((n_own >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(&own_full[os], 2 * TILE);
        tma_load_4d(sOwn + os * 2 * TILE, MODE == BWD_Q ? &mq : &mk, &own_full[os], 0, ot * 128, h, b);
        tma_load_4d(sOwn + os * 2 * TILE + TILE, MODE == BWD_Q ? &mdo : &mv, &own_full[os], 0, ot * 128, h, b);
        ++n_own;
        for (int i = 0; i < inner; ++i) {
          const int st = n_oth & 1;
          ok = mbar_wait(&oth_empty[st], ((n_oth >> 1) & 1) ^ 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(&oth_full[st], 2 * TILE);
          tma_load_4d(sOth + st * 2 * TILE, MODE == BWD_Q ? &mk : &mq, &oth_full[st], 0, i * 128, h, b);
          tma_load_4d(sOth + st * 2 * TILE + TILE, MODE == BWD_Q ? &mv : &mdo, &oth_full[st], 0, i * 128, h, b);
          ++n_oth;
        }
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.error_flag) atomicExch(p.error_flag, 64);
      }
      if (*abort_flag) {
        for (int j = n_own > 2 ? n_own - 2 : 0; j < n_own; ++j) drain(&own_full[j & 1], (j >> 1) & 1);
        for (int j = n_oth > 2 ? n_oth - 2 : 0; j < n_oth; ++j) drain(&oth_full[j & 1], (j >> 1) & 1);
      }
    }
  } else if (warp == 17) {
    if (elect_one()) {
      const uint32_t id_s = make_idesc(128, false, false), id_t = make_idesc(64, true, true), id_q = make_idesc(64, false, true);
      const uint32_t aOwn = smem_u32(sOwn), aOth = smem_u32(sOth), aP = smem_u32(sP), aD = smem_u32(sD);
      const int my_items = items > (int)blockIdx.x ? (items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
      const int total = my_items * inner;
      bool ok = true;
      // scores and dP of iteration t
      auto issue_scores = [&](int t) {
        const int it = t / inner, os = it & 1, st = t & 1;
        if (t % inner == 0 && !mbar_wait(&own_full[os], (it >> 1) & 1, abort_flag)) return false;
        if (!mbar_wait(&oth_full[st], (uint32_t)(t >> 1) & 1u, abort_flag)) return false;
        tc_fence_after();
        const uint32_t own = aOwn + os * 2 * TILE, oth = aOth + st * 2 * TILE;
        const uint32_t qk_a = MODE == BWD_Q ? own : oth, qk_b = MODE == BWD_Q ? oth : own;
        mma_nt64(tS, qk_a, qk_b, id_s);                               // S = Q K^T
        mma_nt64(tDP, qk_a + TILE, qk_b + TILE, id_s);                // dP = dO V^T
        umma_commit(s_full);
        return true;
      };
      // gradients of iteration t
      auto issue_grads = [&](int t) {
        const int it = t / inner, i = t % inner, os = it & 1, st = t & 1;
        if (i == 0 && it > 0 && !mbar_wait(acc_free, (uint32_t)(it - 1) & 1u, abort_flag)) return false;   // the item before has been written
        tc_fence_after();
        const uint32_t own = aOwn + os * 2 * TILE, oth = aOth + st * 2 * TILE;
        if (MODE == BWD_Q) {
          mma_px(tAcc, aD, oth, id_q, i > 0);                         // dQ += dS K
        } else {
          mma_ptx(tAcc, aP, oth + TILE, id_t, i > 0);                 // dV += (P keep)^T dO
          mma_ptx(tAcc + 64, aD, oth, id_t, i > 0);                   // dK += dS^T Q
          if (MODE == BWD_ALL) mma_px(tAcc + 128, aD, own, id_q, false);
        }
        umma_commit(acc_done);
        umma_commit(&oth_empty[st]);
        if (i == inner - 1) umma_commit(&own_empty[os]);
        return true;
      };
      if (total > 0) ok = issue_scores(0);
      for (int t = 0; t < total && ok; ++t) {
        // The next scores are multiplied while the second half of the current ones is worked on: their place is free once those have
        // been read, which is before P and dS are in shared memory.
        if (MODE != BWD_ALL && t + 1 < total) {
          ok = mbar_wait(s_read, (uint32_t)t & 1u, abort_flag);
          if (!ok) break;
          tc_fence_after();
          ok = issue_scores(t + 1);
          if (!ok) break;
        }
        ok = mbar_wait(pd_full, (uint32_t)t & 1u, abort_flag);        // P and dS are in shared memory
        if (!ok) break;
        tc_fence_after();
        ok = issue_grads(t);
        if (MODE == BWD_ALL && ok && t + 1 < total) ok = issue_scores(t + 1);      // an item ends here: its gradients are waited for next
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.error_flag) atomicExch(p.error_flag, 65);
      }
    }
  } else {
    const int q = warp & 3, cb = warp >> 2;                // TMEM lane quarter, block of 32 keys
    const int r = q * 32 + lane;
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    const float inv_keep = inverse_keep(p.drop_p);
    const float scale2 = p.scale * kLog2e, log2_keep = __log2f(inv_keep), delta_scale = p.scale / inv_keep;
    const int words = attn_keep_words(p.S);
    const uint32_t row_smem = (uint32_t)(cb >> 1) * TILE + (uint32_t)r * 128u;
    const uint32_t swz = (uint32_t)(r & 7);
    const uint32_t aP = smem_u32(sP), aD = smem_u32(sD);
    // What an iteration reads from memory is requested one iteration ahead (and not touched before its turn): the row's log sum
    // and delta, the mask of this lane's key and the decision bits of the row's 32 keys.
    struct Row { float lse, delta, mask; uint32_t keep; };
    auto fetch = [&](int item, int i) {
      Row f{INFINITY, 0.f, -INFINITY, 0xffffffffu};        // rows and keys that do not exist: P = 0
      const int ot = own_tile(item), h = head_of(item), b = batch_of(item);
      const int qt = MODE == BWD_Q ? ot : i, kt = MODE == BWD_Q ? i : ot;
      const int row = qt * 128 + r, key = kt * 128 + cb * 32 + lane;
      if (row < p.S) {
        const long long at = ((long long)b * p.heads + h) * p.S + row;
        f.lse = p.lse[at];
        f.delta = p.delta[at];
        if (p.drop_p > 0.f) f.keep = p.keep[at * words + kt * 4 + cb];
      }
      if (key < p.S) f.mask = p.mask != nullptr ? p.mask[(long long)b * p.S + key] : 0.f;
      return f;
    };
    bool ok = true, stored = false;
    int t = 0;
    Row next{INFINITY, 0.f, -INFINITY, 0xffffffffu};
    if ((int)blockIdx.x < items) next = fetch(blockIdx.x, 0);
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int ot = own_tile(item), h = head_of(item), b = batch_of(item);
      for (int i = 0; i < inner; ++i, ++t) {
        const Row now = next;
        if (i + 1 < inner) next = fetch(item, i + 1);
        else if (item + (int)gridDim.x < items) next = fetch(item + gridDim.x, 0);
        // With ps = P / keep probability: P keep = ps where kept, dS = ps * (scale * dP where kept - delta * scale * keep probability).
        // Most blocks of 32 keys carry one mask value; the exponent's argument is then one fused multiply-add.
        const float mask2 = mask_base2(now.mask), mask0 = __shfl_sync(0xffffffffu, mask2, 0);
        const bool plain = __all_sync(0xffffffffu, mask2 == mask0);
        const float row_off = log2_keep - now.lse * kLog2e, nd = -now.delta * delta_scale;
        const float off0 = mask0 + row_off;
        const uint64_t scale2x = both(scale2), scalex = both(p.scale), ndx = both(nd);
        soft_wait(s_full, (uint32_t)t & 1u, abort_flag, ok);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float s[16], d[16];
          __syncwarp();
          tmem_ld16(tS + lane_base + cb * 32 + c * 16, s);
          tmem_ld16(tDP + lane_base + cb * 32 + c * 16, d);
          if (MODE != BWD_ALL && c == 1) {                 // this warp has read its scores
            tc_fence_before();
            __syncwarp();
            if (elect_one()) mbar_arrive(s_read);
          }
          if (plain) {
            const uint64_t off = both(off0);
#pragma unroll
            for (int e = 0; e < 16; e += 2) {
              const float2 arg = unpack_f32x2(fma2(pack_f32x2(s[e], s[e + 1]), scale2x, off));
              s[e] = ex2(arg.x);
              s[e + 1] = ex2(arg.y);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) s[e] = ex2(fmaf(s[e], scale2, __shfl_sync(0xffffffffu, mask2, c * 16 + e) + row_off));
          }
          uint32_t pw[8], dw[8];
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            const float p0 = s[e], p1 = s[e + 1];
            const float2 g = unpack_f32x2(fma2(pack_f32x2(d[e], d[e + 1]), scalex, ndx));
            const bool k0 = (now.keep >> (c * 16 + e)) & 1u, k1 = (now.keep >> (c * 16 + e + 1)) & 1u;
            pw[e / 2] = pack_bf16x2(k0 ? p0 : 0.f, k1 ? p1 : 0.f);
            dw[e / 2] = round2(mul2(pack_f32x2(p0, p1), pack_f32x2(k0 ? g.x : nd, k1 ? g.y : nd)));
          }
          if (c == 0) {
            if (t > 0) soft_wait(acc_done, (uint32_t)(t - 1) & 1u, abort_flag, ok);      // P and dS of the iteration before have been multiplied
            if (stored) {                                  // the last item's gradients have left the staging the next lines write over
              if (elect_one()) bulk_wait_read<0>();
              __syncwarp();
              named_sync(2 + q, 128);                      // the four warps of these rows
              stored = false;
            }
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const uint32_t at = row_smem + (((uint32_t)((cb & 1) * 4 + c * 2 + e) ^ swz) << 4);
            if (MODE != BWD_Q) st_shared_v4(aP + at, pw[4 * e], pw[4 * e + 1], pw[4 * e + 2], pw[4 * e + 3]);
            st_shared_v4(aD + at, dw[4 * e], dw[4 * e + 1], dw[4 * e + 2], dw[4 * e + 3]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (elect_one()) mbar_arrive(pd_full);
      }
      // The item's gradients. Direct stores would write 32-byte pieces of rows 3 * heads * 128 bytes apart; instead warp (q, a) stages 32
      // rows of accumulator a (dV, dK, dQ) in the idle P / dS buffers and hands the box to the TMA unit. Rows past S are clipped.
      soft_wait(acc_done, (uint32_t)(t - 1) & 1u, abort_flag, ok);
      tc_fence_after();
      constexpr int N = MODE == BWD_ALL ? 3 : (MODE == BWD_KV ? 2 : 1);
      if (cb < N) {
        const uint32_t box = (cb < 2 ? aP + cb * TILE : aD) + (uint32_t)(q * 32) * 128u;
        const uint32_t line = box + (uint32_t)lane * 128u;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float v[32];
          __syncwarp();
          tmem_ld32(tAcc + lane_base + cb * 64 + e * 32, v);
#pragma unroll
          for (int x = 0; x < 4; ++x)
            st_shared_v4(line + (((uint32_t)(e * 4 + x) ^ swz) << 4), pack_bf16x2(v[8 * x], v[8 * x + 1]), pack_bf16x2(v[8 * x + 2], v[8 * x + 3]),
                         pack_bf16x2(v[8 * x + 4], v[8 * x + 5]), pack_bf16x2(v[8 * x + 6], v[8 * x + 7]));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (elect_one() && ok) {
          tma_store_4d(&grads.m[MODE == BWD_Q ? 0 : 2 - cb], box, 0, ot * 128 + q * 32, h, b);      // dqkv holds q, k, v
          bulk_commit();
        }
      }
      stored = true;
      tc_fence_before();
      __syncwarp();
      if (elect_one()) mbar_arrive(acc_free);
    }
    if (elect_one()) bulk_wait_read<0>();                    // this warp's copies have left their buffers (the end of the grid waits for them to land)
    if (!ok && lane == 0 && p.error_flag) atomicExch(p.error_flag, 66);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 17) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

template <int MODE>
cudaError_t launch_bwd(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const CUtensorMap& dctx, const AttnGradMaps& grads,
                       const AttnParams& p, int num_sms, cudaStream_t stream) {
  static const cudaError_t configured = cudaFuncSetAttribute(attn_bwd_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM);
  if (configured != cudaSuccess) return configured;
  const long long items = (long long)p.B * p.heads * (MODE == BWD_ALL ? 1 : (p.S + 127) / 128);
  const int grid = (int)(items < num_sms ? items : num_sms);
  return launch_pdl(attn_bwd_kernel<MODE>, dim3(grid), dim3(BWD_THREADS), BWD_SMEM, stream, q, k, v, dctx, grads, p);
}

}  // namespace

cudaError_t launch_attn_fwd(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const AttnParams& p, cudaStream_t stream) {
  if (p.S < 1 || p.S > FWD_MAX_S || p.B < 1 || p.heads < 1 || (p.drop_p > 0.f && (p.keep == nullptr || p.S % 4 != 0)) || !(p.scale > 0.f)) return cudaErrorInvalidValue;
  static const cudaError_t configured = cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM);
  if (configured != cudaSuccess) return configured;
  const long long grid = (long long)p.B * p.heads * ((p.S + 127) / 128);
  if (grid > 0x7fffffffLL) return cudaErrorInvalidValue;
  return launch_pdl(attn_fwd_kernel, dim3((unsigned)grid), dim3(FWD_THREADS), FWD_SMEM, stream, q, k, v, p);
}

cudaError_t launch_attn_bwd(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const CUtensorMap& dctx, const AttnGradMaps& grads,
                            const AttnParams& p, int num_sms, cudaStream_t stream) {
  if (p.S < 1 || p.S > FWD_MAX_S || p.B < 1 || p.heads < 1) return cudaErrorInvalidValue;
  if ((long long)p.B * p.heads * ((p.S + 127) / 128) > 0x3fffffffLL) return cudaErrorInvalidValue;
  if (p.delta == nullptr || (p.drop_p > 0.f && (p.keep == nullptr || p.S % 4 != 0))) return cudaErrorInvalidValue;
  const long long groups = (long long)p.B * p.S * p.heads, blocks = (groups * 8 + 255) / 256;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  const cudaError_t d = launch_pdl(attn_delta_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, p, groups);
  if (d != cudaSuccess) return d;
  if (p.S <= 128) return launch_bwd<BWD_ALL>(q, k, v, dctx, grads, p, num_sms, stream);
  const cudaError_t e = launch_bwd<BWD_KV>(q, k, v, dctx, grads, p, num_sms, stream);
  return e != cudaSuccess ? e : launch_bwd<BWD_Q>(q, k, v, dctx, grads, p, num_sms, stream);
}

}  // namespace adb200
