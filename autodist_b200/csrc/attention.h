// Host-side interface of the fused attention kernels (see attention.cu).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace adb200 {

// Self-attention of [B, S] tokens with `heads` heads of 64 columns. Maps are 4-D bf16 (64 columns, S, heads, B) with boxes of
// (64, 128, 1, 1) and 128-byte swizzle.
struct AttnParams {
  int B, S, heads;
  float scale;                    // of the scores
  const float* mask;              // additive fp32 [B, S] over the keys, or null
  float* lse;                     // fp32 [B, heads, S]: log of the row sums (written by the forward pass, read by the backward)
  float drop_p;                   // dropout of the probabilities (0 = off); decisions as keep_scale8 of (seed, offset in [B, heads, S, S])
  unsigned long long seed;
  const long long* step;          // device step counter mixed into the seed, or null
  uint32_t* keep;                 // with dropout: [B, heads, S, keep_words(S)] decision bits of 32 keys each (forward writes, backward reads)
  float* delta;                   // backward scratch, fp32 [B, heads, S]: row sums of dctx * ctx
  __nv_bfloat16* ctx;             // [B * S, heads * 64]: written by the forward pass, read by the backward
  const __nv_bfloat16* dctx;      // backward: gradient of ctx
  int* error_flag;
};

// Gradients of q, k, v inside dqkv: 4-D bf16 maps (64 columns, S, heads, B) with boxes of (64, 32, 1, 1), 128-byte swizzle.
struct AttnGradMaps {
  CUtensorMap m[3];
};

// Words of decision bits per query row.
constexpr int attn_keep_words(int S) { return (S + 127) / 128 * 4; }

cudaError_t launch_attn_fwd(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const AttnParams& p, cudaStream_t stream);
cudaError_t launch_attn_bwd(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const CUtensorMap& dctx, const AttnGradMaps& grads,
                            const AttnParams& p, int num_sms, cudaStream_t stream);

}  // namespace adb200
