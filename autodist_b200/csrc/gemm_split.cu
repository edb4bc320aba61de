// The tcgen05 GEMM with the contraction split over a thread-block cluster: D[b][M,N] = A[b][M,K] * B[b][N,K]^T for products
// with fewer output tiles than the chip has SMs (weight gradients of small layers, skinny batches, classifier heads).
//
// A cluster of S CTAs owns one output tile; CTA s contracts the K blocks [s * kb / S, (s + 1) * kb / S) into its own TMEM
// accumulator. The partial tiles are then exchanged on the chip: every CTA
// writes its fp32 accumulator over its (now idle) operand ring in shared memory, the cluster synchronises, and each CTA sums
// its 1/S of the tile's rows over the S partial tiles through distributed shared memory, always in the order 0..S-1 (the
// result does not depend on timing), applies the epilogue and stores it. No workspace, no atomics, no zeroing of the output.
//
// Roles as in the one-CTA kernel: warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 drain the accumulator; all ten warps take
// part in the summation. One tile per cluster (the launcher only splits products that leave SMs idle), so there is one
// accumulator and nothing to double-buffer. No multicast loads: each CTA fetches its own tiles.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <array>

#include "gemm_epilogue.cuh"
#include "gemm_tcgen05.h"
#include "pair_tcgen05.cuh"
#include "pdl.cuh"
#include "tcgen05_common.cuh"

namespace adb200 {
namespace {

using namespace tc;

template <int BN> struct SplitCfg {
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 256 ? 4 : (BN == 128 ? 6 : 8);
  static constexpr int TILE = BM * BN * 4;                 // fp32 partial tile, laid over the operand ring
  static constexpr int RING = STAGES * STAGE;
  static constexpr int BODY = RING > TILE ? RING : TILE;
  static constexpr int SMEM = BODY + 1024 /*align*/ + 256 /*barriers*/;
  static constexpr int TMEM_COLS = BN;
};
constexpr int kSplitThreads = 64 + 32 * 8;

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

// S is a template parameter so that the loads of all partial tiles are in flight together.
template <int BN, int S>
__device__ __forceinline__ void reduce_and_store(const GemmParams& p, uint32_t tile, uint32_t rank, int m0, int n0, long long batch_off) {
  const int rows = min(BM, p.M - m0);                        // rows of the tile that exist
  const int r0 = (int)rank * rows / S, r1 = ((int)rank + 1) * rows / S;
  constexpr int CH = BN / 4;                                 // 16-byte chunks per row
  uint32_t peer[S];
#pragma unroll
  for (int s = 0; s < S; ++s) peer[s] = map_to_cta(tile, (uint32_t)s);
#pragma unroll 2
  for (int u = r0 * CH + (int)threadIdx.x; u < r1 * CH; u += kSplitThreads) {
    const int r = u / CH, c = u % CH;
    const uint32_t off = (uint32_t)(r * BN * 4) + (uint32_t)((c ^ (r & 7)) << 4);
    float4 x[S];
#pragma unroll
    for (int s = 0; s < S; ++s) x[s] = ld_cluster_f4(peer[s] + off);
    float v[4] = {x[0].x, x[0].y, x[0].z, x[0].w};
#pragma unroll
    for (int s = 1; s < S; ++s) { v[0] += x[s].x; v[1] += x[s].y; v[2] += x[s].z; v[3] += x[s].w; }
    const int row = m0 + r, col0 = n0 + 4 * c;
    const int ncols = min(4, p.N - col0);
    if (ncols <= 0) continue;
    const bool wide = ncols == 4 && p.vec_ok != 0;
    const long long coff = batch_off + (long long)row * p.ldc;
    gemm_epilogue_math<4>(p, v, col0, ncols, coff, p.vec_ok != 0);
    if (p.c_is_fp32) {
      float* dst = reinterpret_cast<float*>(p.C) + coff + col0;
      if (wide) {
        float4 o = make_float4(v[0], v[1], v[2], v[3]);
        if (p.beta != 0.0f) {
          const float4 old = *reinterpret_cast<const float4*>(dst);
          o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
        }
        *reinterpret_cast<float4*>(dst) = o;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (j < ncols) dst[j] = p.beta != 0.0f ? dst[j] + v[j] : v[j];
      }
    } else {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + coff + col0;
      if (wide) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (j < ncols) dst[j] = __float2bfloat16(v[j]);
      }
      if (p.epilogue == EPI_BIAS_GELU) {
        __nv_bfloat16* dst2 = p.C2 + coff + col0;
        if (wide) {
          *reinterpret_cast<uint2*>(dst2) = make_uint2(pack_bf16x2(gelu_tanh(v[0]), gelu_tanh(v[1])), pack_bf16x2(gelu_tanh(v[2]), gelu_tanh(v[3])));
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) if (j < ncols) dst2[j] = __float2bfloat16(gelu_tanh(v[j]));
        }
      }
    }
  }
}

template <int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p, const int split) {
  using C = SplitCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + C::STAGES * A_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::BODY);
  uint64_t* full = bars;
  uint64_t* empty = bars + C::STAGES;
  uint64_t* tfull = bars + 2 * C::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(tfull, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(C::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_sync();

  const int tiles_m = (p.M + BM - 1) / BM;
  const int tiles_n = (p.N + BN - 1) / BN;
  const int t = (int)(blockIdx.x / (unsigned)split);
  const int b = t / (tiles_m * tiles_n), rem = t % (tiles_m * tiles_n);
  const int tn = rem / tiles_m, tm = rem % tiles_m;
  const int b_lo = b % p.batch_lo, b_hi = b / p.batch_lo;
  const int m0 = tm * BM, n0 = tn * BN;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long long)num_kb * rank / split), kb1 = (int)((long long)num_kb * (rank + 1) / split);

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0; uint32_t phase = 0; bool ok = true; int issued = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) { ok = false; break; }
        ++issued;
        uint8_t* a_dst = sA + stage * A_BYTES;
        uint8_t* b_dst = sB + stage * C::B_BYTES;
        const int k0 = kb * BK;
        mbar_expect_tx(&full[stage], C::STAGE);
        if (A_MN) {
#pragma unroll
          for (int j = 0; j < 2; ++j) tma_load_4d(a_dst + j * (BK * 128), &tmA, &full[stage], m0 + 64 * j, k0, b_lo, b_hi);
        } else {
          tma_load_4d(a_dst, &tmA, &full[stage], k0, m0, b_lo, b_hi);
        }
        if (B_MN) {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_4d(b_dst + j * (BK * 128), &tmB, &full[stage], n0 + 64 * j, k0, b_lo, b_hi);
        } else {
          tma_load_4d(b_dst, &tmB, &full[stage], k0, n0, b_lo, b_hi);
        }
        if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.error_flag) atomicExch(p.error_flag, 51);
      }
      if (*abort_flag) {                                    // copies in flight land before the ring is written over or the CTA leaves
        for (int i = issued > C::STAGES ? issued - C::STAGES : 0; i < issued; ++i) {
          const long long w0 = clock64();
          while (!mbar_try(&full[i % C::STAGES], (uint32_t)(i / C::STAGES) & 1u) && clock64() - w0 < 20000000LL) {}
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc(BN, A_MN, B_MN);
      int stage = 0; uint32_t phase = 0; bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full[stage], phase, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(sA + stage * A_BYTES);
        const uint32_t b_addr = smem_u32(sB + stage * C::B_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint64_t da = A_MN ? make_desc(a_addr + k * (UMMA_K * 128), BK * 128, 1024) : make_desc(a_addr + k * (UMMA_K * 2), 16, 1024);
          const uint64_t db = B_MN ? make_desc(b_addr + k * (UMMA_K * 128), BK * 128, 1024) : make_desc(b_addr + k * (UMMA_K * 2), 16, 1024);
          umma(tmem_base, da, db, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
        }
        umma_commit(&empty[stage]);
        if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) {
        umma_commit(tfull);
      } else {
        *abort_flag = 1;
        if (p.error_flag) atomicExch(p.error_flag, 52);
      }
    }
  } else {
    // every MMA of this CTA has completed when tfull flips, so the operand ring is idle and may be written over
    const int q = warp & 3, hc = (warp - 2) >> 2;
    bool ok = mbar_wait(tfull, 0, abort_flag);
    if (ok) {
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(hc * (BN / 2));
      const int r = q * 32 + lane;
      const uint32_t row_addr = smem_u32(smem) + (uint32_t)(r * BN * 4);
      if (m0 + q * 32 < p.M) {                               // rows past the matrix are never summed
#pragma unroll 2
        for (int c = 0; c < BN / 32; ++c) {
          float v[16];
          __syncwarp();
          tmem_ld16(t_row + c * 16, v);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t ch = (uint32_t)(hc * (BN / 8) + c * 4 + i);
            st_shared_v4(row_addr + ((ch ^ (uint32_t)(r & 7)) << 4), __float_as_uint(v[4 * i]), __float_as_uint(v[4 * i + 1]),
                         __float_as_uint(v[4 * i + 2]), __float_as_uint(v[4 * i + 3]));
          }
        }
      }
    } else if (lane == 0) {
      *abort_flag = 1;
      if (p.error_flag) atomicExch(p.error_flag, 53);
    }
  }

  tc_fence_before();
  __syncthreads();
  __syncwarp();
  cluster_sync_all();                                        // all partial tiles of the cluster are in shared memory
  const uint32_t tile = smem_u32(smem);
  const long long batch_off = (long long)b_hi * p.strideC_hi + (long long)b_lo * p.strideC_lo;
  switch (split) {
    case 2: reduce_and_store<BN, 2>(p, tile, rank, m0, n0, batch_off); break;
    case 3: reduce_and_store<BN, 3>(p, tile, rank, m0, n0, batch_off); break;
    case 4: reduce_and_store<BN, 4>(p, tile, rank, m0, n0, batch_off); break;
    case 5: reduce_and_store<BN, 5>(p, tile, rank, m0, n0, batch_off); break;
    case 6: reduce_and_store<BN, 6>(p, tile, rank, m0, n0, batch_off); break;
    case 7: reduce_and_store<BN, 7>(p, tile, rank, m0, n0, batch_off); break;
    default: reduce_and_store<BN, 8>(p, tile, rank, m0, n0, batch_off);
  }
  __syncwarp();
  cluster_sync_all();                                        // nobody leaves while a peer still reads its partial tile
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::TMEM_COLS) : "memory");
  }
}

template <int BN, bool A_MN, bool B_MN>
cudaError_t configure() {
  static const cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<BN, A_MN, B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitCfg<BN>::SMEM);
  return e;
}

template <int BN, bool A_MN, bool B_MN>
cudaError_t launch_split(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, int split, cudaStream_t stream) {
  const cudaError_t configured = configure<BN, A_MN, B_MN>();
  if (configured != cudaSuccess) return configured;
  const long long tiles = (long long)((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN) * p.batch_lo * p.batch_hi;
  if (tiles <= 0) return cudaSuccess;
  if (tiles * split > 0x7fffffffLL) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * split));
  cfg.blockDim = dim3(kSplitThreads);
  cfg.dynamicSmemBytes = SplitCfg<BN>::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr; cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, gemm_split_kernel<BN, A_MN, B_MN>, tmA, tmB, p, split);
}

template <int BN>
cudaError_t launch_layout(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, int split, bool a_mn, bool b_mn, cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_split<BN, false, false>(tmA, tmB, p, split, stream);
  if (!a_mn && b_mn) return launch_split<BN, false, true>(tmA, tmB, p, split, stream);
  if (a_mn && !b_mn) return launch_split<BN, true, false>(tmA, tmB, p, split, stream);
  return launch_split<BN, true, true>(tmA, tmB, p, split, stream);
}

template <int BN>
int max_clusters(int split, int num_sms) {
  if (configure<BN, false, false>() != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(num_sms / split * split));
  cfg.blockDim = dim3(kSplitThreads);
  cfg.dynamicSmemBytes = SplitCfg<BN>::SMEM;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_split_kernel<BN, false, false>, &cfg) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  return n;
}

}  // namespace

int gemm_split_max_clusters(int split, int num_sms) {
  // one CTA fills an SM at every tile width (192 KB of shared memory), so the count depends on the cluster size alone
  static const std::array<int, 9> counts = [num_sms] {
    std::array<int, 9> c{};
    for (int s = 2; s <= 8; ++s) c[s] = max_clusters<128>(s, num_sms);
    return c;
  }();
  return split >= 2 && split <= 8 ? counts[split] : 0;
}

cudaError_t launch_gemm_split(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, int bn, int split, bool a_mn, bool b_mn,
                              cudaStream_t stream) {
  if (p.b_shard_rows > 0 || p.epilogue == EPI_SOFTMAX || p.epilogue == EPI_SOFTMAX_GRAD) return cudaErrorInvalidValue;
  if (split < 2 || split > 8 || split > (p.K + BK - 1) / BK) return cudaErrorInvalidValue;
  if (bn == 256) return launch_layout<256>(tmA, tmB, p, split, a_mn, b_mn, stream);
  if (bn == 128) return launch_layout<128>(tmA, tmB, p, split, a_mn, b_mn, stream);
  if (bn == 64) return launch_layout<64>(tmA, tmB, p, split, a_mn, b_mn, stream);
  return cudaErrorInvalidValue;
}

}  // namespace adb200
