// 2-D convolution as an implicit GEMM on the 5th-generation tensor cores (sm_100a): forward, input gradient and
// weight gradient over channels-last bf16 activations, no im2col matrix in memory.
//
// Same persistent, warp-specialised shape as the GEMM (gemm_tcgen05.cu):
//   warps 0, 10 TMA producers per K block one box of the activation patch shifted by the filter tap (zero fill outside
//                            the image = the padding) and one box of the weight, 128-byte swizzle, ring of stages
//   warp 1    MMA issuer     tcgen05.mma 128 x BN x 16, bf16 -> fp32 in TMEM, two accumulator buffers
//   warps 2-9 epilogue       tcgen05.ld, then
//                              forward:         + bias, evaluation-mode batch-norm, residual, ReLU, per-channel sum / sum of
//                                               squares (batch-norm statistics, reduced in shared memory across the
//                                               CTA's tiles), bf16 store
//                              input gradient:  bf16 store (strided positions for a strided convolution)
//                              weight gradient: fp32 store or vector atomic add (split-K)
//
// M rows of a forward / input-gradient tile are a patch of pixels (tw x th x tn <= 128) so that one 4-D box covers all of
// them for any tap; the weight gradient contracts over 64-pixel patches with both operands MN-major.
//
// Every mbarrier wait is bounded; a wait that gives up sets `error_flag`, the CTA lets its copies land, frees its
// TMEM and returns.
//
// The reference's convolutions are tf.keras layers running in cuDNN (examples/benchmark/imagenet.py:232-249).
#include <type_traits>

#include "conv_tcgen05.h"
#include "eval_norm.cuh"
#include "pdl.cuh"
#include "tcgen05_common.cuh"

namespace adb200 {
namespace {

using namespace tc;

template <int BN, int MODE> struct ConvCfg {
  static constexpr int B_BYTES = BN * BK * 2;
  // Pixel modes keep two output boxes (128 pixels x 64 channels, 16 KB) per half of the epilogue warps; 64-wide tiles share them.
  static constexpr int STAGING = (MODE == CONV_WGRAD) ? 0 : (BN == 64 ? 2 : 4) * A_BYTES;
  static constexpr int STAGES = (MODE == CONV_WGRAD) ? (BN == 256 ? 4 : (BN == 128 ? 6 : 8)) : (BN == 256 ? 3 : (BN == 128 ? 4 : 7));
  static constexpr int TMEM_COLS = 2 * BN;
  // Eight epilogue warps: two per TMEM lane quarter, half of the tile's columns each. Layers with a short contraction
  // (1 x 1 convolutions) spend longer draining a tile than multiplying it, and four warps could not keep up.
  static constexpr int EPI_WARPS = 8;
  static constexpr int THREADS = 96 + 32 * EPI_WARPS;           // two producer warps, the MMA issuer, the epilogue
  static constexpr int CHUNKS = BN / 16 / (EPI_WARPS / 4);      // 16-column chunks per epilogue warp
  static constexpr int STAT_BYTES = (MODE == CONV_FPROP || MODE == CONV_EVAL) ? 2 * kMaxStatChannels * 4 : 0;
  static constexpr int SMEM = STAGES * (A_BYTES + B_BYTES) + STAGING + 1024 /*align*/ + 256 /*barriers*/ + STAT_BYTES;
};

struct TileCoord {
  int w0, h0, n0;       // patch origin in the pixel grid
  int c0;               // first column of the GEMM N extent
  int m0;               // weight gradient: first output channel
  int tap;              // weight gradient: tap of this tile
  int kbeg, kend;       // weight gradient: patch range of this tile
};

template <int BN, int MODE>
__device__ __forceinline__ TileCoord decode_tile(const ConvParams& p, long long t) {
  TileCoord c;
  if (MODE != CONV_WGRAD) {
    const int m_tiles = p.tiles_w * p.tiles_h * p.tiles_n;
    const int ct = (int)(t / m_tiles), m = (int)(t % m_tiles);
    c.w0 = (m % p.tiles_w) * p.tw;
    c.h0 = ((m / p.tiles_w) % p.tiles_h) * p.th;
    c.n0 = (m / (p.tiles_w * p.tiles_h)) * p.tn;
    c.c0 = ct * BN;
    c.m0 = 0; c.tap = 0; c.kbeg = 0; c.kend = 0;
  } else {
    const int m_tiles = (p.Mc + BM - 1) / BM, c_tiles = (p.Nc + BN - 1) / BN;
    long long r = t;
    c.m0 = (int)(r % m_tiles) * BM; r /= m_tiles;
    c.c0 = (int)(r % c_tiles) * BN; r /= c_tiles;
    c.tap = (int)(r % p.ntaps);
    const int ks = (int)(r / p.ntaps);
    const long long P = (long long)p.tiles_w * p.tiles_h * p.tiles_n;
    c.kbeg = (int)(P * ks / p.ksplit);
    c.kend = (int)(P * (ks + 1) / p.ksplit);
    c.w0 = c.h0 = c.n0 = 0;
  }
  return c;
}

__device__ __forceinline__ long long total_tiles(const ConvParams& p, int bn, int mode) {
  const int c_tiles = (p.Nc + bn - 1) / bn;
  if (mode != CONV_WGRAD) return (long long)p.tiles_w * p.tiles_h * p.tiles_n * c_tiles;
  return (long long)((p.Mc + BM - 1) / BM) * c_tiles * p.ntaps * p.ksplit;
}

// Sum of v[0..15] over the 32 lanes of a warp, column j ends up in the lanes whose bits 4..1 spell j (both lanes of a
// pair hold it). 16 shuffles instead of 80: every step halves the columns a lane is responsible for.
__device__ __forceinline__ float warp_column_sums16(float* v, int lane) {
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int half = 8 >> s;
    const bool upper = (lane & (16 >> s)) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = upper ? v[i] : v[i + half];
      const float keep = upper ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16 >> s);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

__device__ __forceinline__ void store_box(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void sts4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint4 lds4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
// Evaluation mode, 32 rows x 32 columns of one warp: bias, batch-norm, residual, ReLU, rounded to bf16 wherever layers of their own would
// round (see eval_norm.cuh). A thread that owns a row needs the four coefficients of every column, 128 floats per 32 outputs, and the
// shared-memory reads of those bounded the drain; so the accumulator is read in the fragment layout: lane l holds columns
// 8 k + 2 (l % 4), + 1 of the rows l / 4 + 8 i, and a column's coefficients serve four rows (one ResNet-50 evaluation pass of 32 images:
// a row per thread 1285 us, this 1133).
// `tab`: the columns' coefficients, BN floats between two of them; `rows`: shared address of the warp's 32 staged lines.
template <int BN>
__device__ __forceinline__ void eval_piece(uint32_t taddr, int cols, const float* tab, bool bias, bool add, bool relu, uint32_t rows, int chunk, int lane) {
  uint32_t r[32];
  __syncwarp();
  tmem_ld_frag32(taddr, r);
  const uint32_t swz = (uint32_t)(lane >> 2);  // line % 8 of every row of this lane
  const uint32_t mine = rows + (uint32_t)(lane >> 2) * 128u + (uint32_t)(lane & 3) * 4u;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (8 * k >= cols) break;                  // columns come in groups of 8
    const float* t = tab + 8 * k + 2 * (lane & 3);
    const uint64_t neg_mean = *reinterpret_cast<const uint64_t*>(t), inv = *reinterpret_cast<const uint64_t*>(t + BN);
    const uint64_t gamma = *reinterpret_cast<const uint64_t*>(t + 2 * BN), beta = *reinterpret_cast<const uint64_t*>(t + 3 * BN);
    const uint64_t b = bias ? *reinterpret_cast<const uint64_t*>(t + 4 * BN) : 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t* a = r + (i >> 1) * 16 + k * 4 + (i & 1) * 2;
      const uint32_t at = mine + (uint32_t)i * 1024u + (((uint32_t)(chunk + k) ^ swz) << 4);
      uint64_t v = pack_f32x2(__uint_as_float(a[0]), __uint_as_float(a[1]));
      if (bias) v = add2(v, b);
      v = widen2(round2(v));                                                    // the convolution's result
      uint32_t w = round2(fma2(mul2(gamma, add2(v, neg_mean)), inv, beta));     // normalised (eval_norm)
      if (add) w = round2(add2(widen2(w), widen2(lds1(at))));
      if (relu) asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(w) : "r"(w), "r"(0u));  // a NaN stays a NaN
      sts1(at, w);
    }
  }
}

// Epilogue of the pixel modes through shared memory. A 1 x 1 convolution multiplies a tile in a few microseconds, so the drain is
// what bounds it: direct stores wrote 32 rows in 16-byte pieces per instruction, and the batch-norm sums took 34 shuffles per
// 16 columns. Here the warps stage boxes of 128 pixels x 64 channels in the 128-byte-swizzled layout (row = pixel of the patch, the
// order of the input boxes), one thread per half hands a box to the TMA unit, and the sums are taken from the staged
// bf16 values: lane l adds channels 2l, 2l + 1 over its warp's 32 rows, 32 conflict-free reads per 64 channels. The addend (residual or
// fork gradient) comes by TMA into the box ahead of the accumulator and is replaced by the result.
// 64 images, 1 x 1, with sums (without the staging -> now, us): 64 -> 256 channels at 56 x 56 91 -> 34, 128 -> 512 at 28 x 28
// 52 -> 21.5, 256 -> 1024 at 14 x 14 29 -> 16; input gradient with addend: to 256 channels at 56 x 56 66 -> 44, to 512 at
// 28 x 28 39 -> 28, to 1024 at 14 x 14 21 -> 13. The staging takes one to two of the operand stages; the 3 x 3 layers, which those
// feed, did not slow down (256 -> 256 at 14 x 14: 19.5 -> 18.4).
// Warps: TMEM lane quarter q = warp % 4, half hf: columns [hf * BN / 2, (hf + 1) * BN / 2). BN 256: two boxes per half; 128: one;
// 64: both halves share a box. Box buffers alternate; they are free again once the issuing thread has seen its copies read.
template <int BN, int MODE>
__device__ __forceinline__ bool staged_epilogue(const ConvParams& p, const ConvMaps& maps, long long total, uint32_t tmem_base, uint64_t* tfull,
                                                uint64_t* tempty, uint64_t* add_bars, uint32_t staging, float* s_stat, bool do_stats,
                                                volatile int* abort_flag, long long* trace) {
  constexpr bool EVAL = MODE == CONV_EVAL, FWD = MODE != CONV_DGRAD;
  constexpr int CW = BN / 2;                           // columns of this warp
  constexpr int BOXES = BN == 256 ? 2 : 1;             // boxes it takes part in per tile
  constexpr int PARTY = BN == 64 ? 256 : 128;          // threads that fill a box together
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int q = warp & 3, hf = (warp - 2) >> 2;
  const int r = q * 32 + lane;
  const int rows = p.tw * p.th * p.tn;
  const bool issuing = BN == 64 ? warp == 2 : (warp - 2) % 4 == 0;   // its elected lane issues the copies
  const int bar_id = BN == 64 ? 2 : 2 + hf;
  const uint32_t boxes = staging + (BN == 64 ? 0u : (uint32_t)hf * 2u * A_BYTES);       // two buffers
  uint64_t* abar = add_bars + (BN == 64 ? 0 : 2 * hf);
  const uint32_t swz = (uint32_t)(r & 7);
  const bool add = (MODE == CONV_DGRAD || EVAL) && p.addend != nullptr;
  const bool bias = FWD && p.bias != nullptr;
  auto meet = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "n"(PARTY) : "memory"); };
  // Evaluation-mode batch-norm: the coefficients of the tile's columns (-mean, 1 / deviation, gamma, beta and the convolution's bias,
  // BN floats each, in the statistics table's space - the two never occur together) are rebuilt when the columns change, while the
  // tile is multiplied.
  int norm_c0 = -1;
  bool ok = true;
  auto wait = [&](uint64_t* bar, uint32_t parity) {    // a warp that gives up walks on, so that nobody is left behind at a barrier
    if (ok && !mbar_wait(bar, parity, abort_flag)) { ok = false; *abort_flag = 1; }
  };
  int as = 0; uint32_t aphase = 0;
  uint32_t use[2] = {0, 0};                            // how often each buffer received an addend
  // Batch-norm sums of this lane's two channels per box (sum, sum, squares, squares), kept in registers while the tiles of this
  // CTA cover the same channels: atomics on shared memory per tile cost as much as the drain.
  float acc[BOXES][4];
  int acc_c0 = -1;
  auto flush = [&]() {
    if (acc_c0 < 0) return;
#pragma unroll
    for (int g = 0; g < BOXES; ++g) {
      const int c = (BN == 64 ? acc_c0 : acc_c0 + hf * CW) + 64 * g + 2 * lane;
      if (c < p.Nc) {
        atomicAdd(&s_stat[c], acc[g][0]);
        atomicAdd(&s_stat[c + 1], acc[g][1]);
        atomicAdd(&s_stat[p.Nc + c], acc[g][2]);
        atomicAdd(&s_stat[p.Nc + c + 1], acc[g][3]);
      }
    }
  };
  int buf = 0;
  for (long long t = blockIdx.x; t < total; t += gridDim.x) {
    const TileCoord tc_ = decode_tile<BN, MODE>(p, t);
    const int c_w = tc_.c0 + hf * CW;                  // first column of this warp
    const int c_box = BN == 64 ? tc_.c0 : c_w;         // first column of its first box
    const long long tw0 = trace != nullptr ? clock64() : 0;
    if (issuing && elect_one()) {
      store_wait_read();                               // the copies of the tile before have left the buffers
      if (add) {
#pragma unroll
        for (int g = 0; g < BOXES; ++g) {
          const int bb = BOXES == 2 ? g : buf;
          if (c_box + 64 * g >= p.Nc) continue;
          mbar_expect_tx(&abar[bb], (uint32_t)rows * 128u);
          asm volatile(
              "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
              ::"r"(boxes + (uint32_t)bb * A_BYTES), "l"(&maps.add), "r"(smem_u32(&abar[bb])), "r"(c_box + 64 * g), "r"(tc_.w0), "r"(tc_.h0), "r"(tc_.n0)
              : "memory");
        }
      }
    }
    float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);       // four columns of the bias per lane, handed around by shuffles
    if (!EVAL && bias && lane * 4 < CW) {
      const int c = c_w + lane * 4;                    // Nc is a multiple of 8: four columns exist together
      if (c < p.Nc) b4 = make_float4(__ldg(p.bias + c), __ldg(p.bias + c + 1), __ldg(p.bias + c + 2), __ldg(p.bias + c + 3));
    }
    bool valid = true;
    if (do_stats) {
      const int gw = tc_.w0 + r % p.tw, gh = tc_.h0 + (r / p.tw) % p.th, gn = tc_.n0 + r / (p.tw * p.th);
      valid = r < rows && gw < p.GW && gh < p.GH && gn < p.GN;
    }
    bool table = false;
    if constexpr (EVAL) {
      // nobody reads the old table any more: the party met after its last box
      table = tc_.c0 != norm_c0;
      norm_c0 = tc_.c0;
      if (table) {
        constexpr int COLS = BN == 64 ? BN : CW;       // columns of this party
        const int t0 = BN == 64 ? 0 : hf * CW;
        for (int c = (int)threadIdx.x - 64 - (BN == 64 ? 0 : hf * 128); c < COLS; c += PARTY)
          if (tc_.c0 + t0 + c < p.Nc) {
            const int ch = tc_.c0 + t0 + c;
            const float4 n = eval_norm_of(p.bn_mean, p.bn_var, p.bn_gamma, p.bn_beta, p.bn_eps, ch);
            float* at = s_stat + t0 + c;
            at[0] = -n.x; at[BN] = n.y; at[2 * BN] = n.z; at[3 * BN] = n.w;
            at[4 * BN] = bias ? p.bias[ch] : 0.f;
          }
      }
    }
    if (!add || table) meet();                         // with an addend its arrival says that the buffer may be written
    wait(&tfull[as], aphase);
    const long long tw1 = trace != nullptr ? clock64() : 0;
    tc_fence_after();
    const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * BN + hf * CW);
    if (MODE == CONV_FPROP && do_stats && tc_.c0 != acc_c0) {
      flush();
      acc_c0 = tc_.c0;
#pragma unroll
      for (int g = 0; g < BOXES; ++g) acc[g][0] = acc[g][1] = acc[g][2] = acc[g][3] = 0.f;
    }
    bool released = false;
#pragma unroll
    for (int g = 0; g < BOXES; ++g) {
      const int bb = BOXES == 2 ? g : buf;
      const int col0 = c_w + 64 * g;                   // first column of this warp in the box
      if (c_box + 64 * g >= p.Nc) break;               // uniform over the party
      const uint32_t box = boxes + (uint32_t)bb * A_BYTES;
      const uint32_t line = box + (uint32_t)r * 128u;
      if (add) wait(&abar[bb], use[bb] & 1u);
      if (add) ++use[bb];
#pragma unroll
      for (int h = 0; h < CW / 32 / BOXES; ++h) {
        const int ch = (BN == 64 ? hf * 4 : h * 4);    // first 16-byte chunk of the 32 columns inside the box line
        if constexpr (EVAL) {
          eval_piece<BN>(t_row + g * 64 + h * 32, p.Nc - (col0 + h * 32), s_stat + hf * CW + g * 64 + h * 32, bias, add, p.relu != 0,
                         box + (uint32_t)(q * 32) * 128u, ch, lane);
          continue;
        }
        float v[32];
        __syncwarp();
        tmem_ld32(t_row + g * 64 + h * 32, v);
        if (bias) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const int src = (g * 64 + h * 32 + j) >> 2;
            v[j] += __shfl_sync(0xffffffffu, b4.x, src);
            v[j + 1] += __shfl_sync(0xffffffffu, b4.y, src);
            v[j + 2] += __shfl_sync(0xffffffffu, b4.z, src);
            v[j + 3] += __shfl_sync(0xffffffffu, b4.w, src);
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t at = line + (((uint32_t)(ch + j) ^ swz) << 4);
          float* w = v + 8 * j;
          if (add) {
            float a[8];
            unpack8_bf16(lds4(at), a);
#pragma unroll
            for (int x = 0; x < 8; ++x) w[x] += a[x];
          }
          if (FWD && p.relu) {
#pragma unroll
            for (int x = 0; x < 8; ++x) w[x] = fmaxf(w[x], 0.f);
          }
          if (do_stats && !valid) {                    // pixels that do not exist count for nothing
#pragma unroll
            for (int x = 0; x < 8; ++x) w[x] = 0.f;
          }
          sts4(at, pack2(w[0], w[1]), pack2(w[2], w[3]), pack2(w[4], w[5]), pack2(w[6], w[7]));
        }
      }
      if (g == BOXES - 1) {                            // the accumulator has been read
        tc_fence_before();
        mbar_arrive(&tempty[as]);
        released = true;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      meet();
      if (issuing && elect_one() && ok) store_box(&maps.out, box, c_box + 64 * g, tc_.w0, tc_.h0, tc_.n0);
      if constexpr (MODE == CONV_FPROP) {
        if (do_stats) {
          // statistics of what the next layer reads: the staged bf16 values. 64-wide tiles: each half takes 16 of the quarter's rows.
          constexpr int NR = BN == 64 ? 16 : 32;
          const uint32_t base = box + (uint32_t)(q * 32 + (BN == 64 ? hf * 16 : 0)) * 128u;
#pragma unroll
          for (int i = 0; i < NR; ++i) {
            const uint32_t u = lds1(base + (uint32_t)i * 128u + ((((uint32_t)(lane >> 2)) ^ (uint32_t)(i & 7)) << 4) + (uint32_t)(lane & 3) * 4u);
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
            acc[g][0] += f.x; acc[g][1] += f.y;
            acc[g][2] = fmaf(f.x, f.x, acc[g][2]); acc[g][3] = fmaf(f.y, f.y, acc[g][3]);
          }
        }
      }
    }
    if (!released) {                                   // this warp's last columns lie past the matrix
      tc_fence_before();
      mbar_arrive(&tempty[as]);
    }
    if (trace != nullptr && threadIdx.x == 64) { trace[5] += clock64() - tw1; trace[6] += tw1 - tw0; }
    if (BOXES == 1) buf ^= 1;
    if (++as == 2) { as = 0; aphase ^= 1; }
  }
  if (MODE == CONV_FPROP && do_stats) flush();
  if (issuing && elect_one()) {
    store_wait_read();                                 // this thread's copies have left the buffers (the end of the grid waits for them to land)
    for (int b = 0; add && !ok && b < 2; ++b) {        // addends nobody waited for land before the CTA leaves
      const long long w0 = clock64();
      while (!mbar_try(&abar[b], use[b] & 1u) && clock64() - w0 < 2000000LL) {}
    }
  }
  return ok;
}

template <int BN, int MODE>
__global__ void __launch_bounds__(ConvCfg<BN, MODE>::THREADS, 1)
conv_kernel(const __grid_constant__ ConvMaps maps, const __grid_constant__ ConvParams p) {
  using C = ConvCfg<BN, MODE>;
  constexpr bool A_MN = MODE == CONV_WGRAD;
  constexpr bool FWD = MODE == CONV_FPROP || MODE == CONV_EVAL;
  constexpr bool EVAL = MODE == CONV_EVAL;
  constexpr bool B_MN = !FWD;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + C::STAGES * A_BYTES;
  uint8_t* staging = smem + C::STAGES * (A_BYTES + C::B_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + C::STAGING);
  uint64_t* full = bars;
  uint64_t* empty = bars + C::STAGES;
  uint64_t* tfull = bars + 2 * C::STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* add_bars = tempty + 3;                 // pixel modes: two per half of the epilogue warps (behind the slot and the flag)
  float* s_stat = reinterpret_cast<float*>(staging + C::STAGING + 256);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const bool do_stats = (MODE == CONV_FPROP) && p.stats != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&tfull[s], 1); mbar_init(&tempty[s], 32 * C::EPI_WARPS); }
    for (int s = 0; s < 4; ++s) mbar_init(&add_bars[s], 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (MODE == CONV_FPROP) {
    if (do_stats) for (int i = threadIdx.x; i < 2 * p.Nc; i += C::THREADS) s_stat[i] = 0.f;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(C::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_sync();       // everything above touched only this CTA's shared and tensor memory; global memory is read from here on

  // trace (when given): 0 start, 1 first load issued, 2 last load issued, 3 first stage full, 4 last MMA committed,
  // 5 cycles the first epilogue warp spent between "accumulator full" and "accumulator released" (summed over tiles),
  // 6 cycles it waited for full accumulators, 7 end
  long long* trace = p.trace != nullptr ? p.trace + (long long)blockIdx.x * 8 : nullptr;
  if (trace != nullptr && threadIdx.x == 0) trace[0] = clock64();
  const long long total = total_tiles(p, BN, MODE);
  const int kcb = (p.Kc + BK - 1) / BK;
  const int rows = p.tw * p.th * p.tn;
  const int col_rows = p.th * p.tn;                 // rows of one patch column (wsplit boxes)

  // One operand per producer warp (A and the byte count: the first warp, B: the last). A K block takes one to six copies, and a
  // single thread that issued all of them bounded every narrow or MN-major tile. Weight gradients of 3 x 3 layers, 32 images (one
  // producer that divided per patch / without the divisions / two producers, us): 64 -> 64 at 224 x 224 602 / 462 / 467,
  // 128 -> 128 at 112 x 112 200 / 157 / 127, 256 -> 256 at 56 x 56 125 / 103 / 90.
  auto produce = [&](auto operand) {
    constexpr bool LOAD_A = decltype(operand)::value == 0, LOAD_B = !LOAD_A;
    {
      int stage = 0; uint32_t phase = 0; bool ok = true;
      if (LOAD_A && trace != nullptr) trace[1] = clock64();
      for (long long t = blockIdx.x; t < total && ok; t += gridDim.x) {
        const TileCoord tc_ = decode_tile<BN, MODE>(p, t);
        if (MODE != CONV_WGRAD) {
          const uint32_t a_bytes = (uint32_t)rows * 128u;
          for (int tp = 0; tp < p.ntaps && ok; ++tp) {
            const ConvTap tap = p.taps[tp];
            const CUtensorMap* mapA = &maps.act[tap.amap];
            for (int cb = 0; cb < kcb; ++cb) {
              if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) { ok = false; break; }
              if (LOAD_A) mbar_expect_tx(&full[stage], a_bytes + C::B_BYTES);
              uint8_t* a_dst = sA + stage * A_BYTES;
              uint8_t* b_dst = sB + stage * C::B_BYTES;
              if (LOAD_B) {
              } else if (!p.wsplit) {
                tma_load_4d(a_dst, mapA, &full[stage], cb * BK, tc_.w0 + tap.dw, tc_.h0 + tap.dh, tc_.n0);
              } else {
                for (int j = 0; j < p.tw; ++j)
                  tma_load_4d(a_dst + j * col_rows * 128, mapA, &full[stage], (tc_.w0 + j) * p.xstep, tc_.h0 + tap.dh, tc_.n0, 0);
              }
              if (LOAD_A) {
              } else if (FWD) {
                tma_load_4d(b_dst, &maps.w, &full[stage], cb * BK, tap.wtap, tc_.c0, 0);
              } else {
#pragma unroll
                for (int j = 0; j < BN / 64; ++j)
                  tma_load_4d(b_dst + j * (BK * 128), &maps.w, &full[stage], tc_.c0 + 64 * j, tap.wtap, cb * BK, 0);
              }
              if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
            }
          }
        } else {
          const ConvTap tap = p.taps[tc_.tap];
          const CUtensorMap* mapX = &maps.act[tap.amap];
          // the patch walks on by additions: divisions per patch made this one thread the bound of narrow tiles
          int w0 = (tc_.kbeg % p.tiles_w) * p.tw;
          int h0 = ((tc_.kbeg / p.tiles_w) % p.tiles_h) * p.th;
          int n0 = (tc_.kbeg / (p.tiles_w * p.tiles_h)) * p.tn;
          const int w_end = p.tiles_w * p.tw, h_end = p.tiles_h * p.th;
          auto next_patch = [&]() {
            w0 += p.tw;
            if (w0 >= w_end) { w0 = 0; h0 += p.th; if (h0 >= h_end) { h0 = 0; n0 += p.tn; } }
          };
          for (int pi = tc_.kbeg; pi < tc_.kend; ++pi, next_patch()) {
            if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) { ok = false; break; }
            // output channels beyond Cout need no load: those accumulator rows are never stored
            const int a_chunks = (tc_.m0 + 64 < p.Mc) ? 2 : 1;
            if (LOAD_A) mbar_expect_tx(&full[stage], a_chunks * (BK * 128) + C::B_BYTES);
            uint8_t* a_dst = sA + stage * A_BYTES;
            uint8_t* b_dst = sB + stage * C::B_BYTES;
            if (!p.wsplit) {
              for (int j = 0; LOAD_A && j < a_chunks; ++j) tma_load_4d(a_dst + j * (BK * 128), &maps.dy, &full[stage], tc_.m0 + 64 * j, w0, h0, n0);
#pragma unroll
              for (int j = 0; LOAD_B && j < BN / 64; ++j)
                tma_load_4d(b_dst + j * (BK * 128), mapX, &full[stage], tc_.c0 + 64 * j, w0 + tap.dw, h0 + tap.dh, n0);
            } else {
              for (int jw = 0; jw < p.tw; ++jw) {
                for (int j = 0; LOAD_A && j < a_chunks; ++j)
                  tma_load_4d(a_dst + j * (BK * 128) + jw * col_rows * 128, &maps.dy, &full[stage], tc_.m0 + 64 * j, w0 + jw, h0, n0);
                if (LOAD_B) tma_load_4d(b_dst + jw * col_rows * 128, mapX, &full[stage], (w0 + jw) * p.xstep, h0 + tap.dh, n0, 0);
              }
            }
            if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
          }
        }
      }
      if (LOAD_A && trace != nullptr) trace[2] = clock64();
      if (!ok) {
        *abort_flag = 1;
        if (p.error_flag) atomicExch(p.error_flag, 11);
      }
      if (*abort_flag) {
        for (int s = 0; s < C::STAGES; ++s) {
          const long long t0 = clock64();
          while (!mbar_try(&full[s], 0) && !mbar_try(&full[s], 1) && clock64() - t0 < 20000000LL) {}
        }
      }
    }
  };
  if (warp == 0) {
    if (elect_one()) produce(std::integral_constant<int, 0>{});
  } else if (warp == 2 + C::EPI_WARPS) {
    if (elect_one()) produce(std::integral_constant<int, 1>{});
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc(BN, A_MN, B_MN);
      int stage = 0; uint32_t phase = 0; int as = 0; uint32_t aphase = 0; bool ok = true;
      for (long long t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int num_kb;
        if (MODE != CONV_WGRAD) {
          num_kb = p.ntaps * kcb;
        } else {
          const TileCoord tc_ = decode_tile<BN, MODE>(p, t);
          num_kb = tc_.kend - tc_.kbeg;
        }
        if (num_kb <= 0) continue;
        if (!mbar_wait(&tempty[as], aphase ^ 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(as * BN);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&full[stage], phase, abort_flag)) { ok = false; break; }
          if (trace != nullptr && t == blockIdx.x && kb == 0) trace[3] = clock64();
          tc_fence_after();
          const uint32_t a_addr = smem_u32(sA + stage * A_BYTES);
          const uint32_t b_addr = smem_u32(sB + stage * C::B_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t da = A_MN ? make_desc(a_addr + k * (UMMA_K * 128), BK * 128, 1024)
                                     : make_desc(a_addr + k * (UMMA_K * 2), 16, 1024);
            const uint64_t db = B_MN ? make_desc(b_addr + k * (UMMA_K * 128), BK * 128, 1024)
                                     : make_desc(b_addr + k * (UMMA_K * 2), 16, 1024);
            umma(d_tmem, da, db, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(&empty[stage]);
          if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(&tfull[as]);
        if (trace != nullptr) trace[4] = clock64();
        if (++as == 2) { as = 0; aphase ^= 1; }
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.error_flag) atomicExch(p.error_flag, 12);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5 -> TMEM lane quarter warp % 4)
    const int q = warp & 3;
    const int c_lo = ((warp - 2) >> 2) * C::CHUNKS;      // first 16-column chunk of this warp's share of the tile
    int as = 0; uint32_t aphase = 0; bool ok = true;
    const int r = q * 32 + lane;
    // bias and evaluation-mode batch-norm of 16 forward outputs starting at column col0
    auto affine16 = [&](float* v, int col0) {
      if (p.bias != nullptr) {
#pragma unroll
        for (int jj = 0; jj < 16; ++jj) if (col0 + jj < p.Nc) v[jj] += __ldg(p.bias + col0 + jj);
      }
      if (EVAL) {
#pragma unroll
        for (int jj = 0; jj < 16; ++jj)
          if (col0 + jj < p.Nc)
            v[jj] = round_bf16(eval_norm(round_bf16(v[jj]), eval_norm_of(p.bn_mean, p.bn_var, p.bn_gamma, p.bn_beta, p.bn_eps, col0 + jj)));
      }
    };
    bool staged = false;
    if constexpr (MODE != CONV_WGRAD) {
      staged = p.staged != 0;
      if (staged) ok = staged_epilogue<BN, MODE>(p, maps, total, tmem_base, tfull, tempty, add_bars, smem_u32(staging), s_stat, do_stats, abort_flag, trace);
    }
    if constexpr (MODE != CONV_DGRAD)                    // the input gradient is always staged (see launch_conv)
    for (long long t = blockIdx.x; t < total && ok && !staged; t += gridDim.x) {
      const TileCoord tc_ = decode_tile<BN, MODE>(p, t);
      if (MODE == CONV_WGRAD && tc_.kend <= tc_.kbeg) continue;
      bool valid;
      long long off;
      if (MODE != CONV_WGRAD) {
        int j, i, nn;
        if (!p.wsplit) { j = r % p.tw; i = (r / p.tw) % p.th; nn = r / (p.tw * p.th); }
        else { j = r / col_rows; const int rem = r % col_rows; i = rem % p.th; nn = rem / p.th; }
        const int gw = tc_.w0 + j, gh = tc_.h0 + i, gn = tc_.n0 + nn;
        valid = r < rows && gw < p.GW && gh < p.GH && gn < p.GN;
        off = (((long long)gn * p.OH + (long long)gh * p.os + p.oh0) * p.OW + (long long)gw * p.os + p.ow0) * p.ldc;
      } else {
        const int row = tc_.m0 + r;
        valid = row < p.Mc;
        off = (long long)row * p.ldc + (long long)p.taps[tc_.tap].wtap * p.wtap_stride;
      }
      const long long tw0 = trace != nullptr ? clock64() : 0;
      if (!mbar_wait(&tfull[as], aphase, abort_flag)) { ok = false; break; }
      const long long tw1 = trace != nullptr ? clock64() : 0;
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * BN);
#pragma unroll 1
      for (int c = c_lo; c < c_lo + C::CHUNKS; ++c) {
        const int col0 = tc_.c0 + c * 16;
        if (col0 >= p.Nc) break;                 // uniform over the warp
        float v[16];
        __syncwarp();
        tmem_ld16(t_row + c * 16, v);
        const int ncols = valid ? min(16, p.Nc - col0) : 0;
        if (MODE == CONV_WGRAD) {
          if (ncols > 0) {
            float* dst = reinterpret_cast<float*>(p.out) + off + col0;
            const bool vec = ncols == 16 && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0);
            if (p.accumulate) {
              if (vec) {
#pragma unroll
                for (int jj = 0; jj < 16; jj += 4) atomicAdd(reinterpret_cast<float4*>(dst + jj), make_float4(v[jj], v[jj + 1], v[jj + 2], v[jj + 3]));
              } else {
#pragma unroll
                for (int jj = 0; jj < 16; ++jj) if (jj < ncols) atomicAdd(dst + jj, v[jj]);
              }
            } else if (vec) {
#pragma unroll
              for (int jj = 0; jj < 16; jj += 4) *reinterpret_cast<float4*>(dst + jj) = make_float4(v[jj], v[jj + 1], v[jj + 2], v[jj + 3]);
            } else {
#pragma unroll
              for (int jj = 0; jj < 16; ++jj) if (jj < ncols) dst[jj] = v[jj];
            }
          }
        } else {
          if (FWD) {
            affine16(v, col0);
            if (EVAL && p.addend != nullptr) {
#pragma unroll
              for (int jj = 0; jj < 16; ++jj) if (jj < ncols) v[jj] += __bfloat162float(p.addend[off + col0 + jj]);
            }
            if (p.relu && EVAL) {                  // like the library's evaluation path: a NaN stays a NaN
#pragma unroll
              for (int jj = 0; jj < 16; ++jj) v[jj] = v[jj] < 0.f ? 0.f : v[jj];
            } else if (p.relu) {
#pragma unroll
              for (int jj = 0; jj < 16; ++jj) v[jj] = fmaxf(v[jj], 0.f);
            }
          }
          if (ncols > 0) {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.out) + off + col0;
            if (ncols == 16 && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
              store8_bf16(dst, v);
              store8_bf16(dst + 8, v + 8);
            } else {
#pragma unroll
              for (int jj = 0; jj < 16; ++jj) if (jj < ncols) dst[jj] = __float2bfloat16(v[jj]);
            }
          }
          if (MODE == CONV_FPROP) {
            if (do_stats) {
              // statistics of what the next layer will read: the values as rounded to bf16
              float s1[16], s2[16];
#pragma unroll
              for (int jj = 0; jj < 16; ++jj) {
                const float x = (jj < ncols) ? __bfloat162float(__float2bfloat16(v[jj])) : 0.f;
                s1[jj] = x; s2[jj] = x * x;
              }
              const float a = warp_column_sums16(s1, lane);
              const float b = warp_column_sums16(s2, lane);
              // both lanes of a pair hold one column: bits 4..1 of the lane, most significant first
              const int colm = col0 + (((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1));
              if ((lane & 1) == 0 && colm < p.Nc) {
                atomicAdd(&s_stat[colm], a);
                atomicAdd(&s_stat[p.Nc + colm], b);
              }
            }
          }
        }
      }
      __syncwarp();
      tc_fence_before();
      mbar_arrive(&tempty[as]);
      if (trace != nullptr && threadIdx.x == 64) { trace[5] += clock64() - tw1; trace[6] += tw1 - tw0; }
      if (++as == 2) { as = 0; aphase ^= 1; }
    }
    if (trace != nullptr && threadIdx.x == 64) trace[7] = clock64();
    if (!ok && lane == 0) {
      *abort_flag = 1;
      if (p.error_flag) atomicExch(p.error_flag, 13);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::TMEM_COLS) : "memory");
  }
  if (MODE == CONV_FPROP) {
    if (do_stats) {
      for (int i = threadIdx.x; i < 2 * p.Nc; i += C::THREADS) {
        const float x = s_stat[i];
        if (x != 0.f) atomicAdd(p.stats + i, x);
      }
    }
  }
}

template <int BN, int MODE>
cudaError_t launch_one(const ConvMaps& maps, const ConvParams& p, int num_sms, cudaStream_t stream) {
  using C = ConvCfg<BN, MODE>;
  auto kern = conv_kernel<BN, MODE>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  const int c_tiles = (p.Nc + BN - 1) / BN;
  long long tiles;
  if (MODE != CONV_WGRAD) tiles = (long long)p.tiles_w * p.tiles_h * p.tiles_n * c_tiles;
  else tiles = (long long)((p.Mc + BM - 1) / BM) * c_tiles * p.ntaps * p.ksplit;
  if (tiles <= 0) return cudaSuccess;
  const int grid = (int)(tiles < num_sms ? tiles : num_sms);
  launch_pdl(kern, dim3(grid), dim3(C::THREADS), C::SMEM, stream, maps, p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_conv(const ConvMaps& maps, const ConvParams& p, int bn, int num_sms, cudaStream_t stream) {
  if (p.tw * p.th * p.tn > BM || p.ntaps < 1 || p.ntaps > kMaxConvTaps) return cudaErrorInvalidValue;
  if (p.mode == CONV_WGRAD && (p.tw * p.th * p.tn != BK || p.ksplit < 1)) return cudaErrorInvalidValue;
  if ((p.mode == CONV_EVAL || (p.mode == CONV_FPROP && p.stats != nullptr)) && p.Nc > kMaxStatChannels) return cudaErrorInvalidValue;
  if (p.mode == CONV_DGRAD && p.staged == 0) return cudaErrorInvalidValue;
  if ((p.mode == CONV_EVAL) != (p.bn_mean != nullptr) || (p.mode == CONV_EVAL && p.stats != nullptr)) return cudaErrorInvalidValue;
#define ADB_CONV_DISPATCH(BN_)                                                                      \
  if (bn == BN_) {                                                                                  \
    if (p.mode == CONV_FPROP) return launch_one<BN_, CONV_FPROP>(maps, p, num_sms, stream);          \
    if (p.mode == CONV_DGRAD) return launch_one<BN_, CONV_DGRAD>(maps, p, num_sms, stream);          \
    if (p.mode == CONV_WGRAD) return launch_one<BN_, CONV_WGRAD>(maps, p, num_sms, stream);          \
    if (p.mode == CONV_EVAL) return launch_one<BN_, CONV_EVAL>(maps, p, num_sms, stream);            \
  }
  ADB_CONV_DISPATCH(256)
  ADB_CONV_DISPATCH(128)
  ADB_CONV_DISPATCH(64)
#undef ADB_CONV_DISPATCH
  return cudaErrorInvalidValue;
}

}  // namespace adb200
