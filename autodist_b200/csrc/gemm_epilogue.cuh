// The generic epilogue of the tcgen05 GEMM kernels: one thread owns one accumulator row (TMEM lane) and walks it in
// chunks of 16 columns - scale, bias / GELU / tanh / addend, then bf16 or fp32 row stores (see GemmParams).
#pragma once
#include "gemm_tcgen05.h"
#include "tcgen05_common.cuh"

namespace adb200 {
namespace tc {

// The auxiliary operand's part: addend, or GELU derivative at a pre-activation.
template <int NV>
__device__ __forceinline__ void gemm_epilogue_aux(const GemmParams& p, float* v, const float* x) {
  if (p.epilogue == EPI_ADD) {
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] += x[j];
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] *= gelu_tanh_grad(x[j]);
  }
}

// The arithmetic of the epilogue on NV (16 or 4) accumulator values of one row, in place: scale, then bias (+ tanh), addend
// or GELU derivative. `ncols` of the NV columns starting at `col0` (a multiple of NV) exist (0: nothing is read from memory).
template <int NV>
__device__ __forceinline__ void gemm_epilogue_math(const GemmParams& p, float* v, int col0, int ncols, long long coff, bool vec_ok) {
#pragma unroll
  for (int j = 0; j < NV; ++j) v[j] *= p.alpha;
  if (p.epilogue == EPI_BIAS || p.epilogue == EPI_BIAS_GELU || p.epilogue == EPI_BIAS_TANH) {
    if (ncols == NV && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0) {
#pragma unroll
      for (int j = 0; j < NV; j += 4) {                      // col0 is a multiple of 4: aligned 16-byte loads
        const float4 b4 = __ldg(reinterpret_cast<const float4*>(p.bias + col0 + j));
        v[j] += b4.x; v[j + 1] += b4.y; v[j + 2] += b4.z; v[j + 3] += b4.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < NV; ++j) if (j < ncols) v[j] += __ldg(p.bias + col0 + j);
    }
    if (p.epilogue == EPI_BIAS_TANH) {
#pragma unroll
      for (int j = 0; j < NV; ++j) v[j] = tanhf(v[j]);
    }
  } else if (p.epilogue == EPI_ADD || p.epilogue == EPI_MUL_GELU_GRAD) {
    const __nv_bfloat16* aux = p.aux + coff + col0;
    float x[NV];
    if (ncols == NV && vec_ok) {
      if constexpr (NV == 16) {
        const uint4 u0 = *reinterpret_cast<const uint4*>(aux), u1 = *reinterpret_cast<const uint4*>(aux + 8);
        unpack8_bf16(u0, x);
        unpack8_bf16(u1, x + 8);
      } else {
        const uint2 u = *reinterpret_cast<const uint2*>(aux);
        const float2 f0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
        const float2 f1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
        x[0] = f0.x; x[1] = f0.y; x[2] = f1.x; x[3] = f1.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < NV; ++j) x[j] = (j < ncols) ? __bfloat162float(aux[j]) : 0.f;
    }
    gemm_epilogue_aux<NV>(p, v, x);
  }
}
__device__ __forceinline__ void gemm_epilogue_math16(const GemmParams& p, float* v, int col0, int ncols, long long coff, bool vec_ok) {
  gemm_epilogue_math<16>(p, v, col0, ncols, coff, vec_ok);
}

// ---------------------------------------------------------------------------------------------------------------------
// Output through shared memory and TMA, for the tiles of 256 and 192 columns. Direct stores leave a warp writing 32 different rows in
// 16-byte pieces - partial sectors that cost the L2 as much as full ones and compete with the operand loads. Here each
// epilogue warp owns 32 rows x 64 G columns (G = 2 for 256-wide tiles), stages 32 rows x 128 bytes (64 bf16 or 32 fp32 columns) in the 128-byte-swizzled layout
// and one lane hands the box to the TMA unit, which writes whole lines (or adds them into an fp32 output: beta = 1). Rows and
// columns past the matrix are clipped by the copy itself. The 4 KB buffers of a warp take turns, so staging overlaps the copy.
//
// What the epilogue reads is requested while the tile is still being multiplied: the auxiliary operand (addend or pre-activation)
// comes by TMA into the staging buffers and is replaced there by the result, the bias into registers. The accumulator of a bf16
// output is read in the fragment layout (tmem_ld_frag32), where a lane needs 32 values of the bias for its 32 rows x 128 columns,
// and the arithmetic is on pairs of values.
// A tile's drain is exposed once per launch and, with a short contraction, once per tile: with GELU it took longer than the
// multiplication of a 1024-deep tile. 4096 x 4096 x 1024 on SM pairs, back to back (a row per thread, the bias handed around by
// shuffles -> now, us): bias + GELU 36.0 -> 32.9, GELU derivative 36.3 -> 31.5, plain 26.8 -> 25.7. Sixteen warps of 32 x 64 with one
// buffer each: 34.3, 32.4, and 0.4 us more on every product.
//
// G: groups of 64 columns per warp, and staging buffers: two for the 256-wide tiles, one for 192 (twelve warps, three per lane quarter).
template <int G>
struct EpiStage {
  const CUtensorMap* tmC;      // output map, box (128 bytes of columns, 32 rows, 1, 1), 128-byte swizzle
  const CUtensorMap* tmC2;     // EPI_BIAS_GELU: second output; EPI_ADD / EPI_MUL_GELU_GRAD: the auxiliary operand (same box)
  uint32_t smem;               // shared address of this warp's G staging buffers of 4 KB (1024-byte aligned)
  uint64_t* aux_bar;           // G barriers of this warp: auxiliary box g has landed in buffer g
  int units;                   // copies issued so far by this warp (picks the buffer)
  uint32_t aux_phase;          // bit g: parity the next wait on aux_bar[g] expects
  uint32_t aux_pending;        // bit g: a load into buffer g has been requested and not yet waited for
  float2 bias[8 * G];          // columns 8 k + 2 (lane % 4) and the next of this warp's 64 G (0 past the matrix or without a bias)
};

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) { return pack2(a, b); }
__device__ __forceinline__ bool epi_has_bias(const GemmParams& p) {
  return p.epilogue == EPI_BIAS || p.epilogue == EPI_BIAS_GELU || p.epilogue == EPI_BIAS_TANH;
}

// Requests what the epilogue of the next tile reads (see EpiStage); n0: first of this warp's columns.
template <int G>
__device__ __forceinline__ void gemm_epilogue_prefetch(const GemmParams& p, EpiStage<G>& st, int box_row, int n0, int b_lo, int b_hi, int lane) {
  if (box_row >= p.M) return;
  if (epi_has_bias(p)) {
#pragma unroll
    for (int k = 0; k < 8 * G; ++k) {
      const int col = n0 + 8 * k + 2 * (lane & 3);
      st.bias[k] = make_float2(col < p.N ? __ldg(p.bias + col) : 0.f, col + 1 < p.N ? __ldg(p.bias + col + 1) : 0.f);
    }
  } else if (p.epilogue == EPI_ADD || p.epilogue == EPI_MUL_GELU_GRAD) {
    if (elect_one()) bulk_wait_read<0>();             // the previous tile's copies have left the buffers
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (n0 + g * 64 >= p.N) break;
      if (elect_one()) {
        mbar_expect_tx(&st.aux_bar[g], 4096);
        asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
            ::"r"(st.smem + (uint32_t)g * 4096u), "l"(st.tmC2), "r"(smem_u32(&st.aux_bar[g])), "r"(n0 + g * 64), "r"(box_row), "r"(b_lo), "r"(b_hi)
            : "memory");
      }
      st.aux_pending |= 1u << g;
    }
  }
}

// Before the warp leaves: auxiliary boxes that nobody waited for (another role gave up) land first.
template <int G>
__device__ __forceinline__ void gemm_epilogue_drain(EpiStage<G>& st) {
  for (int g = 0; g < G; ++g)
    if (st.aux_pending & (1u << g)) {
      const long long t0 = clock64();
      while (!mbar_try(&st.aux_bar[g], (st.aux_phase >> g) & 1u) && clock64() - t0 < 20000000LL) {}
    }
}

// The staged lines of a buffer -> the TMA unit.
__device__ __forceinline__ void gemm_epilogue_hand_over(const CUtensorMap* map, uint32_t base, int col, int box_row, int b_lo, int b_hi, bool add) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (elect_one()) {
    if (add) tma_reduce_add_4d(map, base, col, box_row, b_lo, b_hi);
    else tma_store_4d(map, base, col, box_row, b_lo, b_hi);
    bulk_commit();
  }
}
// The buffer about to be written is no longer being read: all but the last G - 1 copies have left theirs.
template <int G>
__device__ __forceinline__ void gemm_epilogue_buffer_free() {
  if (elect_one()) bulk_wait_read<G - 1>();
  __syncwarp();
}

// A warp's 32 x 64 G accumulator elements, bf16 outputs. EPI is the product's epilogue: one copy of the code per kind, since a test
// per element costs more than the arithmetic. Returns false when an auxiliary box did not arrive in time.
template <int EPI, int G, class Release>
__device__ __forceinline__ bool gemm_epilogue_bf16(const GemmParams& p, EpiStage<G>& st, uint32_t t_w, int box_row, int n0, int b_lo, int b_hi, int lane,
                                                   volatile int* abort_flag, Release& release) {
  constexpr bool BIAS = EPI == EPI_BIAS || EPI == EPI_BIAS_GELU || EPI == EPI_BIAS_TANH, AUX = EPI == EPI_ADD || EPI == EPI_MUL_GELU_GRAD;
  const uint32_t swz = (uint32_t)(lane >> 2);         // line % 8 of every row of this lane
  const uint32_t mine = (uint32_t)(lane >> 2) * 128u + (uint32_t)(lane & 3) * 4u;
  const uint64_t alpha = both(p.alpha);
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const int col0 = n0 + g * 64;
    if (col0 >= p.N) {                                // uniform over the warp; the first group exists
      release();
      break;
    }
    uint32_t base;
    if (AUX) {
      base = st.smem + (uint32_t)g * 4096u;           // the auxiliary box is already there
      if (!mbar_wait(&st.aux_bar[g], (st.aux_phase >> g) & 1u, abort_flag)) return false;
      st.aux_phase ^= 1u << g;
      st.aux_pending &= ~(1u << g);
    } else {
      gemm_epilogue_buffer_free<G>();
      base = st.smem + (uint32_t)(st.units % G) * 4096u;
    }
    uint32_t act[EPI == EPI_BIAS_GELU ? 32 : 1];      // GELU values (two outputs: the pre-activation, then its GELU)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t r[32];
      __syncwarp();                                   // tcgen05.ld is warp-collective
      tmem_ld_frag32(t_w + g * 64 + h * 32, r);
      if (g == G - 1 && h == 1) release();
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t at = base + mine + (uint32_t)i * 1024u + (((uint32_t)(h * 4 + k) ^ swz) << 4);
          const uint32_t* a = r + (i >> 1) * 16 + k * 4 + (i & 1) * 2;
          uint64_t v = mul2(pack_f32x2(__uint_as_float(a[0]), __uint_as_float(a[1])), alpha);
          if (BIAS) v = add2(v, pack_f32x2(st.bias[g * 8 + h * 4 + k].x, st.bias[g * 8 + h * 4 + k].y));
          if (EPI == EPI_BIAS_TANH) {
            const float2 f = unpack_f32x2(v);
            v = pack_f32x2(tanhf(f.x), tanhf(f.y));
          }
          if (EPI == EPI_ADD) v = add2(v, widen2(lds1(at)));
          if (EPI == EPI_MUL_GELU_GRAD) v = mul2(v, gelu_tanh_grad2(widen2(lds1(at))));
          sts1(at, round2(v));
          if (EPI == EPI_BIAS_GELU) act[h * 16 + k * 4 + i] = round2(gelu_tanh2(v));
        }
    }
    gemm_epilogue_hand_over(st.tmC, base, col0, box_row, b_lo, b_hi, false);
    st.units += 1;
    if (EPI == EPI_BIAS_GELU) {                       // the second output through the other buffer
      gemm_epilogue_buffer_free<G>();
      base = st.smem + (uint32_t)(st.units % G) * 4096u;
#pragma unroll
      for (int j = 0; j < 32; ++j) sts1(base + mine + (uint32_t)(j & 3) * 1024u + (((uint32_t)(j >> 2) ^ swz) << 4), act[j]);
      gemm_epilogue_hand_over(st.tmC2, base, col0, box_row, b_lo, b_hi, false);
      st.units += 1;
    }
  }
  return true;
}

// The same for fp32 outputs (boxes of 32 columns): a row per lane, whose staged lines are written in 16-byte pieces without bank
// conflicts. Bias is the only epilogue such outputs take; it is read again here.
template <int G, class Release>
__device__ __forceinline__ void gemm_epilogue_f32(const GemmParams& p, EpiStage<G>& st, uint32_t t_w, int box_row, int n0, int b_lo, int b_hi, int lane,
                                                  Release& release) {
  const uint32_t swz = (uint32_t)(lane & 7);
  const bool bias = epi_has_bias(p);
#pragma unroll 1
  for (int g = 0; g < 2 * G; ++g) {
    const int col0 = n0 + g * 32;
    if (col0 >= p.N) break;                           // uniform over the warp
    gemm_epilogue_buffer_free<G>();
    const uint32_t base = st.smem + (uint32_t)(st.units % G) * 4096u, buf = base + (uint32_t)lane * 128u;
    float v[32];
    __syncwarp();                                     // tcgen05.ld is warp-collective
    tmem_ld32(t_w + g * 32, v);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] *= p.alpha;
    if (bias) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (col0 + j < p.N) v[j] += __ldg(p.bias + col0 + j);
        if (p.epilogue == EPI_BIAS_TANH) v[j] = tanhf(v[j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      st_shared_v4(buf + (((uint32_t)i ^ swz) << 4), __float_as_uint(v[4 * i]), __float_as_uint(v[4 * i + 1]), __float_as_uint(v[4 * i + 2]),
                   __float_as_uint(v[4 * i + 3]));
    gemm_epilogue_hand_over(st.tmC, base, col0, box_row, b_lo, b_hi, p.beta != 0.0f);
    st.units += 1;
  }
  release();
}

// t_w: TMEM address of this warp's 32 lanes at the first of its columns; box_row: first of its output rows. `release` is called once,
// when the accumulator has been read. Returns false when an auxiliary box did not arrive in time (`release` has not been called then).
template <int G, class Release>
__device__ __forceinline__ bool gemm_epilogue_tma(const GemmParams& p, EpiStage<G>& st, uint32_t t_w, int box_row, int n0, int b_lo, int b_hi, int lane,
                                                  volatile int* abort_flag, Release&& release) {
  if (box_row >= p.M || n0 >= p.N) {                  // none of this warp's elements exist
    release();
    return true;
  }
  if (p.c_is_fp32) {
    gemm_epilogue_f32(p, st, t_w, box_row, n0, b_lo, b_hi, lane, release);
    return true;
  }
  if (p.epilogue == EPI_ADD) return gemm_epilogue_bf16<EPI_ADD>(p, st, t_w, box_row, n0, b_lo, b_hi, lane, abort_flag, release);
  if (p.epilogue == EPI_MUL_GELU_GRAD) return gemm_epilogue_bf16<EPI_MUL_GELU_GRAD>(p, st, t_w, box_row, n0, b_lo, b_hi, lane, abort_flag, release);
  if (p.epilogue == EPI_BIAS) return gemm_epilogue_bf16<EPI_BIAS>(p, st, t_w, box_row, n0, b_lo, b_hi, lane, abort_flag, release);
  if (p.epilogue == EPI_BIAS_GELU) return gemm_epilogue_bf16<EPI_BIAS_GELU>(p, st, t_w, box_row, n0, b_lo, b_hi, lane, abort_flag, release);
  if (p.epilogue == EPI_BIAS_TANH) return gemm_epilogue_bf16<EPI_BIAS_TANH>(p, st, t_w, box_row, n0, b_lo, b_hi, lane, abort_flag, release);
  return gemm_epilogue_bf16<EPI_NONE>(p, st, t_w, box_row, n0, b_lo, b_hi, lane, abort_flag, release);
}

// t_row: TMEM address of this thread's lane at the first column of the accumulator; row: output row (may be >= M);
// n0: first output column of the tile; coff: element offset of (row, 0) in C.
template <int BN>
__device__ __forceinline__ void gemm_epilogue_row(const GemmParams& p, uint32_t t_row, int row, int n0, long long coff, bool vec_ok) {
#pragma unroll 1
  for (int c = 0; c < BN / 16; ++c) {
    float v[16];
    __syncwarp();                          // tcgen05.ld is warp-collective: reconverge after predicated stores
    tmem_ld16(t_row + c * 16, v);
    const int col0 = n0 + c * 16;
    const int ncols = (row < p.M) ? min(16, p.N - col0) : 0;
    if (ncols > 0) {
    gemm_epilogue_math16(p, v, col0, ncols, coff, vec_ok);
    if (p.c_is_fp32) {
      float* dst = reinterpret_cast<float*>(p.C) + coff + col0;
      if (p.beta != 0.0f) {
        if (ncols == 16 && vec_ok) {
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            float4 o = *reinterpret_cast<float4*>(dst + j);
            o.x += v[j]; o.y += v[j + 1]; o.z += v[j + 2]; o.w += v[j + 3];
            *reinterpret_cast<float4*>(dst + j) = o;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) if (j < ncols) dst[j] += v[j];
        }
      } else if (ncols == 16 && vec_ok) {
#pragma unroll
        for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) if (j < ncols) dst[j] = v[j];
      }
    } else {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + coff + col0;
      if (ncols == 16 && vec_ok) {
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
          w[j] = *reinterpret_cast<uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(dst + 8) = make_uint4(w[4], w[5], w[6], w[7]);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) if (j < ncols) dst[j] = __float2bfloat16(v[j]);
      }
      if (p.epilogue == EPI_BIAS_GELU) {
        __nv_bfloat16* dst2 = p.C2 + coff + col0;
        if (ncols == 16 && vec_ok) {
          uint32_t w[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            __nv_bfloat162 h = __floats2bfloat162_rn(gelu_tanh(v[2 * j]), gelu_tanh(v[2 * j + 1]));
            w[j] = *reinterpret_cast<uint32_t*>(&h);
          }
          *reinterpret_cast<uint4*>(dst2) = make_uint4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<uint4*>(dst2 + 8) = make_uint4(w[4], w[5], w[6], w[7]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) if (j < ncols) dst2[j] = __float2bfloat16(gelu_tanh(v[j]));
        }
      }
    }
    }  // ncols > 0
  }
}

}  // namespace tc
}  // namespace adb200
