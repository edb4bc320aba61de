// Python bindings of the sm_100a kernels: tensor-map construction, argument checks, launches on the current stream.
#include <cstdlib>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda.h>
#include <cuda_runtime.h>
#include <torch/extension.h>

#include <algorithm>
#include <mutex>
#include <tuple>
#include <unordered_map>
#include <vector>

#include "attention.h"
#include "comm.h"
#include "elementwise.h"
#include "gemm_tcgen05.h"
#include "sampled_softmax.h"
#include "sm_count.h"

void register_conv(pybind11::module& m);

namespace {

using at::Tensor;
using c10::optional;

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
    TORCH_CHECK(e == cudaSuccess && p != nullptr, "cuTensorMapEncodeTiled is not available from this driver");
    fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

int num_sms() { return adb200::sm_count(); }

Tensor as4d(const Tensor& t) {
  TORCH_CHECK(t.dim() >= 2 && t.dim() <= 4, "operand must have 2 to 4 dimensions");
  Tensor v = t;
  while (v.dim() < 4) v = v.unsqueeze(0);
  return v;
}

// 4-D bf16 tiled map over a strided view [b_hi, b_lo, outer, inner] (inner stride 1), 128-byte swizzle.
CUtensorMap make_map(const Tensor& v, int box_outer) {
  TORCH_CHECK(v.scalar_type() == at::kBFloat16, "GEMM operands must be bf16");
  TORCH_CHECK(v.stride(3) == 1, "innermost dimension must be contiguous");
  TORCH_CHECK(reinterpret_cast<uintptr_t>(v.data_ptr()) % 16 == 0, "operand base must be 16-byte aligned");
  cuuint64_t dims[4] = {(cuuint64_t)v.size(3), (cuuint64_t)v.size(2), (cuuint64_t)v.size(1), (cuuint64_t)v.size(0)};
  cuuint64_t strides[3];
  int64_t prev = v.size(3);
  for (int i = 0; i < 3; ++i) {
    const int d = 2 - i;   // tensor dim of map dim i+1
    int64_t s = v.size(d) > 1 ? v.stride(d) : prev;
    TORCH_CHECK((s * 2) % 16 == 0 && s > 0, "operand strides must be positive multiples of 8 elements, got ", s);
    strides[i] = (cuuint64_t)s * 2;
    prev = s * v.size(d);
  }
  cuuint32_t box[4] = {64, (cuuint32_t)box_outer, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUtensorMap m;
  CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, v.data_ptr(), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TORCH_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with code ", (int)r);
  return m;
}

// 4-D map over an output view [b_hi, b_lo, rows, cols] (bf16 or fp32, inner stride 1) for the TMA-store epilogue: boxes of
// 128 bytes of columns x 32 rows, 128-byte swizzle. Returns false when the view cannot be described (a base or a stride
// that is not a multiple of 16 bytes): the caller then keeps the direct stores.
bool make_store_map(const Tensor& v, CUtensorMap* out) {
  const bool f32 = v.scalar_type() == at::kFloat;
  const int64_t esz = f32 ? 4 : 2;
  if (v.stride(3) != 1 || reinterpret_cast<uintptr_t>(v.data_ptr()) % 16 != 0) return false;
  cuuint64_t dims[4] = {(cuuint64_t)v.size(3), (cuuint64_t)v.size(2), (cuuint64_t)v.size(1), (cuuint64_t)v.size(0)};
  cuuint64_t strides[3];
  int64_t prev = v.size(3);
  for (int i = 0; i < 3; ++i) {
    const int d = 2 - i;
    const int64_t s = v.size(d) > 1 ? v.stride(d) : prev;
    if (s <= 0 || (s * esz) % 16 != 0) return false;
    strides[i] = (cuuint64_t)(s * esz);
    prev = s * v.size(d);
  }
  cuuint32_t box[4] = {(cuuint32_t)(128 / esz), 32, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = encode_fn()(out, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, v.data_ptr(), dims, strides, box,
                           estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Whether every row of a 4-D output view starts on a 16-byte boundary.
bool rows_aligned(const Tensor& v) {
  const int64_t n = 16 / v.element_size();
  if (reinterpret_cast<uintptr_t>(v.data_ptr()) % 16 != 0) return false;
  for (int d = 0; d < 3; ++d)
    if (v.size(d) > 1 && v.stride(d) % n != 0) return false;
  return true;
}

// Tuning aid: when set (int64 CUDA tensor of at least 8 x SM-count words, zeroed by the caller), launches of the two-CTA
// GEMM record nanosecond marks per CTA into it (see gemm_tcgen05_2cta.cu).
long long* g_gemm_trace = nullptr;
void gemm_set_trace(const optional<Tensor>& t) {
  if (t.has_value()) {
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kLong && t->is_contiguous() && t->numel() >= 8LL * num_sms(), "int64 [SMs, 8] needed");
    g_gemm_trace = reinterpret_cast<long long*>(t->data_ptr<int64_t>());
  } else {
    g_gemm_trace = nullptr;
  }
}

// Which kernel runs a product: the tile width (512: the two-CTA kernel) and how many CTAs share the contraction of one tile.
// The estimate in microseconds is launch + fill + first wave's K blocks of 64 + last drain, plus, per further wave of tiles, its K
// blocks or the drain of a tile, whichever is longer. A K block costs more the more SMs take part (`load`): their fills share the L2.
// The drain counts by kind (plain; bias or addend; activation; fp32 output): 64 and 128 columns store directly and read what they
// need when they need it, wider tiles go through shared memory and TMA. Splitting the contraction adds the exchange through
// distributed shared memory; it wins wherever the tiles leave SMs idle (256 x 256 x 16384 94.7 -> 14.7 us, 640 x 1024 x 30522
// 172 -> 39). Splits run one cluster per tile, so they are only considered while every cluster is resident at once.
// The constants are fitted to 170 products from 32 x 128 x 1000 to 8192 x 4096 x 1024 and 4096 x 25088 x 32 with every tile width and
// split (B200, replayed back to back): the estimates' choices take 0.6 % more time in sum than the fastest kernel of each product.
// Where the lines lie, in us:
//   192 columns fill the SMs where 256 leave a third of them idle (128 x 192 tiles and 256 x 256 pairs):
//     3072 x 1024 x 4096 20.0 (pairs 25.5), 4096 x 768 x 3072 16.2 (20.8), 1792 x 3072 x 768 with GELU 13.9 (15.7)
//   pairs win once there are waves of them: 4096 x 4096 x 1024 with GELU 32.8 (192 columns 38.4), 8192 x 1024 x 4096 52.8 (68.9)
//   256 columns on one CTA in between: 4096 x 1024 x 1024 10.1 (pairs 11.3, 192 columns 12.8)
//
// A width changes no bit of the result: every kernel adds the products of an output in ascending order of K. The number of shares
// does, since each share is summed by itself. See broad_choice for products whose sums must not move with these constants.
struct GemmChoice { int64_t bn, split; };
struct GemmTiles { int64_t tiles, slots; };              // output tiles of a width, and how many of them run at once
// false: the width does not suit the product
bool gemm_tiles(int bn, int64_t M, int64_t N, int64_t batch, bool allow_pair, GemmTiles* t) {
  const bool pair = bn == 512;
  if (pair && (!allow_pair || M < 256 || N < 256)) return false;
  if (!pair && bn > 64 && N <= bn / 2) return false;                      // more than half of the tile would be padding
  const int64_t tm = pair ? 256 : 128, tn = pair ? 256 : bn;
  *t = {((M + tm - 1) / tm) * ((N + tn - 1) / tn) * batch, pair ? num_sms() / 2 : num_sms()};
  return true;
}
bool gemm_split_fits(int64_t tiles, int s) { return tiles * s <= num_sms() && tiles <= adb200::gemm_split_max_clusters(s, (int)num_sms()); }

// shares: how many CTAs have to share the contraction; 0: as many as the estimate says.
GemmChoice choose_gemm(int64_t M, int64_t N, int64_t K, int64_t batch, bool allow_pair, bool allow_split, int64_t epilogue, bool both_mn, bool fp32_out,
                       int shares) {
  struct Cost { int bn; double base, kb, load, mn, epi[4], wave, exchange; };      // exchange 0: no split of this width
  static const Cost costs[5] = {{64, 2.87, 0.143, 0.17, 1.03, {1.3, 2.6, 3.5, 4.2}, 0.4, 2.0},
                                {128, 3.35, 0.169, 0.31, 1.00, {2.8, 5.2, 6.8, 7.9}, 0.4, 2.0},
                                {192, 3.16, 0.238, 0.18, 0.96, {3.4, 3.7, 5.7, 5.0}, 1.2, 0.0},
                                {256, 3.29, 0.310, 0.31, 0.98, {4.0, 4.3, 6.4, 6.4}, 1.1, 5.0},
                                {512, 4.24, 0.281, 0.22, 0.97, {4.0, 5.0, 6.7, 6.7}, 0.4, 0.0}};
  const int kind = fp32_out ? 3 : (epilogue == adb200::EPI_NONE ? 0 : (epilogue == adb200::EPI_BIAS || epilogue == adb200::EPI_ADD || epilogue == adb200::EPI_BIAS_TANH ? 1 : 2));
  const int64_t kbs = (K + 63) / 64, sms = num_sms();
  // Terms that the fit does not hold, with the sums over random products whose choice they decide, in us, with the term / without it,
  // replayed on one set of operands; and on sets that do not fit the L2:
  //   margin  a split has to be estimated that much faster: launching clusters costs more beside neighbours than back to back
  //           24 products 158.7 / 163.3; 161.5 / 164.9
  //   sparse  192 and 256 columns, whose epilogue has many warps, only where they fill close to half of the SMs
  //           22 products 124.6 / 135.1; 127.3 / 141.9   (tiny BERT 377 -> 360 us, base tied 3757 -> 3660, with the margin)
  //   narrow  in several waves of long contractions the widest tiles read the least from memory
  //           22 products 939 / 919; 966 / 1015
  //   beside  long weight gradients stay on pairs, whose idle SMs run the optimizer beside them; without one they pay for it
  //           22 products 694 / 615; 704 / 695           (BERT-large step 12.26 ms / 12.35)
  const double margin = shares > 0 ? 0.0 : 0.8;
  GemmChoice best{64, shares > 0 ? shares : 1};
  double best_us = 1e30;
  for (const Cost& c : costs) {
    GemmTiles t;
    if (!gemm_tiles(c.bn, M, N, batch, allow_pair, &t)) continue;
    const double extra = c.epi[kind] - c.epi[0];                       // the last wave's drain (the plain one is part of the base)
    auto blocks = [&](int64_t ctas, int64_t n) { return c.kb * (both_mn ? c.mn : 1.0) * (1.0 + c.load * std::min(1.0, (double)ctas / (double)t.slots)) * (double)n; };
    const bool sparse = (c.bn == 192 || c.bn == 256) && 2 * t.tiles < sms - 20;
    const bool narrow = c.bn < 256 && N > 128 && t.tiles > sms && K > 1024;
    const bool beside = c.bn == 192 && fp32_out && K > 2048;
    if (shares <= 1 && !sparse && !narrow && !beside) {
      const double waves = (double)((t.tiles + t.slots - 1) / t.slots);
      const double us = c.base + (waves - 1) * std::max(blocks(t.tiles, kbs) + c.wave, c.epi[kind]) + blocks(t.tiles, kbs) + extra;
      if (us < best_us) { best_us = us; best = {c.bn, 1}; }
    }
    if (c.exchange == 0.0 || !allow_split || shares == 1) continue;
    for (int s = shares > 1 ? shares : 2; s <= (shares > 1 ? shares : 8) && s <= kbs; ++s) {
      if (!gemm_split_fits(t.tiles, s)) continue;
      const double us = c.base + blocks(t.tiles * s, (kbs + s - 1) / s) + c.exchange + extra / s;
      if (us < best_us - margin) { best_us = us; best = {c.bn, s}; }
    }
  }
  return best;
}

// An older and broader estimate, over 60 products from 512 x 128 x 128 to 32 x 4096 x 25088, hot and cold. Its constants stay as they are,
// whatever the kernels and the estimate above become, for the sake of the first of the two things it decides:
// 1. Shares of a contraction for products that ask for them with bn = -1. What is rounded to bf16 behind a product changes by an ulp here and
//    there with the order of its sums; a recurrence carries that on (LM1B's gradients over 20 LSTM steps: 4e-4 of their norm from one number
//    of shares to another), so the LSTM layer and what its gradient comes from ask for these.
// 2. Everything for long contractions over operands whose rows do not start on 128-byte lines. Every box of such an operand lies on two lines
//    per row, so fills cost more than the estimate above knows (a K block of 192 columns 0.48 us instead of 0.25), and it takes
//    tiles that are too narrow and shares that are too few. Sums over random products, us, estimate above / this one / the fastest:
//    K >= 4096 10587 / 10405 / 10366 (217 products; 33 of them more than 10 % slower than with this one), 2048 to 4096 1614 / 1588 / 1574 (84, 15),
//    1024 to 2048 950 / 981 / 919, below 2105 / 2108 / 2026. Rows on lines: 10476 / 10607 / 10286 (594, K from 64 to 32000).
GemmChoice broad_choice(int64_t M, int64_t N, int64_t K, int64_t batch, bool allow_pair, int64_t epilogue, bool both_mn) {
  struct Cost { int bn; double base, kb, epi[3], exchange; };
  static const Cost costs[4] = {{64, 2.9, 0.30, {1.6, 2.0, 3.6}, 2.6},
                                {128, 4.2, 0.33, {2.7, 3.4, 7.5}, 2.6},
                                {256, 4.6, 0.48, {2.5, 3.7, 6.5}, 3.5},
                                {512, 7.0, 0.41, {2.5, 3.7, 6.5}, 0.0}};
  const int kind = epilogue == adb200::EPI_NONE ? 0 : (epilogue == adb200::EPI_BIAS || epilogue == adb200::EPI_BIAS_TANH ? 1 : 2);
  const int64_t kbs = (K + 63) / 64;
  GemmChoice best{64, 1};
  double best_us = 1e30;
  for (const Cost& c : costs) {
    GemmTiles t;
    if (!gemm_tiles(c.bn, M, N, batch, allow_pair, &t)) continue;
    const double kb = c.bn == 128 && both_mn ? 0.42 : c.kb;
    const double extra = c.epi[kind] - c.epi[0], waves = (double)((t.tiles + t.slots - 1) / t.slots);
    const double us = c.base + (waves - 1) * std::max(kb * (double)kbs, c.epi[kind]) + kb * (double)kbs + extra;
    if (us < best_us) { best_us = us; best = {c.bn, 1}; }
    if (c.exchange == 0.0) continue;
    for (int s = 2; s <= 8 && s <= kbs; ++s) {
      if (!gemm_split_fits(t.tiles, s)) continue;
      const double us_s = c.base + kb * (double)((kbs + s - 1) / s) + c.exchange + extra / s;
      if (us_s < best_us) { best_us = us_s; best = {c.bn, s}; }
    }
  }
  return best;
}
constexpr int64_t kLongContraction = 2048;

// The kernel that bn = 0 asks for. AUTODIST_GEMM_PAIR=0 rules the two-CTA kernel out. AUTODIST_GEMM_PAIR_MIN_K sets a fixed rule
// for it in place of the estimate: products with a pair's tile in both extents whose tiles fill the SM pairs, or whose contraction
// is at least that long.
bool g_pair_unavailable = false;               // set when a cluster launch was refused once (see gemm_impl)
GemmChoice auto_choice(int64_t M, int64_t N, int64_t K, int64_t batch, int64_t epilogue, bool both_mn, bool fp32_out, bool fixed,
                       bool off_lines) {
  static const bool pair_default = [] { const char* e = std::getenv("AUTODIST_GEMM_PAIR"); return e == nullptr || e[0] != '0'; }();
  static const int64_t pair_min_k = [] { const char* e = std::getenv("AUTODIST_GEMM_PAIR_MIN_K"); return e != nullptr ? std::atoll(e) : -1LL; }();
  const bool softmax_epi = epilogue == adb200::EPI_SOFTMAX || epilogue == adb200::EPI_SOFTMAX_GRAD;
  bool pair = pair_default && !g_pair_unavailable && !softmax_epi;
  if (pair && pair_min_k >= 0) {
    const int64_t pair_tiles = ((M + 255) / 256) * ((N + 255) / 256) * batch;
    if (M >= 256 && N >= 256 && (pair_tiles >= num_sms() / 2 || K >= pair_min_k)) return {512, 1};
    pair = false;
  }
  if (!softmax_epi && (fixed || (off_lines && K >= kLongContraction))) {
    const GemmChoice broad = broad_choice(M, N, K, batch, pair, epilogue, both_mn);
    if (off_lines && K >= kLongContraction) return broad;
    return choose_gemm(M, N, K, batch, pair, true, epilogue, both_mn, fp32_out, (int)broad.split);
  }
  return choose_gemm(M, N, K, batch, pair, !softmax_epi, epilogue, both_mn, fp32_out, 0);
}
// (tile width, contraction split) of gemm(..., bn = 0) for a product of these extents: 512 is the two-CTA kernel. fp32_out: the type of
// the output; where it is not given, that of a weight gradient (fp32) for two MN-major operands and bf16 for others. fixed: of bn = -1. The operands'
// rows follow one another.
std::tuple<int64_t, int64_t> gemm_choice(int64_t M, int64_t N, int64_t K, int64_t batch, int64_t epilogue, bool both_mn, const optional<bool>& fp32_out,
                                         bool fixed) {
  const bool off_lines = both_mn ? M % 64 != 0 && N % 64 != 0 : K % 64 != 0;
  const GemmChoice g = auto_choice(M, N, K, batch, epilogue, both_mn, fp32_out.value_or(both_mn), fixed, off_lines);
  return {g.bn, g.split};
}

// D = alpha * A.B^T (+ epilogue). a: [.., M, K] (K-major) or [.., K, M] (a_mn); b: [.., N, K] or [.., K, N] (b_mn);
// c: [.., M, N] bf16 or fp32 view with unit inner stride.
void gemm_impl(const Tensor& a_, const Tensor& b_, Tensor c_, bool a_mn, bool b_mn, int64_t epilogue, const optional<Tensor>& bias,
               const optional<Tensor>& c2, const optional<Tensor>& aux, double alpha, double beta, Tensor error_flag, int64_t bn,
               const optional<Tensor>& mask, double drop_p, int64_t drop_seed, const optional<Tensor>& drop_step, int64_t split = 0) {
  const c10::cuda::CUDAGuard guard(a_.device());
  Tensor a = as4d(a_), b = as4d(b_), c = as4d(c_);
  const int M = a_mn ? a.size(3) : a.size(2), K = a_mn ? a.size(2) : a.size(3);
  const int N = b_mn ? b.size(3) : b.size(2), Kb = b_mn ? b.size(2) : b.size(3);
  TORCH_CHECK(K == Kb, "contraction extents differ: ", K, " vs ", Kb);
  TORCH_CHECK(a.size(0) == b.size(0) && a.size(1) == b.size(1), "batch dimensions of A and B differ");
  TORCH_CHECK(c.size(0) == a.size(0) && c.size(1) == a.size(1) && c.size(2) == M && c.size(3) == N, "output shape mismatch");
  TORCH_CHECK(c.stride(3) == 1, "output inner stride must be 1");
  // bn: tile width 64 / 128 / 192 / 256 of the one-CTA kernel, or 512 = the 256 x 256 tile of the two-CTA kernel; 0 picks the kernel
  // (see choose_gemm and auto_choice), -1 only its tile, with the contraction shared as broad_choice says
  const bool softmax_epi = epilogue == adb200::EPI_SOFTMAX || epilogue == adb200::EPI_SOFTMAX_GRAD;
  const bool auto_bn = bn <= 0;
  if (auto_bn) {
    auto off_lines = [](const Tensor& t) { return t.stride(2) % 64 != 0 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 128 != 0; };
    const GemmChoice g = auto_choice(M, N, K, a.size(0) * a.size(1), epilogue, a_mn && b_mn, c.scalar_type() == at::kFloat, bn == -1,
                                     off_lines(a) && off_lines(b));
    bn = g.bn;
    split = g.split;
  }
  TORCH_CHECK(bn == 64 || bn == 128 || bn == 192 || bn == 256 || bn == 512, "bn must be 64, 128, 192, 256 or 512 (two-CTA tile)");
  const bool pair = bn == 512;
  CUtensorMap tmA = make_map(a, a_mn ? 64 : 128);
  adb200::TmapArray tmB;
  tmB.m[0] = make_map(b, b_mn ? 64 : (pair ? 128 : (int)bn));
  for (int i = 1; i < 8; ++i) tmB.m[i] = tmB.m[0];
  adb200::GemmParams p{};
  p.b_shard_rows = 0;
  p.trace = g_gemm_trace;
  p.M = M; p.N = N; p.K = K;
  p.batch_lo = a.size(1); p.batch_hi = a.size(0);
  p.C = c.data_ptr();
  p.ldc = c.stride(2);
  p.strideC_lo = c.size(1) > 1 ? c.stride(1) : 0;
  p.strideC_hi = c.size(0) > 1 ? c.stride(0) : 0;
  TORCH_CHECK(c.scalar_type() == at::kFloat || c.scalar_type() == at::kBFloat16, "output must be fp32 or bf16");
  p.c_is_fp32 = c.scalar_type() == at::kFloat;
  p.epilogue = (int)epilogue;
  p.alpha = (float)alpha;
  p.beta = (float)beta;
  p.bias = nullptr; p.C2 = nullptr; p.aux = nullptr;
  if (epilogue == adb200::EPI_BIAS || epilogue == adb200::EPI_BIAS_GELU || epilogue == adb200::EPI_BIAS_TANH) {
    TORCH_CHECK(bias.has_value() && bias->scalar_type() == at::kFloat && bias->numel() >= N, "fp32 bias of N entries needed");
    p.bias = bias->data_ptr<float>();
  }
  if (epilogue == adb200::EPI_BIAS_GELU) {
    TORCH_CHECK(c2.has_value() && c2->scalar_type() == at::kBFloat16 && !p.c_is_fp32, "bf16 second output needed");
    Tensor c2v = as4d(*c2);
    TORCH_CHECK(c2v.strides() == c.strides(), "second output must share the strides of the first");
    p.C2 = reinterpret_cast<__nv_bfloat16*>(c2v.data_ptr());
  }
  if (epilogue == adb200::EPI_MUL_GELU_GRAD || epilogue == adb200::EPI_ADD) {
    TORCH_CHECK(aux.has_value() && aux->scalar_type() == at::kBFloat16 && !p.c_is_fp32, "bf16 auxiliary operand and bf16 output needed");
    Tensor av = as4d(*aux);
    TORCH_CHECK(av.strides() == c.strides(), "pre-activation must share the strides of the output");
    p.aux = reinterpret_cast<const __nv_bfloat16*>(av.data_ptr());
  }
  p.mask = nullptr; p.drop_p = 0.f; p.drop_seed = 0; p.drop_step = nullptr;
  if (epilogue == adb200::EPI_SOFTMAX || epilogue == adb200::EPI_SOFTMAX_GRAD) {
    TORCH_CHECK(bn == 128 && N == 128 && !p.c_is_fp32 && c.stride(2) == 128, "the softmax epilogues need N == 128 and a contiguous bf16 output row");
    if (mask.has_value()) {
      TORCH_CHECK(mask->scalar_type() == at::kFloat && mask->numel() == a.size(0) * 128, "fp32 mask [batch_hi, 128] needed");
      p.mask = mask->data_ptr<float>();
    }
    p.drop_p = (float)drop_p;
    p.drop_seed = (unsigned long long)drop_seed;
    p.drop_step = drop_step.has_value() ? reinterpret_cast<const long long*>(drop_step->data_ptr<int64_t>()) : nullptr;
    if (epilogue == adb200::EPI_SOFTMAX && c2.has_value()) {
      Tensor c2v = as4d(*c2);
      TORCH_CHECK(c2v.scalar_type() == at::kBFloat16 && c2v.strides() == c.strides(), "dropped copy must share the strides of the output");
      p.C2 = reinterpret_cast<__nv_bfloat16*>(c2v.data_ptr());
    }
    if (epilogue == adb200::EPI_SOFTMAX_GRAD) {
      TORCH_CHECK(aux.has_value() && aux->scalar_type() == at::kBFloat16, "probabilities needed");
      Tensor av = as4d(*aux);
      TORCH_CHECK(av.strides() == c.strides(), "probabilities must share the strides of the output");
      p.aux = reinterpret_cast<const __nv_bfloat16*>(av.data_ptr());
    }
  }
  p.vec_ok = rows_aligned(c) && (p.C2 == nullptr || rows_aligned(as4d(*c2))) && (p.aux == nullptr || rows_aligned(as4d(*aux)));
  TORCH_CHECK(!softmax_epi || p.vec_ok, "the softmax epilogues need outputs that start on 16-byte boundaries");
  p.error_flag = error_flag.data_ptr<int>();
  // Output through shared memory and TMA (whole lines instead of 16-byte pieces of 32 rows per store instruction) for
  // products large enough to care; AUTODIST_GEMM_TMA_STORE=0 keeps direct stores everywhere.
  static const bool tma_store_default = [] { const char* e = std::getenv("AUTODIST_GEMM_TMA_STORE"); return e == nullptr || e[0] != '0'; }();
  CUtensorMap tmC, tmC2;
  p.tma_store = 0;
  if (tma_store_default && !softmax_epi && bn >= 192 && (!p.c_is_fp32 || p.beta == 0.0f || p.beta == 1.0f) && make_store_map(c, &tmC)) {
    p.tma_store = 1;
    tmC2 = tmC;
    if (epilogue == adb200::EPI_BIAS_GELU && !make_store_map(as4d(*c2), &tmC2)) p.tma_store = 0;
    if ((epilogue == adb200::EPI_ADD || epilogue == adb200::EPI_MUL_GELU_GRAD) && !make_store_map(as4d(*aux), &tmC2)) p.tma_store = 0;
  }
  if (split > 1) {
    const cudaError_t e = adb200::launch_gemm_split(tmA, tmB.m[0], p, (int)bn, (int)split, a_mn, b_mn, at::cuda::getCurrentCUDAStream());
    TORCH_CHECK(e == cudaSuccess, "split GEMM launch failed: ", cudaGetErrorString(e));
    return;
  }
  cudaError_t e = pair ? adb200::launch_gemm_pair(tmA, tmB.m[0], p, a_mn, b_mn, num_sms(), at::cuda::getCurrentCUDAStream(),
                                                  p.tma_store ? &tmC : nullptr, p.tma_store ? &tmC2 : nullptr)
                       : adb200::launch_gemm(tmA, tmB, p, (int)bn, a_mn, b_mn, num_sms(), at::cuda::getCurrentCUDAStream(),
                                             p.tma_store ? &tmC : nullptr, p.tma_store ? &tmC2 : nullptr);
  if (pair && auto_bn && e != cudaSuccess) {
    // A device (or partition of one) that cannot schedule clusters of two refuses the launch: remember it and run this and
    // every later product on the one-CTA kernel.
    (void)cudaGetLastError();
    g_pair_unavailable = true;
    tmB.m[0] = make_map(b, b_mn ? 64 : 256);
    for (int i = 1; i < 8; ++i) tmB.m[i] = tmB.m[0];
    e = adb200::launch_gemm(tmA, tmB, p, 256, a_mn, b_mn, num_sms(), at::cuda::getCurrentCUDAStream(), p.tma_store ? &tmC : nullptr,
                            p.tma_store ? &tmC2 : nullptr);
  }
  TORCH_CHECK(e == cudaSuccess, "GEMM launch failed: ", cudaGetErrorString(e));
}

void gemm(const Tensor& a, const Tensor& b, Tensor c, bool a_mn, bool b_mn, int64_t epilogue, const optional<Tensor>& bias,
          const optional<Tensor>& c2, const optional<Tensor>& aux, double alpha, double beta, Tensor error_flag, int64_t bn) {
  TORCH_CHECK(epilogue <= adb200::EPI_BIAS_TANH, "use gemm_softmax for the softmax epilogues");
  gemm_impl(a, b, c, a_mn, b_mn, epilogue, bias, c2, aux, alpha, beta, error_flag, bn, c10::nullopt, 0.0, 0, c10::nullopt);
}

// gemm with the contraction split over `split` CTAs of a cluster (bn 64 / 128 / 256).
void gemm_split(const Tensor& a, const Tensor& b, Tensor c, bool a_mn, bool b_mn, int64_t epilogue, const optional<Tensor>& bias,
                const optional<Tensor>& c2, const optional<Tensor>& aux, double alpha, double beta, Tensor error_flag, int64_t bn, int64_t split) {
  TORCH_CHECK(epilogue <= adb200::EPI_BIAS_TANH, "no softmax epilogue here");
  TORCH_CHECK((bn == 64 || bn == 128 || bn == 256) && split >= 2 && split <= 8, "tile width 64, 128 or 256 and a split of 2 to 8 needed");
  gemm_impl(a, b, c, a_mn, b_mn, epilogue, bias, c2, aux, alpha, beta, error_flag, bn, c10::nullopt, 0.0, 0, c10::nullopt, split);
}

// Attention products with the row softmax in the epilogue (rows of 128):
//   grad == false: c = softmax(alpha * a.b^T + mask), c2 (optional) = dropout(c)
//   grad == true : c = alpha * P * (d - sum(d * P)) with d = (a.b^T) * dropout mask and P = aux
void gemm_softmax(const Tensor& a, const Tensor& b, Tensor c, const optional<Tensor>& c2, const optional<Tensor>& mask,
                  const optional<Tensor>& aux, bool grad, double alpha, double drop_p, int64_t seed, const optional<Tensor>& step,
                  Tensor error_flag) {
  gemm_impl(a, b, c, false, false, grad ? adb200::EPI_SOFTMAX_GRAD : adb200::EPI_SOFTMAX, c10::nullopt, c2, aux, alpha, 0.0, error_flag,
            128, mask, drop_p, seed, step);
}

// Y = A . W^T (+ bias) where W [N, K] is split by rows into `world` equal shards that live in the owners' symmetric
// memory: every B tile is fetched from its owner by a TMA load over NVLink inside the GEMM (no gathered copy of W).
// shard_ptrs: one device address per owner (host list), each a contiguous bf16 [N / world, K] block.
void gemm_gathered_b(const Tensor& a_, const std::vector<int64_t>& shard_ptrs, int64_t rows_per_shard, Tensor c_, int64_t epilogue,
                     const optional<Tensor>& bias, Tensor error_flag, int64_t bn) {
  const c10::cuda::CUDAGuard guard(a_.device());
  Tensor a = as4d(a_), c = as4d(c_);
  const int world = (int)shard_ptrs.size();
  TORCH_CHECK(world >= 1 && world <= 8, "1 to 8 shards");
  const int M = a.size(2), K = a.size(3);
  const int N = (int)rows_per_shard * world;
  TORCH_CHECK(a.size(0) == 1 && a.size(1) == 1, "the gathered-weight GEMM is not batched");
  TORCH_CHECK(c.size(2) == M && c.size(3) == N && c.stride(3) == 1, "output shape mismatch");
  if (bn <= 0) bn = rows_per_shard % 256 == 0 ? 256 : (rows_per_shard % 128 == 0 ? 128 : 64);
  TORCH_CHECK(rows_per_shard % bn == 0, "rows per shard must be a multiple of the tile width ", bn);
  TORCH_CHECK(K % 8 == 0, "K must be a multiple of 8");
  CUtensorMap tmA = make_map(a, 128);
  adb200::TmapArray tmB;
  for (int s = 0; s < 8; ++s) {
    const int src = s < world ? s : 0;
    cuuint64_t dims[4] = {(cuuint64_t)K, (cuuint64_t)rows_per_shard, 1, 1};
    cuuint64_t strides[3] = {(cuuint64_t)K * 2, (cuuint64_t)K * 2 * rows_per_shard, (cuuint64_t)K * 2 * rows_per_shard};
    cuuint32_t box[4] = {64, (cuuint32_t)bn, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = encode_fn()(&tmB.m[s], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, reinterpret_cast<void*>(shard_ptrs[src]), dims, strides, box,
                             estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TORCH_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed for shard ", s, " with code ", (int)r);
  }
  adb200::GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.batch_lo = 1; p.batch_hi = 1;
  p.C = c.data_ptr(); p.ldc = c.stride(2); p.strideC_lo = 0; p.strideC_hi = 0;
  p.vec_ok = rows_aligned(c);
  p.c_is_fp32 = c.scalar_type() == at::kFloat;
  p.epilogue = (int)epilogue; p.alpha = 1.0f; p.beta = 0.0f;
  p.bias = nullptr; p.C2 = nullptr; p.aux = nullptr;
  if (epilogue == adb200::EPI_BIAS) {
    TORCH_CHECK(bias.has_value() && bias->scalar_type() == at::kFloat && bias->numel() >= N, "fp32 bias of N entries needed");
    p.bias = bias->data_ptr<float>();
  } else {
    TORCH_CHECK(epilogue == adb200::EPI_NONE, "only the plain and bias epilogues are offered here");
  }
  p.error_flag = error_flag.data_ptr<int>();
  p.b_shard_rows = (int)rows_per_shard;
  cudaError_t e = adb200::launch_gemm(tmA, tmB, p, (int)bn, false, false, num_sms(), at::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "GEMM launch failed: ", cudaGetErrorString(e));
}

// dX = dY . W where W [N_out, K_in] is split by rows into `world` equal shards in the owners' memories (the input gradient of
// gemm_gathered_b's layer): W is the MN-major B operand and every 64-row K block is fetched from the owner of those rows.
void gemm_gathered_bt(const Tensor& a_, const std::vector<int64_t>& shard_ptrs, int64_t rows_per_shard, int64_t cols, Tensor c_, Tensor error_flag) {
  const c10::cuda::CUDAGuard guard(a_.device());
  Tensor a = as4d(a_), c = as4d(c_);
  const int world = (int)shard_ptrs.size();
  TORCH_CHECK(world >= 1 && world <= 8, "1 to 8 shards");
  const int M = a.size(2), K = a.size(3);
  TORCH_CHECK(K == rows_per_shard * world, "dY width must equal the number of weight rows");
  TORCH_CHECK(a.size(0) == 1 && a.size(1) == 1, "the gathered-weight GEMM is not batched");
  TORCH_CHECK(c.size(2) == M && c.size(3) == cols && c.stride(3) == 1, "output shape mismatch");
  TORCH_CHECK(rows_per_shard % 64 == 0 && cols % 8 == 0, "rows per shard must be a multiple of 64 and the width a multiple of 8");
  const int64_t bn = cols >= 256 ? 256 : (cols > 64 ? 128 : 64);
  CUtensorMap tmA = make_map(a, 128);
  adb200::TmapArray tmB;
  for (int s = 0; s < 8; ++s) {
    const int src = s < world ? s : 0;
    cuuint64_t dims[4] = {(cuuint64_t)cols, (cuuint64_t)rows_per_shard, 1, 1};
    cuuint64_t strides[3] = {(cuuint64_t)cols * 2, (cuuint64_t)cols * 2 * rows_per_shard, (cuuint64_t)cols * 2 * rows_per_shard};
    cuuint32_t box[4] = {64, 64, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = encode_fn()(&tmB.m[s], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, reinterpret_cast<void*>(shard_ptrs[src]), dims, strides, box,
                             estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TORCH_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed for shard ", s, " with code ", (int)r);
  }
  adb200::GemmParams p{};
  p.M = M; p.N = (int)cols; p.K = K; p.batch_lo = 1; p.batch_hi = 1;
  p.C = c.data_ptr(); p.ldc = c.stride(2); p.strideC_lo = 0; p.strideC_hi = 0;
  p.vec_ok = rows_aligned(c);
  p.c_is_fp32 = c.scalar_type() == at::kFloat;
  p.epilogue = adb200::EPI_NONE; p.alpha = 1.0f; p.beta = 0.0f;
  p.error_flag = error_flag.data_ptr<int>();
  p.b_shard_rows = (int)rows_per_shard;
  cudaError_t e = adb200::launch_gemm(tmA, tmB, p, (int)bn, false, true, num_sms(), at::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "GEMM launch failed: ", cudaGetErrorString(e));
}

#define BF(t) reinterpret_cast<__nv_bfloat16*>((t).data_ptr())
#define CBF(t) reinterpret_cast<const __nv_bfloat16*>((t).data_ptr())
#define OPT_BF(t) ((t).has_value() ? reinterpret_cast<__nv_bfloat16*>((t)->data_ptr()) : nullptr)
#define OPT_F(t) ((t).has_value() ? (t)->data_ptr<float>() : nullptr)
#define OPT_I64(t) ((t).has_value() ? (t)->data_ptr<int64_t>() : nullptr)
#define OPT_LL(t) ((t).has_value() ? reinterpret_cast<const long long*>((t)->data_ptr<int64_t>()) : nullptr)
#define STREAM at::cuda::getCurrentCUDAStream()

void ln_fwd(const Tensor& x, const optional<Tensor>& res, const Tensor& gamma, const Tensor& beta, const optional<Tensor>& z, Tensor y,
            Tensor mean, Tensor rstd, double eps, double p_drop, int64_t seed, const optional<Tensor>& step) {
  const int H = x.size(-1), rows = x.numel() / H;
  TORCH_CHECK(H % 8 == 0 && H <= 1024, "layernorm width must be a multiple of 8 and at most 1024");
  adb200::ln_fwd(CBF(x), OPT_BF(res), gamma.data_ptr<float>(), beta.data_ptr<float>(), OPT_BF(z), BF(y), mean.data_ptr<float>(),
                 rstd.data_ptr<float>(), rows, H, (float)eps, (float)p_drop, (uint64_t)seed, OPT_LL(step), STREAM);
}
// part: fp32 scratch of ln_bwd_part_floats(H) elements that must be ZERO on entry (allocate it with zeros once); it is zero again on
// return. dsum (optional, fp32 [H]): column sums of the tensor handed to the layer in front of the residual connection (dx when the dropout
// copy is written, else dz) - the bias gradient of that layer, produced without another pass over the tensor.
void ln_bwd(const Tensor& dy, const Tensor& z, const Tensor& mean, const Tensor& rstd, const Tensor& gamma, const optional<Tensor>& dz_add,
            Tensor dz, const optional<Tensor>& dx, Tensor part, Tensor dgamma, Tensor dbeta, double p_drop, int64_t seed,
            const optional<Tensor>& step, bool accumulate, const optional<Tensor>& dsum) {
  const int H = dy.size(-1), rows = dy.numel() / H;
  TORCH_CHECK(H % 8 == 0 && H <= 1024, "layernorm width must be a multiple of 8 and at most 1024");
  TORCH_CHECK(part.numel() >= adb200::ln_bwd_part_floats(H), "partial buffer too small (ln_bwd_part_floats(H) floats, zero-filled)");
  if (dsum.has_value()) TORCH_CHECK(dsum->scalar_type() == at::kFloat && dsum->numel() >= H, "dsum must be fp32 [H]");
  adb200::ln_bwd(CBF(dy), CBF(z), mean.data_ptr<float>(), rstd.data_ptr<float>(), gamma.data_ptr<float>(), OPT_BF(dz_add), BF(dz),
                 OPT_BF(dx), part.data_ptr<float>(), dgamma.data_ptr<float>(), dbeta.data_ptr<float>(), OPT_F(dsum), rows, H, (float)p_drop,
                 (uint64_t)seed, OPT_LL(step), accumulate ? 1 : 0, STREAM);
}
void embed_sum(const Tensor& word, const Tensor& pos, const Tensor& type, const Tensor& ids, const optional<Tensor>& tt, Tensor z, int64_t S,
               const optional<Tensor>& error_flag) {
  const int H = word.size(1), rows = ids.numel();
  TORCH_CHECK(pos.size(0) >= S, "position table shorter than the sequence");
  adb200::embed_sum(CBF(word), CBF(pos), CBF(type), ids.data_ptr<int64_t>(), OPT_I64(tt), BF(z), rows, (int)S, H, word.size(0), type.size(0),
                    error_flag.has_value() ? error_flag->data_ptr<int>() : nullptr, STREAM);
}
void scatter_add_rows(Tensor dst, const Tensor& idx, const Tensor& src, double scale) {
  adb200::scatter_add_rows(dst.data_ptr<float>(), idx.data_ptr<int64_t>(), CBF(src), idx.numel(), src.size(-1), (float)scale, STREAM);
}
void strided_rowsum(const Tensor& x, Tensor out, int64_t keys, int64_t stride, int64_t count) {
  adb200::strided_rowsum(CBF(x), out.data_ptr<float>(), keys, stride, count, x.size(-1), STREAM);
}
void keyed_colsum(const Tensor& x, const optional<Tensor>& key, Tensor part, Tensor out, int64_t keys, bool accumulate) {
  const int H = x.size(-1), rows = x.numel() / H;
  TORCH_CHECK(H % 8 == 0, "width must be a multiple of 8");
  TORCH_CHECK(part.numel() >= (long long)adb200::colsum_parts(rows) * keys * H, "partial buffer too small");
  adb200::keyed_colsum(CBF(x), OPT_I64(key), part.data_ptr<float>(), out.data_ptr<float>(), rows, H, keys, accumulate ? 1 : 0, STREAM);
}
void gather_rows(const Tensor& src, const Tensor& idx, Tensor out) {
  adb200::gather_rows(CBF(src), idx.data_ptr<int64_t>(), BF(out), idx.numel(), src.size(-1), STREAM);
}
void gather_rows_f32(const Tensor& src, const Tensor& idx, Tensor out) {
  TORCH_CHECK(src.scalar_type() == at::kFloat && src.is_contiguous() && src.size(-1) % 8 == 0, "fp32 contiguous table, width a multiple of 8");
  adb200::gather_rows_f32(src.data_ptr<float>(), idx.data_ptr<int64_t>(), BF(out), idx.numel(), src.size(-1), STREAM);
}
// dst[idx[r]] += src[r] (fp32 both); every index must be a row of dst.
void scatter_add_rows_f32(Tensor dst, const Tensor& idx, const Tensor& src) {
  TORCH_CHECK(dst.is_cuda() && dst.dim() == 2 && dst.is_contiguous() && dst.scalar_type() == at::kFloat && src.is_contiguous() &&
              src.scalar_type() == at::kFloat && idx.is_contiguous() && idx.scalar_type() == at::kLong && src.numel() == idx.numel() * dst.size(1),
              "dst [V, H] and src [n, H] must be contiguous fp32, idx int64 [n]");
  adb200::scatter_add_rows_f32(dst.data_ptr<float>(), idx.data_ptr<int64_t>(), src.data_ptr<float>(), idx.numel(), dst.size(1), STREAM);
}
// One step of a whole-sequence LSTM layer: gates bf16 [B, 4S] (i, j, f, o), c fp32 [B, S], h / dh / dgates bf16; S a multiple of 4.
void check_lstm_seq(const Tensor& gates, const Tensor& c_prev, const Tensor& c, const Tensor& h) {
  const int64_t n = c_prev.numel();
  for (const Tensor& t : {gates, c_prev, c, h})
    TORCH_CHECK(t.is_cuda() && t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0, "contiguous 16-byte aligned CUDA tensors needed");
  TORCH_CHECK(c_prev.dim() == 2 && c_prev.size(1) % 4 == 0 && gates.numel() == 4 * n && c.numel() == n && h.numel() == n &&
              gates.scalar_type() == at::kBFloat16 && h.scalar_type() == at::kBFloat16 && c_prev.scalar_type() == at::kFloat && c.scalar_type() == at::kFloat,
              "gates bf16 [B, 4S], c fp32 [B, S], h bf16 [B, S], S a multiple of 4");
}
void lstm_seq_fwd(const Tensor& gates, const Tensor& c_prev, Tensor c, Tensor h, double forget_bias) {
  check_lstm_seq(gates, c_prev, c, h);
  adb200::lstm_seq_fwd(CBF(gates), c_prev.data_ptr<float>(), c.data_ptr<float>(), BF(h), c_prev.size(0), c_prev.size(1), (float)forget_bias, STREAM);
}
void lstm_seq_bwd(const Tensor& gates, const Tensor& c_prev, const Tensor& c, const Tensor& dh, const optional<Tensor>& dc_next, Tensor dgates,
                  Tensor dc_prev, double forget_bias) {
  check_lstm_seq(gates, c_prev, c, dh);
  check_lstm_seq(dgates, dc_prev, c, dh);
  adb200::lstm_seq_bwd(CBF(gates), c_prev.data_ptr<float>(), c.data_ptr<float>(), CBF(dh), OPT_F(dc_next), BF(dgates), dc_prev.data_ptr<float>(),
                       c_prev.size(0), c_prev.size(1), (float)forget_bias, STREAM);
}
void scatter_add_rows_bf16(Tensor dst, const Tensor& idx, const Tensor& src) {
  adb200::scatter_add_rows_bf16(BF(dst), idx.data_ptr<int64_t>(), CBF(src), idx.numel(), src.size(-1), STREAM);
}
void softmax_fwd(const Tensor& x, const optional<Tensor>& mask, Tensor p, const optional<Tensor>& p_drop, double scale, double pd,
                 int64_t seed, const optional<Tensor>& step) {
  const int S = x.size(-1);
  TORCH_CHECK(adb200::softmax_supported(S) && x.dim() == 4, "scores must be [B, heads, S, S] with S in {64, 128, 256, 512, 1024}");
  const long long rows = x.numel() / S;
  adb200::softmax_fwd(CBF(x), OPT_F(mask), BF(p), OPT_BF(p_drop), rows, S, (int)(x.size(1) * x.size(2)), (float)scale, (float)pd,
                      (uint64_t)seed, OPT_LL(step), STREAM);
}
void softmax_bwd(Tensor dp, const Tensor& p, double scale, double pd, int64_t seed, const optional<Tensor>& step) {
  const int S = p.size(-1);
  adb200::softmax_bwd(BF(dp), CBF(p), p.numel() / S, S, (float)scale, (float)pd, (uint64_t)seed, OPT_LL(step), STREAM);
}
// Fused self-attention over the projection qkv [B * S, 3 * heads * 64] (bf16; q, k, v side by side): writes ctx [B * S, heads * 64]
// and lse [B, heads, S], with dropout also the decisions (keep). mask: additive fp32 [B, S] over the keys.
adb200::AttnParams attn_params(const Tensor& qkv, const optional<Tensor>& mask, const Tensor& ctx, const Tensor& lse, int64_t B, int64_t S,
                               int64_t heads, double scale, double pd, int64_t seed, const optional<Tensor>& step, Tensor error_flag,
                               const optional<Tensor>& keep) {
  const int64_t H = heads * 64;
  TORCH_CHECK(B > 0 && heads > 0 && S > 0 && S <= 1024, "attention takes 1 to 1024 tokens");
  TORCH_CHECK(!(pd > 0) || S % 4 == 0, "attention with dropout takes a multiple of 4 tokens (one random number decides four neighbouring scores)");
  TORCH_CHECK(qkv.is_cuda() && qkv.scalar_type() == at::kBFloat16 && qkv.is_contiguous() && qkv.numel() == B * S * 3 * H, "qkv must be contiguous bf16 [B * S, 3 * heads * 64]");
  TORCH_CHECK(ctx.scalar_type() == at::kBFloat16 && ctx.is_contiguous() && ctx.numel() == B * S * H, "ctx must be contiguous bf16 [B * S, heads * 64]");
  TORCH_CHECK(lse.scalar_type() == at::kFloat && lse.is_contiguous() && lse.numel() == B * heads * S, "lse must be fp32 [B, heads, S]");
  TORCH_CHECK(reinterpret_cast<uintptr_t>(ctx.data_ptr()) % 16 == 0, "ctx must be 16-byte aligned");
  if (mask.has_value()) TORCH_CHECK(mask->scalar_type() == at::kFloat && mask->is_contiguous() && mask->numel() == B * S, "mask must be fp32 [B, S]");
  adb200::AttnParams p{};
  p.B = (int)B; p.S = (int)S; p.heads = (int)heads;
  p.scale = (float)scale;
  p.mask = OPT_F(mask);
  p.lse = lse.data_ptr<float>();
  p.drop_p = (float)pd; p.seed = (unsigned long long)seed; p.step = OPT_LL(step);
  if (pd > 0) {
    TORCH_CHECK(keep.has_value() && keep->scalar_type() == at::kInt && keep->is_contiguous() && keep->numel() >= B * heads * S * adb200::attn_keep_words((int)S),
                "dropout needs int32 [B, heads, S, 4 * ceil(S / 128)] for its decisions");
    p.keep = reinterpret_cast<uint32_t*>(keep->data_ptr<int>());
  }
  p.ctx = reinterpret_cast<__nv_bfloat16*>(ctx.data_ptr());
  p.error_flag = error_flag.data_ptr<int>();
  return p;
}
// [B, heads, S, 64] view of 64 columns per head starting at column `off` of a [B * S, ld] matrix
CUtensorMap head_map(const Tensor& t, int64_t B, int64_t S, int64_t heads, int64_t ld, int64_t off, int rows = 128) {
  return make_map(t.view({B, S, ld}).narrow(2, off, heads * 64).view({B, S, heads, 64}).permute({0, 2, 1, 3}), rows);
}
void attn_fwd(const Tensor& qkv, const optional<Tensor>& mask, Tensor ctx, Tensor lse, int64_t B, int64_t S, int64_t heads, double scale,
              double pd, int64_t seed, const optional<Tensor>& step, Tensor error_flag, const optional<Tensor>& keep) {
  const c10::cuda::CUDAGuard guard(qkv.device());
  const adb200::AttnParams p = attn_params(qkv, mask, ctx, lse, B, S, heads, scale, pd, seed, step, error_flag, keep);
  const int64_t H = heads * 64;
  cudaError_t e = adb200::launch_attn_fwd(head_map(qkv, B, S, heads, 3 * H, 0), head_map(qkv, B, S, heads, 3 * H, H),
                                          head_map(qkv, B, S, heads, 3 * H, 2 * H), p, STREAM);
  TORCH_CHECK(e == cudaSuccess, "attention launch failed: ", cudaGetErrorString(e));
}
// dqkv = gradient of qkv given dctx, with ctx, lse and keep as the forward pass left them. delta: scratch of lse's shape.
void attn_bwd(const Tensor& qkv, const optional<Tensor>& mask, const Tensor& ctx, const Tensor& dctx, const Tensor& lse, Tensor delta, Tensor dqkv,
              int64_t B, int64_t S, int64_t heads, double scale, double pd, Tensor error_flag, const optional<Tensor>& keep) {
  const c10::cuda::CUDAGuard guard(qkv.device());
  adb200::AttnParams p = attn_params(qkv, mask, ctx, lse, B, S, heads, scale, pd, 0, c10::nullopt, error_flag, keep);
  TORCH_CHECK(delta.scalar_type() == at::kFloat && delta.is_contiguous() && delta.numel() == lse.numel(), "delta must match lse");
  p.delta = delta.data_ptr<float>();
  const int64_t H = heads * 64;
  TORCH_CHECK(dctx.scalar_type() == at::kBFloat16 && dctx.is_contiguous() && dctx.numel() == B * S * H, "dctx must match ctx");
  TORCH_CHECK(dqkv.scalar_type() == at::kBFloat16 && dqkv.is_contiguous() && dqkv.numel() == qkv.numel(), "dqkv must match qkv");
  p.dctx = CBF(dctx);
  adb200::AttnGradMaps grads;
  for (int i = 0; i < 3; ++i) grads.m[i] = head_map(dqkv, B, S, heads, 3 * H, i * H, 32);
  cudaError_t e = adb200::launch_attn_bwd(head_map(qkv, B, S, heads, 3 * H, 0), head_map(qkv, B, S, heads, 3 * H, H),
                                          head_map(qkv, B, S, heads, 3 * H, 2 * H), head_map(dctx, B, S, heads, H, 0), grads, p, num_sms(), STREAM);
  TORCH_CHECK(e == cudaSuccess, "attention launch failed: ", cudaGetErrorString(e));
}
void xent(Tensor logits, const Tensor& labels, const optional<Tensor>& weights, Tensor denom, Tensor loss_sum, int64_t V, double loss_scale,
          bool compute_denom, double eps) {
  const int ld = logits.size(-1), rows = logits.numel() / ld;
  if (compute_denom) {
    TORCH_CHECK(weights.has_value(), "weights needed to compute the denominator");
    adb200::weight_sum(weights->data_ptr<float>(), rows, denom.data_ptr<float>(), (float)eps, STREAM);
  }
  adb200::xent(BF(logits), labels.data_ptr<int64_t>(), OPT_F(weights), denom.data_ptr<float>(), loss_sum.data_ptr<float>(), rows, (int)V, ld,
               (float)loss_scale, STREAM);
}
void gelu_bwd(const Tensor& dy, const Tensor& u, Tensor dx) { adb200::gelu_bwd(CBF(dy), CBF(u), BF(dx), u.numel(), STREAM); }
void tanh_bwd(const Tensor& dy, const Tensor& y, Tensor dx) { adb200::tanh_bwd(CBF(dy), CBF(y), BF(dx), y.numel(), STREAM); }
void add_bf16(const Tensor& a, const Tensor& b, Tensor out) {
  TORCH_CHECK(a.numel() % 8 == 0, "length must be a multiple of 8");
  adb200::add_bf16(CBF(a), CBF(b), BF(out), a.numel(), STREAM);
}
void adam_update(Tensor p, const Tensor& g, Tensor m, Tensor v, const optional<Tensor>& p16, const Tensor& lr, double b1, double b2, double eps,
                 double wd, bool decoupled, const Tensor& step, double grad_scale) {
  adb200::adam_update(p.data_ptr<float>(), g.data_ptr<float>(), m.data_ptr<float>(), v.data_ptr<float>(), OPT_BF(p16), p.numel(),
                      lr.data_ptr<float>(), (float)b1, (float)b2, (float)eps, (float)wd, decoupled ? 1 : 0,
                      reinterpret_cast<const long long*>(step.data_ptr<int64_t>()), (float)grad_scale, STREAM);
}
void sgd_update(Tensor p, const Tensor& g, const optional<Tensor>& mom, const optional<Tensor>& p16, const Tensor& lr, double momentum,
                double dampening, double wd, bool nesterov, const Tensor& step, double grad_scale) {
  adb200::sgd_update(p.data_ptr<float>(), g.data_ptr<float>(), OPT_F(mom), OPT_BF(p16), p.numel(), lr.data_ptr<float>(), (float)momentum,
                     (float)dampening, (float)wd, nesterov ? 1 : 0, reinterpret_cast<const long long*>(step.data_ptr<int64_t>()),
                     (float)grad_scale, STREAM);
}
void adagrad_update(Tensor p, const Tensor& g, Tensor acc, const optional<Tensor>& p16, const Tensor& lr, double eps, double wd, double grad_scale) {
  adb200::adagrad_update(p.data_ptr<float>(), g.data_ptr<float>(), acc.data_ptr<float>(), OPT_BF(p16), p.numel(), lr.data_ptr<float>(),
                         (float)eps, (float)wd, (float)grad_scale, STREAM);
}
void sparse_rows_update(Tensor p, const optional<Tensor>& s1, const optional<Tensor>& s2, const optional<Tensor>& p16, const Tensor& rows,
                        const Tensor& g, int64_t kind, const Tensor& lr, double b1, double b2, double eps, const optional<Tensor>& step,
                        double grad_scale) {
  TORCH_CHECK(p.dim() == 2 && p.is_contiguous() && p.scalar_type() == at::kFloat, "parameter must be a contiguous fp32 [V, H] table");
  TORCH_CHECK(g.scalar_type() == at::kFloat && g.is_contiguous() && g.dim() == 2 && g.size(0) == rows.numel() && g.size(1) == p.size(1),
              "gradient rows must be fp32 [n, H]");
  TORCH_CHECK(rows.scalar_type() == at::kLong && rows.is_contiguous(), "row ids must be int64");
  TORCH_CHECK(kind == 0 || (s1.has_value() && s1->sizes() == p.sizes()), "state 1 must match the table");
  TORCH_CHECK(kind != 1 || (s2.has_value() && s2->sizes() == p.sizes() && step.has_value()), "lazy Adam needs both moments and the step");
  adb200::sparse_rows_update(p.data_ptr<float>(), OPT_F(s1), OPT_F(s2), OPT_BF(p16), rows.data_ptr<int64_t>(), g.data_ptr<float>(),
                             (int)rows.numel(), (int)p.size(1), p.size(0), (int)kind, lr.data_ptr<float>(), (float)b1, (float)b2,
                             (float)eps, OPT_LL(step), (float)grad_scale, STREAM);
}
// Owner-side update of the flagged rows of a shard (p, g, s1, s2: fp32 [rows, H]; flags: uint8 [rows]); clears what it used.
void flagged_rows_update(Tensor p, const optional<Tensor>& s1, const optional<Tensor>& s2, const optional<Tensor>& p16, Tensor g, Tensor flags,
                         int64_t rows, int64_t H, int64_t kind, const Tensor& lr, double b1, double b2, double eps, const optional<Tensor>& step) {
  TORCH_CHECK(p.scalar_type() == at::kFloat && g.scalar_type() == at::kFloat && flags.scalar_type() == at::kByte, "fp32 table / gradient, uint8 flags");
  TORCH_CHECK(p.numel() >= rows * H && g.numel() >= rows * H && flags.numel() >= rows, "buffers smaller than rows x H");
  TORCH_CHECK(kind == 0 || s1.has_value(), "state 1 needed");
  TORCH_CHECK(kind != 1 || (s2.has_value() && step.has_value()), "Adam needs both moments and the step");
  adb200::flagged_rows_update(p.data_ptr<float>(), OPT_F(s1), OPT_F(s2), OPT_BF(p16), g.data_ptr<float>(), flags.data_ptr<uint8_t>(), rows, (int)H,
                              (int)kind, lr.data_ptr<float>(), (float)b1, (float)b2, (float)eps, OPT_LL(step), STREAM);
}
void lstm_cell_fwd(const Tensor& gates, const Tensor& c_prev, Tensor c, Tensor h, double forget_bias) {
  const int B = c_prev.size(0), S = c_prev.size(1);
  TORCH_CHECK(gates.scalar_type() == at::kFloat && gates.size(1) == 4 * S && gates.is_contiguous(), "gates must be fp32 [B, 4S]");
  adb200::lstm_cell_fwd(gates.data_ptr<float>(), c_prev.data_ptr<float>(), c.data_ptr<float>(), BF(h), B, S, (float)forget_bias, STREAM);
}
void lstm_cell_bwd(const Tensor& gates, const Tensor& c_prev, const Tensor& c, const Tensor& dh, const optional<Tensor>& dc_next,
                   Tensor dgates, Tensor dc_prev, double forget_bias) {
  const int B = c_prev.size(0), S = c_prev.size(1);
  adb200::lstm_cell_bwd(gates.data_ptr<float>(), c_prev.data_ptr<float>(), c.data_ptr<float>(), dh.data_ptr<float>(), OPT_F(dc_next),
                        dgates.data_ptr<float>(), dc_prev.data_ptr<float>(), B, S, (float)forget_bias, STREAM);
}
void sumsq(const Tensor& x, Tensor acc, double weight) { adb200::sumsq(x.data_ptr<float>(), x.numel(), acc.data_ptr<float>(), (float)weight, STREAM); }
void clip_scale(Tensor x, const Tensor& acc, double max_norm) { adb200::clip_scale(x.data_ptr<float>(), x.numel(), acc.data_ptr<float>(), (float)max_norm, STREAM); }
// Batch-norm over a channels-last matrix x [rows, C] (training mode statistics), optional residual addend and fused ReLU:
// y = relu?(bn(x) + res). `keep` (uint8, one byte per 8 channels) receives which outputs a fused ReLU let through. `sums`
// (optional, fp32 [2, C]) holds sum x and sum x^2 already (from the convolution's epilogue).
void bn_fwd(const Tensor& x, const Tensor& gamma, const Tensor& beta, const optional<Tensor>& res, Tensor y, Tensor mean, Tensor rstd,
            double eps, bool relu, const optional<Tensor>& sums_in, const optional<Tensor>& run_mean, const optional<Tensor>& run_var,
            const optional<Tensor>& batches, double momentum, const optional<Tensor>& keep) {
  const int C = x.size(-1), rows = x.numel() / C;
  float* rm = nullptr; float* rv = nullptr; long long* nb = nullptr;
  if (run_mean.has_value()) {
    TORCH_CHECK(run_var.has_value() && run_mean->scalar_type() == at::kFloat && run_var->scalar_type() == at::kFloat && run_mean->numel() == C &&
                run_var->numel() == C && run_mean->is_contiguous() && run_var->is_contiguous(), "running statistics must be fp32 [C]");
    rm = run_mean->data_ptr<float>(); rv = run_var->data_ptr<float>();
  }
  if (batches.has_value()) nb = reinterpret_cast<long long*>(batches->data_ptr<int64_t>());
  TORCH_CHECK(C % 8 == 0 && x.is_contiguous() && x.scalar_type() == at::kBFloat16, "x must be contiguous bf16 [.., C], C % 8 == 0");
  TORCH_CHECK(y.is_contiguous() && y.numel() == x.numel() && mean.numel() == C && rstd.numel() == C && gamma.numel() == C && beta.numel() == C,
              "output and per-channel tensors must match x");
  if (res.has_value()) TORCH_CHECK(res->is_contiguous() && res->numel() == x.numel() && res->scalar_type() == at::kBFloat16, "residual must match x");
  uint8_t* kp = nullptr;
  if (keep.has_value()) {
    TORCH_CHECK(keep->scalar_type() == at::kByte && keep->is_contiguous() && keep->numel() * 8 == x.numel(), "keep must hold one byte per 8 elements");
    kp = keep->data_ptr<uint8_t>();
  }
  if (sums_in.has_value()) {
    TORCH_CHECK(sums_in->scalar_type() == at::kFloat && sums_in->numel() == 2 * C && sums_in->is_contiguous(), "sums must be fp32 [2, C]");
    adb200::bn_fwd(CBF(x), gamma.data_ptr<float>(), beta.data_ptr<float>(), OPT_BF(res), BF(y), kp, mean.data_ptr<float>(),
                   rstd.data_ptr<float>(), nullptr, sums_in->data_ptr<float>(), rows, C, (float)eps, relu ? 1 : 0, 1, rm, rv, nb, (float)momentum, STREAM);
    return;
  }
  Tensor part = at::empty({(int64_t)adb200::bn_parts(rows, C) * 2 * C}, x.options().dtype(at::kFloat));
  Tensor sums = at::empty({2 * C}, x.options().dtype(at::kFloat));
  adb200::bn_fwd(CBF(x), gamma.data_ptr<float>(), beta.data_ptr<float>(), OPT_BF(res), BF(y), kp, mean.data_ptr<float>(), rstd.data_ptr<float>(),
                 part.data_ptr<float>(), sums.data_ptr<float>(), rows, C, (float)eps, relu ? 1 : 0, 0, rm, rv, nb, (float)momentum,
                 STREAM);
}
// The same from a logical [N, C, H, W] tensor with every view and allocation made here: an eager step is bounded by host time, and the
// Python steps around a call cost more than its launches. Returns x as it was read (bf16 [N, H, W, C]), y (logical [N, C, H, W]), the
// keep bytes (with relu), mean, rstd and gamma in fp32.
std::tuple<Tensor, Tensor, optional<Tensor>, Tensor, Tensor, Tensor> bn_fwd_nchw(const Tensor& x, const Tensor& gamma, const Tensor& beta,
                                                                                 const optional<Tensor>& res, double eps, bool relu,
                                                                                 const optional<Tensor>& sums, const optional<Tensor>& run_mean,
                                                                                 const optional<Tensor>& run_var, const optional<Tensor>& batches,
                                                                                 double momentum) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 4, "x must be a CUDA [N, C, H, W] tensor");
  auto nhwc = [](const Tensor& t) { return t.permute({0, 2, 3, 1}).to(at::kBFloat16).contiguous(); };
  const Tensor xh = nhwc(x);
  const Tensor g32 = gamma.detach().to(at::kFloat).contiguous(), b32 = beta.detach().to(at::kFloat).contiguous();
  Tensor y = at::empty_like(xh);
  Tensor mean = at::empty({xh.size(3)}, xh.options().dtype(at::kFloat)), rstd = at::empty_like(mean);
  optional<Tensor> r, keep;
  if (res.has_value()) r = nhwc(*res);
  if (relu) keep = at::empty({xh.numel() / 8}, xh.options().dtype(at::kByte));
  bn_fwd(xh, g32, b32, r, y, mean, rstd, eps, relu, sums, run_mean, run_var, batches, momentum, keep);
  return {xh, y.permute({0, 3, 1, 2}), keep, mean, rstd, g32};
}
// y = relu?(x * scale + shift (+ res)) over a channels-last matrix [rows, C] with the running statistics (evaluation mode).
void bn_eval(const Tensor& x, const optional<Tensor>& res, Tensor y, const Tensor& gamma, const Tensor& beta, const Tensor& mean,
             const Tensor& var, double eps, bool relu) {
  const int C = x.size(-1), rows = x.numel() / C;
  TORCH_CHECK(C % 8 == 0 && C <= 4096 && x.is_contiguous() && x.scalar_type() == at::kBFloat16 && y.is_contiguous() && y.numel() == x.numel(),
              "x and y must be contiguous bf16 [.., C], C % 8 == 0, C <= 4096");
  if (res.has_value()) TORCH_CHECK(res->is_contiguous() && res->numel() == x.numel() && res->scalar_type() == at::kBFloat16, "residual must match x");
  for (const Tensor& t : {gamma, beta, mean, var})
    TORCH_CHECK(t.scalar_type() == at::kFloat && t.numel() == C && t.is_contiguous(), "batch-norm parameters must be fp32 [C]");
  if (x.numel() == 0) return;
  adb200::bn_eval(CBF(x), OPT_BF(res), BF(y), gamma.data_ptr<float>(), beta.data_ptr<float>(), mean.data_ptr<float>(), var.data_ptr<float>(),
                  (float)eps, rows, C, relu ? 1 : 0, STREAM);
}
// Per-channel sum and sum of squares [2, C] of a channels-last matrix, as a convolution's epilogue leaves them.
Tensor bn_sums(const Tensor& x) {
  const int C = x.size(-1), rows = x.numel() / std::max(C, 1);
  TORCH_CHECK(C > 0 && C % 8 == 0 && rows > 0 && x.is_contiguous() && x.scalar_type() == at::kBFloat16, "x must be contiguous bf16 [.., C], C % 8 == 0");
  Tensor part = at::empty({(int64_t)adb200::bn_parts(rows, C) * 2 * C}, x.options().dtype(at::kFloat));
  Tensor sums = at::empty({2, C}, x.options().dtype(at::kFloat));
  adb200::bn_sums(CBF(x), part.data_ptr<float>(), sums.data_ptr<float>(), rows, C, STREAM);
  return sums;
}
// Returns [dbeta, dgamma] stacked as a [2, C] fp32 tensor; writes dx and (optional) dres = dy masked by the ReLU.
// dgamma_acc / dbeta_acc (optional, fp32 [C]): the batch-norm parameters' gradient buffers; the sums are added into them.
// add (optional, bf16, logical [N, C, H, W] with x [N, H, W, C]): another gradient of x, added to dx. A channel slice of a
// channels-last tensor, whose rows lie a constant distance apart, is read in place.
Tensor bn_bwd(const Tensor& dy, const Tensor& x, const optional<Tensor>& keep, const Tensor& mean, const Tensor& rstd, const Tensor& gamma, Tensor dx,
              const optional<Tensor>& dres, bool relu, const optional<Tensor>& dgamma_acc, const optional<Tensor>& dbeta_acc,
              const optional<Tensor>& add) {
  const int C = x.size(-1), rows = x.numel() / C;
  TORCH_CHECK(C % 8 == 0 && C <= 16384 && x.is_contiguous() && dy.is_contiguous() && dx.is_contiguous() && dy.numel() == x.numel() && dx.numel() == x.numel(),
              "dy, x, dx must be contiguous bf16 [.., C] of one shape, C % 8 == 0");
  if (dres.has_value()) TORCH_CHECK(dres->is_contiguous() && dres->numel() == x.numel() && dres->scalar_type() == at::kBFloat16, "dres must match x");
  Tensor other;
  int64_t other_ld = 0;
  if (add.has_value()) {
    TORCH_CHECK(x.dim() == 4 && add->is_cuda() && add->scalar_type() == at::kBFloat16 && add->dim() == 4 && add->size(0) == x.size(0) &&
                add->size(1) == C && add->size(2) == x.size(1) && add->size(3) == x.size(2), "the addend must be bf16 [N, C, H, W]");
    other = add->permute({0, 2, 3, 1});
    other_ld = C;
    const int64_t pixels[3] = {(int64_t)x.size(1) * x.size(2), x.size(2), 1};      // pixels between two neighbours of a dimension
    for (int d = 2; d >= 0; --d)
      if (x.size(d) > 1) { other_ld = other.stride(d) / pixels[d]; break; }
    bool regular = other.stride(3) == 1 && other_ld >= C && other_ld % 8 == 0 && reinterpret_cast<uintptr_t>(other.data_ptr()) % 16 == 0;
    for (int d = 0; d < 3; ++d) regular &= x.size(d) <= 1 || other.stride(d) == other_ld * pixels[d];
    if (!regular) { other = other.clone(at::MemoryFormat::Contiguous); other_ld = C; }
  }
  TORCH_CHECK(!relu || (keep.has_value() && keep->scalar_type() == at::kByte && keep->is_contiguous() && keep->numel() * 8 == x.numel()),
              "the forward pass's keep bytes are needed with a fused ReLU");
  // partial sums: a per-device scratch that the kernels keep zero between calls (they add into it and clear what they read);
  // batch-norm backward calls of one device are issued on one stream
  static std::unordered_map<int, Tensor> scratch;
  Tensor& part = scratch[x.get_device()];
  if (!part.defined() || part.numel() < adb200::bn_bwd_part_floats(C))
    part = at::zeros({(int64_t)adb200::bn_bwd_part_floats(std::max(C, 4096))}, x.options().dtype(at::kFloat));
  Tensor sums = at::empty({5, C}, x.options().dtype(at::kFloat));              // [dbeta, dgamma, A, B, K]
  adb200::bn_bwd(CBF(dy), CBF(x), relu ? keep->data_ptr<uint8_t>() : nullptr, mean.data_ptr<float>(), rstd.data_ptr<float>(), gamma.data_ptr<float>(), BF(dx), OPT_BF(dres),
                 part.data_ptr<float>(), sums.data_ptr<float>(), sums.data_ptr<float>() + 2 * C, rows, C, relu ? 1 : 0, OPT_F(dgamma_acc),
                 OPT_F(dbeta_acc), other.defined() ? CBF(other) : nullptr, other_ld, STREAM);
  return sums.narrow(0, 0, 2);
}
// code: uint8 [N, Ho, Wo, C], the window position of each output's first maximum
void maxpool_fwd(const Tensor& x, Tensor y, Tensor code, int64_t k, int64_t stride, int64_t pad) {
  TORCH_CHECK(x.dim() == 4 && x.is_contiguous() && x.size(3) % 8 == 0 && x.scalar_type() == at::kBFloat16, "x must be contiguous bf16 [N, H, W, C]");
  TORCH_CHECK(y.is_contiguous() && code.is_contiguous() && code.scalar_type() == at::kByte && code.numel() == y.numel() && k * k < 255 &&
              y.size(0) == x.size(0) && y.size(3) == x.size(3), "y / code must be [N, Ho, Wo, C]");
  adb200::maxpool_fwd(CBF(x), BF(y), code.data_ptr<uint8_t>(), x.size(0), x.size(1), x.size(2), x.size(3), k, stride, pad, y.size(1),
                      y.size(2), STREAM);
}
void maxpool_bwd(const Tensor& code, const Tensor& dy, Tensor dx, int64_t k, int64_t stride, int64_t pad) {
  TORCH_CHECK(dx.dim() == 4 && dx.is_contiguous() && dy.is_contiguous() && code.is_contiguous() && code.numel() == dy.numel() &&
              dx.size(3) % 8 == 0, "dx [N, H, W, C], dy / code [N, Ho, Wo, C], contiguous");
  adb200::maxpool_bwd(code.data_ptr<uint8_t>(), CBF(dy), BF(dx), dx.size(0), dx.size(1), dx.size(2), dx.size(3), k, stride, pad, dy.size(1),
                      dy.size(2), STREAM);
}
void im2col(const Tensor& x, Tensor cols, int64_t KH, int64_t KW, int64_t stride, int64_t pad) {
  TORCH_CHECK(x.dim() == 4 && x.is_contiguous() && x.scalar_type() == at::kBFloat16 && x.size(3) % 8 == 0, "x must be contiguous bf16 [N, H, W, C], C % 8 == 0");
  const int N = x.size(0), H = x.size(1), W = x.size(2), C = x.size(3);
  const int Ho = (H + 2 * pad - KH) / stride + 1, Wo = (W + 2 * pad - KW) / stride + 1;
  TORCH_CHECK(cols.numel() == (int64_t)N * Ho * Wo * KH * KW * C, "cols has the wrong size");
  adb200::im2col(CBF(x), BF(cols), N, H, W, C, KH, KW, stride, pad, Ho, Wo, STREAM);
}
void col2im(const Tensor& dcols, Tensor dx, int64_t KH, int64_t KW, int64_t stride, int64_t pad) {
  TORCH_CHECK(dx.dim() == 4 && dx.is_contiguous() && dx.scalar_type() == at::kBFloat16 && dx.size(3) % 8 == 0, "dx must be contiguous bf16 [N, H, W, C]");
  const int N = dx.size(0), H = dx.size(1), W = dx.size(2), C = dx.size(3);
  const int Ho = (H + 2 * pad - KH) / stride + 1, Wo = (W + 2 * pad - KW) / stride + 1;
  TORCH_CHECK(dcols.numel() == (int64_t)N * Ho * Wo * KH * KW * C, "dcols has the wrong size");
  adb200::col2im(CBF(dcols), BF(dx), N, H, W, C, KH, KW, stride, pad, Ho, Wo, STREAM);
}
// Image [N, C, H, W] (any strides, fp32 or bf16, C <= 8) -> bf16 [N, Hp, Wp, 8] with the pixels at offset (pad, pad) and zeros elsewhere.
void pad_image8(const Tensor& x, Tensor xp, int64_t pad) {
  TORCH_CHECK(x.dim() == 4 && x.size(1) <= 8 && (x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16), "x must be [N, C<=8, H, W] fp32 or bf16");
  TORCH_CHECK(xp.dim() == 4 && xp.size(3) == 8 && xp.is_contiguous() && xp.scalar_type() == at::kBFloat16 && xp.size(0) == x.size(0) &&
              xp.size(1) >= x.size(2) + pad && xp.size(2) >= x.size(3) + pad, "xp must be contiguous bf16 [N, Hp, Wp, 8]");
  adb200::pad_image8(x.data_ptr(), x.scalar_type() == at::kFloat ? 1 : 0, x.stride(0), x.stride(1), x.stride(2), x.stride(3), x.size(0),
                     x.size(1), x.size(2), x.size(3), BF(xp), xp.size(1), xp.size(2), (int)pad, STREAM);
}
// Bias gradient of a convolution over channels-last dy [.., C]: out (fp32 [C]) = column sums of dy, or of dy masked by y > 0
// when the convolution had a fused ReLU, in which case the masked gradient is also written to dx. accumulate: out += sums.
void relu_bwd_colsum(const Tensor& dy, const optional<Tensor>& y, const optional<Tensor>& dx, Tensor out, bool accumulate) {
  const int C = dy.size(-1), rows = dy.numel() / C;
  TORCH_CHECK(C % 8 == 0 && dy.is_contiguous() && dy.scalar_type() == at::kBFloat16 && out.scalar_type() == at::kFloat && out.numel() == C &&
              out.is_contiguous(), "dy must be contiguous bf16 [.., C] (C % 8 == 0), out fp32 [C]");
  TORCH_CHECK(y.has_value() == dx.has_value(), "y and dx come together");
  if (y.has_value()) TORCH_CHECK(y->is_contiguous() && dx->is_contiguous() && y->numel() == dy.numel() && dx->numel() == dy.numel(), "y, dx must match dy");
  Tensor part = at::empty({(int64_t)adb200::bn_parts(rows, C) * C}, dy.options().dtype(at::kFloat));
  adb200::relu_bwd_colsum(CBF(dy), y.has_value() ? CBF(*y) : nullptr, dx.has_value() ? BF(*dx) : nullptr, part.data_ptr<float>(),
                          out.data_ptr<float>(), rows, C, accumulate ? 1 : 0, STREAM);
}
void relu_bwd(const Tensor& dy, const Tensor& y, Tensor dx) {
  TORCH_CHECK(dy.is_contiguous() && y.is_contiguous() && dx.is_contiguous() && dy.numel() == y.numel() && dx.numel() == y.numel() && y.numel() % 8 == 0,
              "contiguous bf16 tensors of one size (a multiple of 8)");
  adb200::relu_bwd(CBF(dy), CBF(y), BF(dx), y.numel(), STREAM);
}
void psgd_p(Tensor M, const optional<Tensor>& err, const Tensor& Q, Tensor P) {
  const int m = M.size(0), n = M.size(1), r = Q.size(1);
  TORCH_CHECK(r >= 1 && r <= 4 && M.is_contiguous() && Q.is_contiguous() && P.is_contiguous(), "rank 1..4, contiguous fp32 operands");
  adb200::psgd_p(M.data_ptr<float>(), OPT_F(err), Q.data_ptr<float>(), P.data_ptr<float>(), m, n, r, STREAM);
}
void psgd_q(const Tensor& M, const Tensor& P, Tensor Qn) {
  const int m = M.size(0), n = M.size(1), r = P.size(1);
  TORCH_CHECK(r >= 1 && r <= 4 && M.is_contiguous() && P.is_contiguous() && Qn.is_contiguous(), "rank 1..4, contiguous fp32 operands");
  adb200::psgd_q(M.data_ptr<float>(), P.data_ptr<float>(), Qn.data_ptr<float>(), m, n, r, STREAM);
}
void psgd_d(Tensor M, Tensor err, const Tensor& P, const Tensor& Q) {
  const int m = M.size(0), n = M.size(1), r = P.size(1);
  adb200::psgd_d(M.data_ptr<float>(), err.data_ptr<float>(), P.data_ptr<float>(), Q.data_ptr<float>(), m, n, r, STREAM);
}
// One pass of PowerSGD over every matrix of the step (see elementwise.cu). off / p_off / q_off / *_prefix: int64 device tensors,
// m / n: int32 device tensors; phase 0 = P = (grad + err) Q, 1 = orthogonalise P, 2 = Q = grad^T P, 3 = err = grad - P Q^T, grad = P Q^T.
void psgd_batched(int64_t phase, Tensor grad, Tensor err, Tensor P, Tensor Q, const Tensor& off, const Tensor& m, const Tensor& n,
                  const Tensor& p_off, const Tensor& q_off, const Tensor& row_prefix, const Tensor& blk_prefix, const Tensor& elem_prefix,
                  int64_t rank, int64_t rows, int64_t blocks, int64_t elems) {
  const int nmat = m.numel();
  TORCH_CHECK(rank >= 1 && rank <= 4 && grad.scalar_type() == at::kFloat && err.scalar_type() == at::kFloat && P.scalar_type() == at::kFloat &&
              Q.scalar_type() == at::kFloat, "fp32 buffers, rank 1..4");
  TORCH_CHECK(off.numel() == nmat && n.numel() == nmat && p_off.numel() == nmat && q_off.numel() == nmat && row_prefix.numel() == nmat + 1 &&
              blk_prefix.numel() == nmat + 1 && elem_prefix.numel() == nmat + 1 && m.scalar_type() == at::kInt && n.scalar_type() == at::kInt,
              "table arrays of the wrong length or type");
  auto ll = [](const Tensor& t) { return reinterpret_cast<const long long*>(t.data_ptr<int64_t>()); };
  adb200::psgd_batched((int)phase, grad.data_ptr<float>(), err.data_ptr<float>(), P.data_ptr<float>(), Q.data_ptr<float>(), ll(off),
                       m.data_ptr<int>(), n.data_ptr<int>(), ll(p_off), ll(q_off), ll(row_prefix), ll(blk_prefix), ll(elem_prefix), nmat, (int)rank,
                       rows, blocks, elems, STREAM);
}
void cast_f32_bf16(const Tensor& x, Tensor y) { adb200::cast_f32_bf16(x.data_ptr<float>(), BF(y), x.numel(), STREAM); }
void increment(Tensor c) { adb200::increment(reinterpret_cast<long long*>(c.data_ptr<int64_t>()), STREAM); }

// ---------------------------------------------------------------------------------------------- communication
adb200::SymCtx make_ctx(const Tensor& flag_ptrs, Tensor epochs, Tensor error, int64_t rank, int64_t world, double timeout_s) {
  adb200::SymCtx c;
  c.flags = reinterpret_cast<uint32_t* const*>(flag_ptrs.data_ptr<int64_t>());
  c.epochs = reinterpret_cast<uint32_t*>(epochs.data_ptr<int32_t>());
  c.error = error.data_ptr<int32_t>();
  c.rank = (int)rank;
  c.world = (int)world;
  c.timeout_ns = (unsigned long long)(timeout_s * 1e9);
  TORCH_CHECK(world >= 1 && world <= 8, "1 to 8 ranks supported");
  TORCH_CHECK(epochs.numel() >= adb200::kMaxCommBlocks + 2, "epoch array too small (blocks + 2 words)");
  return c;
}

// buf_ptrs: int64 device tensor with every rank's wire-buffer address; mc_ptr: multicast address or 0.
void allreduce(const Tensor& flag_ptrs, Tensor epochs, Tensor error, int64_t rank, int64_t world, double timeout_s, const Tensor& buf_ptrs,
               int64_t mc_ptr, int64_t wire, int64_t n, const optional<Tensor>& src32, const optional<Tensor>& residual,
               const optional<Tensor>& dst32, double scale, int64_t blocks) {
  adb200::SymCtx c = make_ctx(flag_ptrs, epochs, error, rank, world, timeout_s);
  const int vec = wire == adb200::WIRE_F32 ? 4 : 8;
  TORCH_CHECK(n % vec == 0, "bucket length must be a multiple of ", vec);
  if (blocks <= 0) blocks = adb200::comm_grid(n / vec / world, adb200::kMaxCommBlocks);
  TORCH_CHECK(blocks <= adb200::kMaxCommBlocks, "too many blocks");
  adb200::launch_allreduce(c, reinterpret_cast<void* const*>(buf_ptrs.data_ptr<int64_t>()), reinterpret_cast<void*>(mc_ptr), (int)wire, n,
                           OPT_F(src32), OPT_F(residual), OPT_F(dst32), (float)scale, (int)blocks, STREAM);
}

void reduce_scatter_update(const Tensor& flag_ptrs, Tensor epochs, Tensor error, int64_t rank, int64_t world, double timeout_s,
                           const Tensor& grad_ptrs, const Tensor& p16_ptrs, const optional<Tensor>& p32_ptrs, int64_t mc_grad, int64_t mc_p16,
                           int64_t mc_p32, Tensor master,
                           const optional<Tensor>& s1, const optional<Tensor>& s2, const Tensor& seg_start, const Tensor& seg_len,
                           const Tensor& seg_state, const optional<Tensor>& seg_flags, const Tensor& owned_prefix, int64_t kind, const Tensor& lr, const Tensor& step, double b1,
                           double b2, double eps, double wd, double momentum, double grad_scale, bool decoupled, bool nesterov, double scale,
                           int64_t blocks) {
  adb200::SymCtx c = make_ctx(flag_ptrs, epochs, error, rank, world, timeout_s);
  const int nseg = seg_start.numel();
  TORCH_CHECK(owned_prefix.numel() == nseg + 1, "owned_prefix must have nseg + 1 entries");
  TORCH_CHECK(blocks > 0 && blocks <= adb200::kMaxCommBlocks, "bad block count");
  adb200::launch_reduce_scatter_update(
      c, reinterpret_cast<float* const*>(grad_ptrs.data_ptr<int64_t>()), reinterpret_cast<__nv_bfloat16* const*>(p16_ptrs.data_ptr<int64_t>()),
      p32_ptrs.has_value() ? reinterpret_cast<float* const*>(p32_ptrs->data_ptr<int64_t>()) : nullptr, reinterpret_cast<float*>(mc_grad),
      reinterpret_cast<__nv_bfloat16*>(mc_p16), reinterpret_cast<float*>(mc_p32), master.data_ptr<float>(), OPT_F(s1),
      OPT_F(s2), reinterpret_cast<const long long*>(seg_start.data_ptr<int64_t>()), reinterpret_cast<const long long*>(seg_len.data_ptr<int64_t>()),
      reinterpret_cast<const long long*>(seg_state.data_ptr<int64_t>()),
      seg_flags.has_value() ? reinterpret_cast<const long long*>(seg_flags->data_ptr<int64_t>()) : nullptr,
      reinterpret_cast<const long long*>(owned_prefix.data_ptr<int64_t>()), nseg,
      (int)kind, lr.data_ptr<float>(), reinterpret_cast<const long long*>(step.data_ptr<int64_t>()), (float)b1, (float)b2, (float)eps, (float)wd,
      (float)momentum, (float)grad_scale, decoupled ? 1 : 0, nesterov ? 1 : 0, (float)scale, (int)blocks, STREAM);
}

void sparse_scatter_add(const Tensor& flag_ptrs, Tensor epochs, Tensor error, int64_t rank, int64_t world, double timeout_s,
                        const Tensor& shard_ptrs, const optional<Tensor>& touched_ptrs, const Tensor& ids, const Tensor& vals, int64_t V,
                        double scale, int64_t barriers, int64_t blocks) {
  adb200::SymCtx c = make_ctx(flag_ptrs, epochs, error, rank, world, timeout_s);
  const int H = vals.size(-1);
  TORCH_CHECK(H % 4 == 0, "row width must be a multiple of 4");
  TORCH_CHECK(blocks > 0 && blocks <= adb200::kMaxCommBlocks, "bad block count");
  adb200::launch_sparse_scatter_add(c, reinterpret_cast<float* const*>(shard_ptrs.data_ptr<int64_t>()),
                                    touched_ptrs.has_value() ? reinterpret_cast<uint8_t* const*>(touched_ptrs->data_ptr<int64_t>()) : nullptr,
                                    ids.data_ptr<int64_t>(), vals.data_ptr(),
                                    vals.scalar_type() == at::kBFloat16 ? 1 : 0, ids.numel(), H, V, (float)scale, (int)barriers, (int)blocks, STREAM);
}

void embedding_gather_peers(const Tensor& flag_ptrs, Tensor epochs, Tensor error, int64_t rank, int64_t world, double timeout_s,
                            const Tensor& shard_ptrs, const Tensor& ids, Tensor out, int64_t V, int64_t barriers, int64_t blocks) {
  adb200::SymCtx c = make_ctx(flag_ptrs, epochs, error, rank, world, timeout_s);
  TORCH_CHECK(out.size(-1) % 8 == 0, "row width must be a multiple of 8");
  TORCH_CHECK(blocks > 0 && blocks <= adb200::kMaxCommBlocks, "bad block count");
  adb200::launch_embedding_gather_peers(c, reinterpret_cast<__nv_bfloat16* const*>(shard_ptrs.data_ptr<int64_t>()), ids.data_ptr<int64_t>(),
                                        BF(out), ids.numel(), out.size(-1), V, (int)barriers, (int)blocks, STREAM);
}

void sym_barrier(const Tensor& flag_ptrs, Tensor epochs, Tensor error, int64_t rank, int64_t world, double timeout_s, int64_t blocks) {
  adb200::SymCtx c = make_ctx(flag_ptrs, epochs, error, rank, world, timeout_s);
  TORCH_CHECK(blocks > 0 && blocks <= adb200::kMaxCommBlocks, "block count must be in [1, ", adb200::kMaxCommBlocks, "]");
  adb200::launch_barrier(c, (int)blocks, STREAM);
}

// step (optional int64 device scalar) overrides my_step; staleness < 0 publishes the step without waiting; max_lead (optional int32
// device scalar) keeps the largest lead this rank had when it passed the gate.
void staleness_gate(const Tensor& flag_ptrs, Tensor epochs, Tensor error, int64_t rank, int64_t world, double timeout_s,
                    const Tensor& clock_ptrs, int64_t my_step, int64_t staleness, const optional<Tensor>& step, const optional<Tensor>& max_lead) {
  adb200::SymCtx c = make_ctx(flag_ptrs, epochs, error, rank, world, timeout_s);
  adb200::launch_staleness_gate(c, reinterpret_cast<uint32_t* const*>(clock_ptrs.data_ptr<int64_t>()), (uint32_t)my_step, OPT_LL(step),
                                (int)staleness, max_lead.has_value() ? max_lead->data_ptr<int>() : nullptr, STREAM);
}

// Relaxed parameter server with GPU owners (plain SGD): p32_owner[segment] -= lr * grad_scale * grad[segment], as vector reductions on
// the owners' fp32 copies. Segment tables: int64 device tensors; prefix has nseg + 1 entries; every start / length a multiple of 4.
void relaxed_push_sgd(const Tensor& p32_ptrs, const Tensor& grad, const Tensor& seg_start, const Tensor& seg_len, const Tensor& seg_owner,
                      const Tensor& prefix, const Tensor& lr, double grad_scale, int64_t blocks) {
  const int nseg = seg_start.numel();
  TORCH_CHECK(prefix.numel() == nseg + 1 && seg_owner.numel() == nseg && grad.scalar_type() == at::kFloat, "bad segment tables");
  auto ll = [](const Tensor& t) { return reinterpret_cast<const long long*>(t.data_ptr<int64_t>()); };
  adb200::launch_relaxed_push_sgd(reinterpret_cast<float* const*>(p32_ptrs.data_ptr<int64_t>()), grad.data_ptr<float>(), ll(seg_start), ll(seg_len),
                                  ll(seg_owner), ll(prefix), nseg, lr.data_ptr<float>(), (float)grad_scale, (int)blocks, STREAM);
}
// Refresh this rank's fp32 and bf16 copies of every segment from the segment's owner.
void relaxed_pull(const Tensor& p32_ptrs, Tensor master, Tensor p16, const Tensor& seg_start, const Tensor& seg_len, const Tensor& seg_owner,
                  const Tensor& prefix, int64_t rank, int64_t blocks) {
  const int nseg = seg_start.numel();
  TORCH_CHECK(prefix.numel() == nseg + 1 && seg_owner.numel() == nseg, "bad segment tables");
  auto ll = [](const Tensor& t) { return reinterpret_cast<const long long*>(t.data_ptr<int64_t>()); };
  adb200::launch_relaxed_pull(reinterpret_cast<float* const*>(p32_ptrs.data_ptr<int64_t>()), master.data_ptr<float>(), BF(p16), ll(seg_start),
                              ll(seg_len), ll(seg_owner), ll(prefix), nseg, (int)rank, (int)blocks, STREAM);
}

// dst[i] <- src[i] for contiguous tensors of one device, sizes and dtypes equal, in one launch per kMaxCopies of them. Returns false, and
// copies nothing, when a pair does not qualify.
bool copy_list(const std::vector<Tensor>& dst, const std::vector<Tensor>& src) {
  if (dst.size() != src.size()) return false;
  for (size_t i = 0; i < dst.size(); ++i) {
    const Tensor &d = dst[i], &s = src[i];
    if (!d.is_cuda() || !s.is_cuda() || d.device() != s.device() || d.device() != dst[0].device() || d.scalar_type() != s.scalar_type() ||
        d.sizes() != s.sizes() || !d.is_contiguous() || !s.is_contiguous() || d.is_conj() != s.is_conj() || d.is_neg() != s.is_neg() ||
        d.numel() * d.element_size() > (1LL << 40))
      return false;
  }
  if (dst.empty()) return true;
  const c10::cuda::CUDAGuard guard(dst[0].device());
  for (size_t i = 0; i < dst.size();) {
    adb200::CopyList c{};
    long long blocks = 0;
    for (; i < dst.size() && c.n < adb200::kMaxCopies; ++i) {
      const long long bytes = (long long)dst[i].numel() * dst[i].element_size();
      if (bytes == 0 || dst[i].data_ptr() == src[i].data_ptr()) continue;
      c.src[c.n] = src[i].data_ptr(); c.dst[c.n] = dst[i].data_ptr(); c.bytes[c.n] = bytes;
      c.first[c.n] = (int)blocks;
      blocks += (bytes + adb200::kCopyBlockBytes - 1) / adb200::kCopyBlockBytes;
      c.first[++c.n] = (int)blocks;
    }
    adb200::copy_list(c, STREAM);
  }
  return true;
}
// A kernel gets the addresses of all of these.
void check_one_gpu(std::initializer_list<const Tensor*> tensors) {
  for (const Tensor* t : tensors) TORCH_CHECK(t->is_cuda() && t->device() == (*tensors.begin())->device(), "tensors on one GPU needed");
}
// Where a kernel reports an id outside its table: a word on the device, or in pinned host memory, which the host reads without waiting.
int* report_word(const Tensor& t) {
  TORCH_CHECK(t.scalar_type() == at::kInt && t.numel() >= 1 && (t.is_cuda() || t.is_pinned()), "an int32 word on the GPU or in pinned memory needed");
  return t.data_ptr<int>();
}
void check_pair_tables(const Tensor& a, const Tensor& b, int64_t mf, const Tensor& users, const Tensor& items) {
  for (const Tensor* t : {&a, &b})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->dim() == 2 && t->is_contiguous() && t->size(1) == a.size(1) &&
                    reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 == 0, "contiguous fp32 tables of one width needed");
  TORCH_CHECK(mf % 4 == 0 && a.size(1) % 4 == 0 && mf > 0 && mf < a.size(1), "both parts of a row must be multiples of 4 columns");
  TORCH_CHECK(users.scalar_type() == at::kLong && items.scalar_type() == at::kLong && users.is_contiguous() && items.is_contiguous() &&
                  users.numel() == items.numel(), "int64 ids needed");
}
// gmf [n, mf] fp32, x [n, 2 h] bf16, kept (optional) [n, 2 mf] fp32; tables [.., mf + h]
void pair_lookup(const Tensor& ut, const Tensor& it, const Tensor& users, const Tensor& items, int64_t mf, Tensor gmf, Tensor x,
                 const optional<Tensor>& kept, Tensor error) {
  check_one_gpu({&ut, &it, &users, &items, &gmf, &x, kept.has_value() ? &*kept : &x});
  const c10::cuda::CUDAGuard guard(ut.device());
  check_pair_tables(ut, it, mf, users, items);
  const int64_t n = users.numel(), h = ut.size(1) - mf;
  TORCH_CHECK(gmf.numel() == n * mf && gmf.scalar_type() == at::kFloat && gmf.is_contiguous() && x.numel() == n * 2 * h &&
                  x.scalar_type() == at::kBFloat16 && x.is_contiguous() && (!kept.has_value() || (kept->numel() == n * 2 * mf && kept->is_contiguous())),
              "outputs must match the lookups");
  adb200::pair_lookup(ut.data_ptr<float>(), it.data_ptr<float>(), users.data_ptr<int64_t>(), items.data_ptr<int64_t>(), gmf.data_ptr<float>(), BF(x), OPT_F(kept),
                      n, (int)mf, (int)h, ut.size(0), it.size(0), report_word(error), STREAM);
}
// dgmf: fp32 [n, mf] with unit inner stride
void pair_lookup_bwd(const Tensor& dgmf, const Tensor& dx, const Tensor& kept, const Tensor& users, const Tensor& items, Tensor gu, Tensor gi) {
  check_one_gpu({&dgmf, &dx, &kept, &users, &items, &gu, &gi});
  const c10::cuda::CUDAGuard guard(dgmf.device());
  const int64_t n = users.numel(), mf = dgmf.size(1);
  check_pair_tables(gu, gi, mf, users, items);
  const int64_t h = gu.size(1) - mf;
  TORCH_CHECK(dgmf.scalar_type() == at::kFloat && dgmf.dim() == 2 && dgmf.size(0) == n && dgmf.stride(1) == 1 && dgmf.stride(0) % 4 == 0 &&
                  reinterpret_cast<uintptr_t>(dgmf.data_ptr()) % 16 == 0, "rows of dgmf must start on 16-byte boundaries");
  TORCH_CHECK(dx.scalar_type() == at::kBFloat16 && dx.is_contiguous() && dx.numel() == n * 2 * h && reinterpret_cast<uintptr_t>(dx.data_ptr()) % 8 == 0 &&
                  kept.scalar_type() == at::kFloat && kept.is_contiguous() && kept.numel() == n * 2 * mf, "gradients must match the lookups");
  adb200::pair_lookup_bwd(dgmf.data_ptr<float>(), dgmf.stride(0), CBF(dx), kept.data_ptr<float>(), users.data_ptr<int64_t>(), items.data_ptr<int64_t>(),
                          gu.data_ptr<float>(), gi.data_ptr<float>(), n, (int)mf, (int)h, gu.size(0), gi.size(0), STREAM);
}
// part[i] = scale * the losses of elements 16384 i ...
void bce_logits(const Tensor& x, const Tensor& y, Tensor part, double scale) {
  check_one_gpu({&x, &y, &part});
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.scalar_type() == at::kFloat && y.scalar_type() == at::kFloat && x.is_contiguous() && y.is_contiguous() && y.numel() == x.numel() &&
                  x.numel() > 0 && part.numel() >= adb200::bce_logits_parts(x.numel()), "contiguous fp32 logits and labels needed");
  adb200::bce_logits(x.data_ptr<float>(), y.data_ptr<float>(), part.data_ptr<float>(), x.numel(), (float)scale, STREAM);
}
void bce_logits_bwd(const Tensor& x, const Tensor& y, const Tensor& grad, Tensor dx, double scale) {
  check_one_gpu({&x, &y, &grad, &dx});
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.scalar_type() == at::kFloat && y.scalar_type() == at::kFloat && dx.scalar_type() == at::kFloat && grad.scalar_type() == at::kFloat,
              "fp32 tensors needed");
  TORCH_CHECK(x.is_contiguous() && y.is_contiguous() && dx.is_contiguous() && y.numel() == x.numel() && dx.numel() == x.numel() && grad.numel() == 1,
              "gradients must match the logits");
  adb200::bce_logits_bwd(x.data_ptr<float>(), y.data_ptr<float>(), grad.data_ptr<float>(), dx.data_ptr<float>(), x.numel(), (float)scale, STREAM);
}
// logits [N, 1 + K] fp32 of the rows' own classes and the sampled ones; ids and corrections are scratch of [K + N] (and [K + N, 2]) that
// the gradient passes read again. dot [N]: the own classes' products, bf16 or fp32.
void sampled_logits(const Tensor& raw, const Tensor& dot, const Tensor& bias, const Tensor& neg, const Tensor& targets, double inv_log_v, double num_sampled,
                    Tensor corrections, Tensor ids, Tensor logits, Tensor error) {
  const c10::cuda::CUDAGuard guard(raw.device());
  check_one_gpu({&raw, &dot, &bias, &neg, &targets, &corrections, &ids, &logits});
  for (const Tensor* t : std::initializer_list<const Tensor*>{&raw, &dot, &bias, &neg, &targets, &corrections, &ids, &logits}) TORCH_CHECK(t->is_contiguous(), "contiguous tensors needed");
  TORCH_CHECK(raw.scalar_type() == at::kBFloat16 && raw.dim() == 2 && raw.size(1) % 8 == 0, "bf16 products in rows of 16-byte multiples needed");
  const int64_t N = raw.size(0), K = raw.size(1);
  TORCH_CHECK(N > 0 && K > 0 && N + K < (1LL << 30) && dot.numel() == N && (dot.scalar_type() == at::kBFloat16 || dot.scalar_type() == at::kFloat),
              "a product per row needed");
  TORCH_CHECK(bias.scalar_type() == at::kFloat && bias.dim() == 1, "fp32 bias needed");
  TORCH_CHECK(neg.scalar_type() == at::kLong && neg.numel() == K && targets.scalar_type() == at::kLong && targets.numel() == N,
              "int64 ids of the sampled classes and of the targets needed");
  TORCH_CHECK(corrections.scalar_type() == at::kFloat && corrections.numel() == 2 * (N + K) && ids.scalar_type() == at::kInt && ids.numel() == N + K &&
                  logits.scalar_type() == at::kFloat && logits.numel() == N * (K + 1), "outputs must match the products");
  adb200::sampled_logits(CBF(raw), dot.data_ptr(), dot.scalar_type() == at::kBFloat16, bias.data_ptr<float>(), neg.data_ptr<int64_t>(),
                         targets.data_ptr<int64_t>(), (int)N, (int)K, bias.numel(), (float)inv_log_v, (float)num_sampled,
                         reinterpret_cast<float2*>(corrections.data_ptr<float>()), ids.data_ptr<int>(), logits.data_ptr<float>(), report_word(error), STREAM);
}
// From the log-softmax of those logits: gradients of the products, of dot, and (dadj [K + N]) of every place's bias.
void sampled_grad(const Tensor& logp, const Tensor& ids, const Tensor& grad, Tensor part, Tensor draw, Tensor ddot, Tensor dadj) {
  const c10::cuda::CUDAGuard guard(logp.device());
  check_one_gpu({&logp, &ids, &grad, &part, &draw, &ddot, &dadj});
  for (const Tensor* t : std::initializer_list<const Tensor*>{&logp, &ids, &grad, &part, &draw, &ddot, &dadj}) TORCH_CHECK(t->is_contiguous(), "contiguous tensors needed");
  TORCH_CHECK(draw.scalar_type() == at::kBFloat16 && draw.dim() == 2 && draw.size(1) % 8 == 0 && draw.numel() > 0, "bf16 gradient of the products needed");
  const int64_t N = draw.size(0), K = draw.size(1);
  TORCH_CHECK(logp.scalar_type() == at::kFloat && logp.numel() == N * (K + 1) && ids.scalar_type() == at::kInt && ids.numel() == N + K, "log-probabilities must match");
  TORCH_CHECK(grad.scalar_type() == at::kFloat && grad.numel() == 1, "fp32 scalar gradient needed");
  TORCH_CHECK(ddot.numel() == N && (ddot.scalar_type() == at::kBFloat16 || ddot.scalar_type() == at::kFloat), "a gradient per row needed");
  TORCH_CHECK(part.scalar_type() == at::kFloat && part.numel() >= (int64_t)adb200::sampled_grad_chunks((int)N, (int)K) * K && dadj.scalar_type() == at::kFloat &&
                  dadj.numel() == N + K, "scratch too small");
  adb200::sampled_grad(logp.data_ptr<float>(), ids.data_ptr<int>(), grad.data_ptr<float>(), (int)N, (int)K, part.data_ptr<float>(), BF(draw), ddot.data_ptr(),
                       ddot.scalar_type() == at::kBFloat16, dadj.data_ptr<float>(), STREAM);
}
// dbias[ids[i]] += dadj[i], in an order that the ids decide; at most SAMPLED_SCAN_MOST of them
void sampled_bias_grad(const Tensor& ids, const Tensor& dadj, Tensor sums, Tensor firsts, Tensor dbias) {
  const c10::cuda::CUDAGuard guard(ids.device());
  check_one_gpu({&ids, &dadj, &sums, &firsts, &dbias});
  for (const Tensor* t : std::initializer_list<const Tensor*>{&ids, &dadj, &sums, &firsts, &dbias}) TORCH_CHECK(t->is_contiguous(), "contiguous tensors needed");
  TORCH_CHECK(ids.scalar_type() == at::kInt && ids.numel() <= adb200::kSampledScanMost && dadj.scalar_type() == at::kFloat && dadj.numel() == ids.numel() &&
                  dbias.scalar_type() == at::kFloat, "int32 ids and fp32 values");
  const int64_t scratch = ids.numel() * adb200::sampled_bias_chunks((int)ids.numel());
  TORCH_CHECK(sums.scalar_type() == at::kFloat && sums.numel() >= scratch && firsts.scalar_type() == at::kInt && firsts.numel() >= scratch, "scratch too small");
  adb200::sampled_bias_grad(ids.data_ptr<int>(), dadj.data_ptr<float>(), sums.data_ptr<float>(), firsts.data_ptr<int>(), dbias.data_ptr<float>(), (int)ids.numel(), STREAM);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("copy_list", &copy_list);
  m.def("pair_lookup", &pair_lookup);
  m.def("pair_lookup_bwd", &pair_lookup_bwd);
  m.def("bce_logits", &bce_logits);
  m.def("bce_logits_bwd", &bce_logits_bwd);
  m.def("bce_logits_parts", &adb200::bce_logits_parts);
  m.def("sampled_logits", &sampled_logits);
  m.def("sampled_grad", &sampled_grad);
  m.def("sampled_bias_grad", &sampled_bias_grad);
  m.def("sampled_grad_chunks", &adb200::sampled_grad_chunks);
  m.def("sampled_bias_chunks", &adb200::sampled_bias_chunks);
  m.attr("SAMPLED_SCAN_MOST") = adb200::kSampledScanMost;
  m.def("gemm_set_trace", &gemm_set_trace);
  m.def("gemm", &gemm);
  m.def("gemm_split", &gemm_split);
  m.def("gemm_choice", &gemm_choice, py::arg("M"), py::arg("N"), py::arg("K"), py::arg("batch"), py::arg("epilogue"), py::arg("both_mn"),
        py::arg("fp32_out") = py::none(), py::arg("fixed") = false);
  m.def("attn_fwd", &attn_fwd);
  m.def("attn_bwd", &attn_bwd);
  m.def("gemm_softmax", &gemm_softmax);
  m.def("gemm_gathered_b", &gemm_gathered_b);
  m.def("gemm_gathered_bt", &gemm_gathered_bt);
  m.def("ln_fwd", &ln_fwd);
  m.def("ln_bwd", &ln_bwd);
  m.def("ln_bwd_part_floats", &adb200::ln_bwd_part_floats);
  m.def("colsum_parts", &adb200::colsum_parts);
  m.def("embed_sum", &embed_sum);
  m.def("scatter_add_rows", &scatter_add_rows);
  m.def("scatter_add_rows_f32", &scatter_add_rows_f32);
  m.def("lstm_seq_fwd", &lstm_seq_fwd);
  m.def("lstm_seq_bwd", &lstm_seq_bwd);
  m.def("strided_rowsum", &strided_rowsum);
  m.def("keyed_colsum", &keyed_colsum);
  m.def("gather_rows", &gather_rows);
  m.def("gather_rows_f32", &gather_rows_f32);
  m.def("scatter_add_rows_bf16", &scatter_add_rows_bf16);
  m.def("softmax_fwd", &softmax_fwd);
  m.def("softmax_bwd", &softmax_bwd);
  m.def("xent", &xent);
  m.def("tanh_bwd", &tanh_bwd);
  m.def("gelu_bwd", &gelu_bwd);
  m.def("add_bf16", &add_bf16);
  m.def("adam_update", &adam_update);
  m.def("sgd_update", &sgd_update);
  m.def("adagrad_update", &adagrad_update);
  m.def("sparse_rows_update", &sparse_rows_update);
  m.def("flagged_rows_update", &flagged_rows_update);
  m.def("cast_f32_bf16", &cast_f32_bf16);
  m.def("bn_fwd", &bn_fwd);
  m.def("bn_fwd_nchw", &bn_fwd_nchw);
  m.def("bn_sums", &bn_sums);
  m.def("bn_eval", &bn_eval);
  m.def("bn_bwd", &bn_bwd);
  m.def("maxpool_fwd", &maxpool_fwd);
  m.def("maxpool_bwd", &maxpool_bwd);
  m.def("im2col", &im2col);
  m.def("col2im", &col2im);
  m.def("pad_image8", &pad_image8);
  m.def("relu_bwd", &relu_bwd);
  m.def("relu_bwd_colsum", &relu_bwd_colsum);
  m.def("psgd_batched", &psgd_batched);
  m.def("psgd_p", &psgd_p);
  m.def("psgd_q", &psgd_q);
  m.def("psgd_d", &psgd_d);
  m.def("lstm_cell_fwd", &lstm_cell_fwd);
  m.def("lstm_cell_bwd", &lstm_cell_bwd);
  m.def("sumsq", &sumsq);
  m.def("clip_scale", &clip_scale);
  m.def("increment", &increment);
  m.def("allreduce", &allreduce);
  m.def("reduce_scatter_update", &reduce_scatter_update);
  m.def("sparse_scatter_add", &sparse_scatter_add);
  m.def("embedding_gather_peers", &embedding_gather_peers);
  m.def("sym_barrier", &sym_barrier);
  m.def("staleness_gate", &staleness_gate);
  m.def("relaxed_push_sgd", &relaxed_push_sgd);
  m.def("relaxed_pull", &relaxed_pull);
  m.attr("MAX_COMM_BLOCKS") = adb200::kMaxCommBlocks;
  register_conv(m);
}
