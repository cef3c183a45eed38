// Flash-attention forward for sm_100a: O = softmax(scale * Q K^T [key-padding / causal mask]) V.
// fp16 operands, fp32 accumulation.  V is consumed in its natural [key, d] layout as an MN-major operand.  Four kernels:
//   * flash_attn_short_kernel (flash_attn_short.cuh): sequences of at most 128 keys, several (head, batch) items per SM;
//   * flash_attn_pipe_kernel (flash_attn_pipe.cuh): longer sequences, one or two query tiles per CTA with an online softmax;
//   * flash_attn_quad_kernel (flash_attn_quad.cuh): head size 64, tiles enough for four CTAs on every SM;
//   * flash_attn_tri_kernel (flash_attn_tri.cuh): the bits of flash_attn_pipe_kernel with three CTAs on every SM.
//
// Q, K, V, O are addressed through (batch, head, seq) strides with d contiguous, so both the
// reference's [B, heads, S, d] tensors and column slices of a fused [tokens, 3*hidden] QKV
// projection are read in place by rank-4 tensor maps.  Rows / keys beyond S read as zero.
#include "zen_common.cuh"
#include "det_math.h"
#include "tma_host.cuh"

namespace zen {

constexpr int FA_BQ = 128;
constexpr int FA_BKV = 128;

// Order in which the CTAs of a long sequence's kernels take the tiles, fastest first (the last of batch, head, tile left out)
enum { FA_ORDER_HEADS_BATCHES = 0, FA_ORDER_HEADS_TILES = 1, FA_ORDER_TILES_HEADS = 2 };

struct FaParams {
  void* o;
  int o_f32;  // the fp16 results are stored as fp32 (the fp32 binding)
  const float *q32, *k32, *v32;  // fp32 operands that the kernel converts itself (no tensor maps then)
  int8_t* oq;
  float o_scale, inv_o_scale;
  int B, H, S;
  int64_t o_sb, o_sh, o_ss;
  const int32_t* kv_lens;
  const int32_t* cu_seqlens;  // unpadded batches (long-sequence kernel only): [B + 1] row offsets, null otherwise
  int rows;                   // ... rows of the packed tensors
  int causal;
  float scale_log2;    // |softmax scale| * log2(e)
  uint32_t qk_negate;  // added to the descriptor of Q K^T: the sign of the scale
  // position of the (seq, head, batch) coordinates in each rank-4 tensor map (dim 0 is d)
  int q_perm[3], k_perm[3], v_perm[3];
  int order;     // FA_ORDER_*
  int box_rows;  // rows of a loaded tile: 128, for shorter sequences what holds all of them
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void fa_tma_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, const int (&perm)[3],
                                            int d0, int s, int h, int b) {
  // selects: an array indexed by `perm` would live in local memory, a round trip in front of every load
  const int c1 = perm[0] == 1 ? s : (perm[1] == 1 ? h : b);
  const int c2 = perm[0] == 2 ? s : (perm[1] == 2 ? h : b);
  const int c3 = perm[0] == 3 ? s : (perm[1] == 3 ? h : b);
  tma_load_4d(dst, map, bar, d0, c1, c2, c3);
}

// The softmax scale as the kernels take it.  A masked score is -inf, which is no maximum and no probability as long as the
// factor is positive: so the sign of the scale goes into Q K^T (the maximum is then the maximum of the scaled scores too), and
// zero becomes a factor that leaves the exponent of every finite score at zero.
struct SoftmaxScale {
  float log2;
  uint32_t negate;
};
inline SoftmaxScale softmax_scale(float scale) {
  const float f = fabsf(scale) * 1.4426950408889634f;
  return {f < 1e-30f ? 1e-30f : f, scale < 0.0f ? uint32_t(IDESC_NEGATE_A) : 0u};
}

}  // namespace zen
#include "flash_attn_pipe.cuh"
#include "flash_attn_quad.cuh"
#include "flash_attn_tri.cuh"
#include "flash_attn_short.cuh"
#include "qkv_attn.cuh"
namespace zen {

// Rank-4 map over (d, seq, head, batch) with the three outer dims ordered by ascending stride.
// `elem_bytes` 2: fp16 with 128-byte swizzle (64-column boxes); 1: int8 with 64-byte swizzle.
static int encode_qkv_map(CUtensorMap* map, const void* base, int B, int H, int S, int D, int64_t sb, int64_t sh,
                          int64_t ss, int (&perm)[3], uint32_t box_rows = FA_BQ, int elem_bytes = 2) {
  struct Dim {
    uint64_t extent;
    int64_t stride;
    uint32_t box;
    int id;
  } dims[3] = {{uint64_t(S), ss, box_rows, 0}, {uint64_t(H), sh, 1u, 1}, {uint64_t(B), sb, 1u, 2}};
  // the stride of an extent-1 dim is never used to form an address: give it a valid, outermost value
  int64_t span = 8;
  for (int i = 0; i < 3; ++i)
    if (dims[i].extent > 1 && int64_t(dims[i].extent) * dims[i].stride > span) span = int64_t(dims[i].extent) * dims[i].stride;
  for (int i = 0; i < 3; ++i)
    if (dims[i].extent == 1) dims[i].stride = (span + 7) / 8 * 8;
  for (int i = 0; i < 3; ++i)
    for (int j = i + 1; j < 3; ++j)
      if (dims[j].stride < dims[i].stride) {
        Dim t = dims[i];
        dims[i] = dims[j];
        dims[j] = t;
      }
  uint64_t gd[4] = {uint64_t(D), 0, 0, 0};
  uint64_t gs[3];
  uint32_t bx[4] = {64u, 0, 0, 0};
  for (int i = 0; i < 3; ++i) {
    gd[i + 1] = dims[i].extent;
    gs[i] = uint64_t(dims[i].stride) * uint64_t(elem_bytes);
    bx[i + 1] = dims[i].box;
    perm[dims[i].id] = i + 1;
    if (dims[i].stride <= 0 || dims[i].stride % (16 / elem_bytes)) return ZEN_ERR_UNSUPPORTED;
  }
  if (elem_bytes == 1)
    return encode_tmap(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, base, gd, gs, bx, CU_TENSOR_MAP_SWIZZLE_64B);
  return encode_tmap(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, base, gd, gs, bx);
}

template <int D, bool F32 = false>
static int launch_fa_short(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaParams& p, cudaStream_t s) {
  auto kernel = flash_attn_short_kernel<D, F32>;
  constexpr size_t smem = fas_smem_bytes<D>();
  if (int st = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem); st != ZEN_OK) return st;
  const int64_t items = int64_t(p.B) * p.H;
  if (items >= (int64_t(1) << 30)) return ZEN_ERR_UNSUPPORTED;
  const unsigned grid = unsigned(items < num_sms() ? items : num_sms());
  return launch_pdl(PDL_ATTENTION, kernel, dim3(grid), dim3(fas_threads<D>()), smem, s, tq, tk, tv, p);
}

// A kernel of `rows` query rows per CTA.
using FaKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, FaParams);
static int launch_fa_tiles(FaKernel kernel, int rows, int threads, size_t smem, const CUtensorMap& tq, const CUtensorMap& tk,
                           const CUtensorMap& tv, const FaParams& p, cudaStream_t s) {
  if (int st = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem); st != ZEN_OK) return st;
  const int64_t ctas = int64_t((p.S + rows - 1) / rows) * p.H * p.B;
  if (ctas >= (int64_t(1) << 31)) return ZEN_ERR_UNSUPPORTED;
  return launch_pdl(PDL_ATTENTION, kernel, dim3(unsigned(ctas)), dim3(unsigned(threads)), smem, s, tq, tk, tv, p);
}

template <int D, int GROUPS, int KV_STAGES, bool F32 = false>
static int launch_fa_pipe(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaParams& p, cudaStream_t s) {
  return launch_fa_tiles(flash_attn_pipe_kernel<D, GROUPS, KV_STAGES, F32>, 128 * GROUPS, fap_threads<GROUPS, F32>(),
                         fap_smem_bytes<D, GROUPS, KV_STAGES>(), tq, tk, tv, p, s);
}

// Head size 64: flash_attn_quad_kernel, where its tiles keep four CTAs on every SM.  With fewer its chains are longer than those
// of flash_attn_pipe_kernel (1900 clocks per 64 keys against 2430 per 128); over long sequences its tiles read K and V from L2
// more often, and the chip is at its power limit.  Measured for 292 shapes of 300 .. 2500 tiles of 160 .. 4096 tokens, time
// against the other kernel, by tiles / (4 SMs):
//   full    S <= 700: 0.5: 1.0 - 1.14, 0.7: 0.82 - 1.12, 0.75 - 1: 0.73 - 1.0, 1.5: 0.70 - 0.96, 3 on: 0.67 - 0.92
//           S = 1024, 1500, 2048, 3000: below 1 from 1.5, 1.7, 2.2, 2.9 on, 0.94 - 0.98 at most; 4096 and longer: 1.02 - 1.2
//   causal  S <= 300: 0.7: 0.89 - 1.11, 0.8 - 1: 0.76 - 0.99, 3 on: 0.70 - 0.77    384 .. 1024: 0.7 - 1: 1.01 - 1.3, 1.1: 0.84 - 1.07,
//           3 on: 0.77 - 0.87    1500 .. 4096: below 1 from 1.5, 2, 2.2, 2.2 on, 0.9 - 0.95 from 3 on; longer: 1.03 - 1.1
// (In short runs 32 x 16 x 384 full 43.8 -> 38.0 us, 8 x 16 x 2048 causal 110.7 -> 99.8; in a stream of passes, where the chip is at
// its power limit, 43.5 -> 39.7 and 118.5 -> 114.6 at 1965 and 1807, 1792 and 1702 MHz.)  The two kernels differ in the last bits, which
// a pass of int8 layers blows up to 3 % of its output (a value moved across a rounding boundary moves others): results with
// an int8 copy stay with one kernel, whatever the batch.  `flags`: ZEN_ATTN_KEYS_64 / _128 of the call.
static bool four_tiles_per_sm(int B, int H, int S, int D, bool causal, bool int8_copy, unsigned flags) {
  if (int8_copy || D != 64 || S <= FA_BKV) return false;
  if (flags != 0) return flags == ZEN_ATTN_KEYS_64;
  if (S > (causal ? 4096 : 3072)) return false;
  const double waves = double((S + 127) / 128) * H * B / (double(FAQ_CTAS) * num_sms());
  if (causal) return waves >= (S <= 320 ? 0.8 : S <= 1100 ? 1.1 : S <= 2100 ? S / 1000.0 : 2.2);
  return waves >= (S <= 768 ? 0.8 : S / 650.0);
}
static bool attn_flags_ok(unsigned flags) { return flags <= ZEN_ATTN_KEYS_128; }  // either of the two, or neither

// Head size 64, with the bits of flash_attn_pipe_kernel: flash_attn_tri_kernel, where the other would need more than two rounds
// of its two CTAs an SM.  Measured for 50 shapes with int8 copy, time against the other kernel:
//   full    up to 576 tiles 1.02 - 1.08; from 624 on S = 160 .. 384: 0.87 - 0.93, 512: 0.94 - 0.98, 700: 0.98 - 1.02, 1024: 0.99 - 1.06
//   causal  up to 576 tiles 1.00 - 1.06; from 624 on S = 160 .. 512: 0.85 - 0.92, 700: 0.93 - 0.96, 1024: 0.95 - 0.98, 2048: 0.99
// Without a copy the output, which the third CTA hides best, is shorter, and the line lies at shorter sequences (144 shapes of
// 600 .. 2400 tiles; by default only the causal ones of 321 .. 1100 tokens and 593 .. 651 tiles come here, the others when
// the call asks for 128 keys at a time):
//   full    S = 160 .. 300: 0.88 - 0.97, 384: 0.95 - 0.98, 512: 0.97 - 1.02, 640: 0.99 - 1.04
//   causal  S = 160 .. 640: 0.84 - 0.96, 700 .. 1024: 0.91 - 0.99, 1500: 0.98 - 1.04, 2048: 1.00 - 1.16
static bool three_tiles_per_sm(int D, const FaParams& p) {
  if (D != 64 || p.S > (p.oq != nullptr ? (p.causal ? 2048 : 640) : (p.causal ? 1100 : 512))) return false;
  return int64_t((p.S + 127) / 128) * p.H * p.B > 4 * num_sms();
}

// Head size 64, otherwise: one or two query tiles per CTA (the same bits): two tiles share K and V, one tile per CTA leaves
// room for two CTAs on an SM.  Up to 2048 tokens one tile: reading K and V once per 128 queries is hidden (32 x 16 heads x 384: 49 us
// against 62; 8 x 16 x 2048: 189 / 192, causal 112 / 121).  Beyond 4096 two (4 x 16 x 8192: 1681 / 1589 us, causal 819 / 797).
// Between, with the last wave: an SM that holds one of its two CTAs runs it faster, one that holds a CTA of two tiles does not.
// Measured at 14 lengths of 2049 .. 5120 for 12 batch x heads of 8 .. 192, two tiles / one tile, by waves of one-tile CTAs:
//   full    0 .. 0.5: 1.32 - 1.35    0.5 .. 1: 0.91 - 0.94    1 .. 1.5: 1.03 - 1.19    1.5 .. 2: 0.92 - 0.96    2 .. 2.5: 1.02 - 1.13
//           2.5 .. 3: 0.94 - 1.10, mean 0.97    3 .. 3.5: 1.01 - 1.10    3.5 .. 4: 0.95 - 0.99    more: 0.95 - 1.09, mean 1.02
//   causal  (the heaviest tiles start first) 0 .. 0.8: 1.06 - 1.29    0.8 .. 2: 0.91 - 1.05, mean 0.97    more: 0.99 - 1.13, mean 1.07
// The choice is 0.3 % from the better one on average.
static bool one_tile_per_cta(const FaParams& p) {
  if (p.S <= 2048 || p.S > 4096) return p.S <= 2048;
  const double waves = double((p.S + 127) / 128) * p.H * p.B / (2.0 * num_sms());
  if (p.causal) return waves <= 0.8 || waves >= 2.0;
  if (waves >= 5.0) return p.S < 4096;
  const double last = waves - double(int64_t(waves));
  return last > 0.0 && last <= 0.5;
}

// The tiles that run at a time should share K and V while those are in L2: with heads and batches before tiles every CTA of a
// wave streams another head's K and V, from HBM where all heads' do not fit L2 (8 x 16 x 8192 x 128: 537 MB, 32 times; the
// power that this takes is what the chip's clock lacks then).  Measured with K and V of 39 .. 537 MB, time against heads, batches,
// tiles, for tiles, heads, batches (heads, tiles, batches):
//   full    d = 128 0.78 at 537 MB (0.83), 0.85 - 0.92 at 100 .. 268 MB (0.87 - 0.90), 0.94 - 0.97 at 39 .. 75 MB
//           d = 64 0.89 - 0.94 at 268 MB (0.92 - 0.95), 0.97 at 134 MB (0.97), 0.98 - 1.04 below
//   causal  heads, tiles, batches: d = 128 0.93 - 1.01 (32 x 16 x 384 0.93, 8 x 16 x 2048 0.95), d = 64 1.00 - 1.23 up to 134 MB, then
//           0.95 - 1.00; tiles innermost 0.93 - 1.27: tiles start from the longest on, and the longest of the last heads start late
// (In short runs 8 x 16 x 8192 x 128 3892 -> 3164 us, 4 x 16 x 4096 x 128 462 -> 415, 8 x 16 x 2048 x 128 causal 156 -> 145; in a
// stream of passes, all at 985 W, 4695 -> 3600 at 1025 and 1440 MHz, 541 -> 476 at 1305 and 1470, 183 -> 169 at 1455 and 1567.)
static int tile_order(int D, const FaParams& p) {
  const double kv_mb = 4e-6 * p.B * p.H * double(p.S) * D;
  if (p.causal) return D == 128 || kv_mb > 200 ? FA_ORDER_HEADS_TILES : FA_ORDER_HEADS_BATCHES;
  return D == 128 || kv_mb > 100 ? FA_ORDER_TILES_HEADS : FA_ORDER_HEADS_BATCHES;
}

// `quad`: four_tiles_per_sm, for which the boxes of K and V were made.
static int launch_fa_long(int D, bool quad, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, FaParams p, cudaStream_t s) {
  p.order = tile_order(D, p);
  if (D == 128) return launch_fa_pipe<128, 2, 2>(tq, tk, tv, p, s);
  if (quad) return launch_fa_tiles(flash_attn_quad_kernel, 128, FAQ_THREADS, faq_smem_bytes(), tq, tk, tv, p, s);
  if (three_tiles_per_sm(D, p)) return launch_fa_tiles(flash_attn_tri_kernel, 128, FAT_THREADS, fat_smem_bytes(), tq, tk, tv, p, s);
  return one_tile_per_cta(p) ? launch_fa_pipe<64, 1, 2>(tq, tk, tv, p, s) : launch_fa_pipe<64, 2, 3>(tq, tk, tv, p, s);
}

// One key block holds the sequence up to 128 tokens.
static int launch_fa(int D, bool quad, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaParams& p, cudaStream_t s) {
  if (p.S > FA_BKV) return launch_fa_long(D, quad, tq, tk, tv, p, s);
  return D == 64 ? launch_fa_short<64>(tq, tk, tv, p, s) : launch_fa_short<128>(tq, tk, tv, p, s);
}

// The load engine works through the rows of a box that lie beyond the sequence too: one of 24 tokens loads 32 rows.
static int fa_box_rows(int S) { return S >= FA_BKV ? FA_BKV : (S + 15) / 16 * 16; }
static uint32_t fa_key_box_rows(bool quad, int S) { return quad ? FAQ_KEYS : uint32_t(fa_box_rows(S)); }

}  // namespace zen

using namespace zen;

ZEN_DEFINE_TU_STATUS(flash_attn)

extern "C" unsigned zen_attention_plan(int B, int H, int S, int D, int causal, int int8_copy) {
  return four_tiles_per_sm(B, H, S, D, causal != 0, int8_copy != 0, 0u) ? ZEN_ATTN_KEYS_64 : ZEN_ATTN_KEYS_128;
}

extern "C" int zen_flash_attention_f16(const void* q, const void* k, const void* v, void* o, int8_t* oq, float o_scale,
                                       int B, int H, int S, int D, int64_t q_sb, int64_t q_sh, int64_t q_ss,
                                       int64_t k_sb, int64_t k_sh, int64_t k_ss, int64_t v_sb, int64_t v_sh,
                                       int64_t v_ss, int64_t o_sb, int64_t o_sh, int64_t o_ss, const int32_t* kv_lens,
                                       int causal, float scale, void* stream) {
  return zen_flash_attention_f16_ex(q, k, v, o, oq, o_scale, B, H, S, D, q_sb, q_sh, q_ss, k_sb, k_sh, k_ss, v_sb, v_sh, v_ss, o_sb, o_sh,
                                    o_ss, kv_lens, causal, scale, 0u, stream);
}

extern "C" int zen_flash_attention_f16_ex(const void* q, const void* k, const void* v, void* o, int8_t* oq, float o_scale,
                                          int B, int H, int S, int D, int64_t q_sb, int64_t q_sh, int64_t q_ss,
                                          int64_t k_sb, int64_t k_sh, int64_t k_ss, int64_t v_sb, int64_t v_sh,
                                          int64_t v_ss, int64_t o_sb, int64_t o_sh, int64_t o_ss, const int32_t* kv_lens,
                                          int causal, float scale, unsigned flags, void* stream) {
  if (!q || !k || !v || !o || B <= 0 || H <= 0 || S <= 0 || !attn_flags_ok(flags)) return ZEN_ERR_INVALID_ARG;
  if (D != 64 && D != 128) return ZEN_ERR_UNSUPPORTED;
  if (H > 65535 || B > 65535) return ZEN_ERR_UNSUPPORTED;
  if (oq && !(o_scale > 0.f)) return ZEN_ERR_INVALID_ARG;
  if (reinterpret_cast<uintptr_t>(o) % 16 || o_sb % 8 || o_sh % 8 || o_ss % 8) return ZEN_ERR_UNSUPPORTED;
  if (oq && (reinterpret_cast<uintptr_t>(oq) % 16 || o_sb % 16 || o_sh % 16 || o_ss % 16)) return ZEN_ERR_UNSUPPORTED;
  FaParams p{};
  p.o = o; p.oq = oq; p.o_scale = o_scale; p.inv_o_scale = oq ? 1.0f / o_scale : 1.0f; p.B = B; p.H = H; p.S = S;
  p.o_sb = o_sb; p.o_sh = o_sh; p.o_ss = o_ss; p.kv_lens = kv_lens; p.causal = causal ? 1 : 0;
  const SoftmaxScale sc = softmax_scale(scale);
  p.scale_log2 = sc.log2; p.qk_negate = sc.negate;
  p.box_rows = fa_box_rows(S);
  const bool quad = four_tiles_per_sm(B, H, S, D, causal != 0, oq != nullptr, flags);
  CUtensorMap tq, tk, tv;
  int st = encode_qkv_map(&tq, q, B, H, S, D, q_sb, q_sh, q_ss, p.q_perm, uint32_t(p.box_rows));
  if (st == ZEN_OK) st = encode_qkv_map(&tk, k, B, H, S, D, k_sb, k_sh, k_ss, p.k_perm, fa_key_box_rows(quad, S));
  if (st == ZEN_OK) st = encode_qkv_map(&tv, v, B, H, S, D, v_sb, v_sh, v_ss, p.v_perm, fa_key_box_rows(quad, S));
  if (st != ZEN_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return launch_fa(D, quad, tq, tk, tv, p, s);
}

extern "C" int zen_convert3_f32_to_f16(const float* a, const float* b, const float* c, void* y, int64_t n, void* stream);

extern "C" size_t zen_flash_attention_f32_workspace_bytes(int B, int H, int S, int D) {
  if (B <= 0 || H <= 0 || S <= 0 || D <= 0) return 0;
  return size_t(3) * size_t(B) * size_t(H) * size_t(S) * size_t(D) * 2;
}

// Whether the attention kernel converts fp32 operands itself, in one launch.  Measured for 230 shapes, time against the two
// launches: up to 128 keys 0.39 - 0.96 at 8 .. 1500 items and 0.70 - 0.94 at 1500 .. 6000 of 48 or more (three of them, or two,
// are converted at a time), but 0.91 - 1.18 at 3000 .. 6000 of 16 and 33; longer sequences
// 0.62 - 0.97 with a tile per SM at most (12 heads x 197: 10.4 -> 7.4 us a call, 18 x 1024: 16.6 -> 16.0), but at head size 128 up
// to 1.04 from 600 causal keys on; 1.04 - 1.8 beyond: K and V are converted once per tile, and one CTA fits an SM.
static bool f32_in_one_launch(int B, int H, int S, int D) {
  const int64_t tiles = int64_t((S + 127) / 128) * H * B;
  if (S > FA_BKV) return tiles <= num_sms() && (D == 64 ? S <= 1024 : S <= 512);
  return S >= 48 || tiles <= 10 * num_sms();
}

extern "C" int zen_flash_attention_f32_direct(const float* q, const float* k, const float* v, float* o, int B, int H, int S, int D,
                                              const int32_t* kv_lens, int causal, float scale, void* stream) {
  if (!q || !k || !v || !o || B <= 0 || H <= 0 || S <= 0) return ZEN_ERR_INVALID_ARG;
  if (D != 64 && D != 128) return ZEN_ERR_UNSUPPORTED;
  if (H > 65535 || B > 65535) return ZEN_ERR_UNSUPPORTED;
  if (reinterpret_cast<uintptr_t>(o) % 16) return ZEN_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) % 16 || !f32_in_one_launch(B, H, S, D))
    return ZEN_ERR_NEEDS_WORKSPACE;
  FaParams p{};
  p.o = o; p.o_f32 = 1; p.q32 = q; p.k32 = k; p.v32 = v; p.B = B; p.H = H; p.S = S;
  p.o_sb = int64_t(H) * S * D; p.o_sh = int64_t(S) * D; p.o_ss = D; p.kv_lens = kv_lens; p.causal = causal ? 1 : 0;
  const SoftmaxScale sc = softmax_scale(scale);
  p.scale_log2 = sc.log2; p.qk_negate = sc.negate;
  p.box_rows = fa_box_rows(S);
  const CUtensorMap none{};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (S <= FA_BKV)
    return D == 64 ? launch_fa_short<64, true>(none, none, none, p, s) : launch_fa_short<128, true>(none, none, none, p, s);
  return D == 64 ? launch_fa_pipe<64, 1, 2, true>(none, none, none, p, s) : launch_fa_pipe<128, 1, 2, true>(none, none, none, p, s);
}

extern "C" int zen_flash_attention_f32(const float* q, const float* k, const float* v, float* o, int B, int H, int S, int D,
                                       const int32_t* kv_lens, int causal, float scale, void* workspace, size_t workspace_bytes,
                                       void* stream) {
  if (!q || !k || !v || !o || !workspace || B <= 0 || H <= 0 || S <= 0) return ZEN_ERR_INVALID_ARG;
  if (D != 64 && D != 128) return ZEN_ERR_UNSUPPORTED;
  if (H > 65535 || B > 65535) return ZEN_ERR_UNSUPPORTED;
  if (workspace_bytes < zen_flash_attention_f32_workspace_bytes(B, H, S, D)) return ZEN_ERR_INVALID_ARG;
  // (the operands may lie anywhere: the conversion has a form for them)
  if (reinterpret_cast<uintptr_t>(o) % 16 || reinterpret_cast<uintptr_t>(workspace) % 16) return ZEN_ERR_UNSUPPORTED;
  if (const int st = zen_flash_attention_f32_direct(q, k, v, o, B, H, S, D, kv_lens, causal, scale, stream); st != ZEN_ERR_NEEDS_WORKSPACE) return st;
  const int64_t n = int64_t(B) * H * S * D;
  if (int st = zen_convert3_f32_to_f16(q, k, v, workspace, n, stream); st != ZEN_OK) return st;
  const __half* w = static_cast<const __half*>(workspace);
  FaParams p{};
  p.o = o; p.o_f32 = 1; p.B = B; p.H = H; p.S = S;
  p.o_sb = int64_t(H) * S * D; p.o_sh = int64_t(S) * D; p.o_ss = D; p.kv_lens = kv_lens; p.causal = causal ? 1 : 0;
  const SoftmaxScale sc = softmax_scale(scale);
  p.scale_log2 = sc.log2; p.qk_negate = sc.negate;
  p.box_rows = fa_box_rows(S);
  const bool quad = four_tiles_per_sm(B, H, S, D, causal != 0, false, 0u);
  CUtensorMap tq, tk, tv;
  int st = encode_qkv_map(&tq, w, B, H, S, D, p.o_sb, p.o_sh, D, p.q_perm, uint32_t(p.box_rows));
  if (st == ZEN_OK) st = encode_qkv_map(&tk, w + n, B, H, S, D, p.o_sb, p.o_sh, D, p.k_perm, fa_key_box_rows(quad, S));
  if (st == ZEN_OK) st = encode_qkv_map(&tv, w + 2 * n, B, H, S, D, p.o_sb, p.o_sh, D, p.v_perm, fa_key_box_rows(quad, S));
  if (st != ZEN_OK) return st;
  return launch_fa(D, quad, tq, tk, tv, p, static_cast<cudaStream_t>(stream));
}

extern "C" int zen_flash_attention_unpadded_f16(const void* q, const void* k, const void* v, void* o, int8_t* oq, float o_scale,
                                                int B, int H, int max_seqlen, int D, int64_t rows, int64_t q_st, int64_t q_sh,
                                                int64_t k_st, int64_t k_sh, int64_t v_st, int64_t v_sh, int64_t o_st,
                                                int64_t o_sh, const int32_t* cu_seqlens, int causal, float scale,
                                                void* stream) {
  return zen_flash_attention_unpadded_f16_ex(q, k, v, o, oq, o_scale, B, H, max_seqlen, D, rows, q_st, q_sh, k_st, k_sh, v_st, v_sh, o_st,
                                             o_sh, cu_seqlens, causal, scale, 0u, stream);
}

extern "C" int zen_flash_attention_unpadded_f16_ex(const void* q, const void* k, const void* v, void* o, int8_t* oq, float o_scale,
                                                   int B, int H, int max_seqlen, int D, int64_t rows, int64_t q_st, int64_t q_sh,
                                                   int64_t k_st, int64_t k_sh, int64_t v_st, int64_t v_sh, int64_t o_st,
                                                   int64_t o_sh, const int32_t* cu_seqlens, int causal, float scale,
                                                   unsigned flags, void* stream) {
  if (!q || !k || !v || !o || !cu_seqlens || B <= 0 || H <= 0 || max_seqlen <= 0 || rows <= 0 || !attn_flags_ok(flags)) return ZEN_ERR_INVALID_ARG;
  if (D != 64 && D != 128) return ZEN_ERR_UNSUPPORTED;
  if (H > 65535 || B > 65535 || rows >= (int64_t(1) << 31)) return ZEN_ERR_UNSUPPORTED;
  if (oq && !(o_scale > 0.f)) return ZEN_ERR_INVALID_ARG;
  if (reinterpret_cast<uintptr_t>(o) % 16 || o_sh % 8 || o_st % 8) return ZEN_ERR_UNSUPPORTED;
  if (oq && (reinterpret_cast<uintptr_t>(oq) % 16 || o_sh % 16 || o_st % 16)) return ZEN_ERR_UNSUPPORTED;
  FaParams p{};
  p.o = o; p.oq = oq; p.o_scale = o_scale; p.inv_o_scale = oq ? 1.0f / o_scale : 1.0f; p.B = B; p.H = H; p.S = max_seqlen;
  p.o_sb = 0; p.o_sh = o_sh; p.o_ss = o_st; p.kv_lens = nullptr; p.cu_seqlens = cu_seqlens; p.rows = int(rows);
  p.causal = causal ? 1 : 0;
  const SoftmaxScale sc = softmax_scale(scale);
  p.scale_log2 = sc.log2; p.qk_negate = sc.negate;
  // the packed tensors as ONE batch of `rows` tokens: a tile may start at any row
  CUtensorMap tq, tk, tv;
  const int R = int(rows);
  const bool quad = four_tiles_per_sm(B, H, max_seqlen, D, causal != 0, oq != nullptr, flags);
  const uint32_t key_rows = quad ? FAQ_KEYS : FA_BKV;
  int st = encode_qkv_map(&tq, q, 1, H, R, D, int64_t(R) * q_st, q_sh, q_st, p.q_perm);
  if (st == ZEN_OK) st = encode_qkv_map(&tk, k, 1, H, R, D, int64_t(R) * k_st, k_sh, k_st, p.k_perm, key_rows);
  if (st == ZEN_OK) st = encode_qkv_map(&tv, v, 1, H, R, D, int64_t(R) * v_st, v_sh, v_st, p.v_perm, key_rows);
  if (st != ZEN_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return launch_fa_long(D, quad, tq, tk, tv, p, s);
}

// Shared body of the padded and the packed entry points.  Padded: S tokens per sequence, kv_lens optional.
// Packed: `rows` valid tokens back to back, cu_seqlens[B + 1] on the device, sequences of at most 128 tokens.
static int qkv_attention_launch(bool packed, const int8_t* xq, int64_t ldx, const int8_t* wqkv, int64_t ldw, int B, int S,
                                int64_t rows, int heads, int K, float x_scale, const float* w_scale, const float* bias,
                                const int32_t* kv_lens, const int32_t* cu_seqlens, float scale, void* ctx, int8_t* ctxq,
                                float ctx_scale, void* qkv_out, const void* next0, size_t next0_bytes, const void* next1,
                                size_t next1_bytes, unsigned flags, void* stream) {
  if (!xq || !wqkv || !ctx || B <= 0 || S <= 0 || heads <= 0 || K <= 0 || rows <= 0) return ZEN_ERR_INVALID_ARG;
  if (packed && !cu_seqlens) return ZEN_ERR_INVALID_ARG;
  if ((next0_bytes != 0 && !next0) || (next1_bytes != 0 && !next1)) return ZEN_ERR_INVALID_ARG;
  if (flags & ~unsigned(ZEN_GEMM_CONST_WEIGHTS)) return ZEN_ERR_INVALID_ARG;
  if (ctxq && !(ctx_scale > 0.f)) return ZEN_ERR_INVALID_ARG;
  if (S > 128 || B > 65535 || heads > 65535) return ZEN_ERR_UNSUPPORTED;  // longer sequences: zen_linear_i8 + zen_flash_attention_f16
  if (rows >= (int64_t(1) << 31)) return ZEN_ERR_UNSUPPORTED;
  if (K % 16 || ldx % 16 || ldw % 16 || ldx < K || ldw < K) return ZEN_ERR_UNSUPPORTED;
  const int hidden = heads * 64;
  if (reinterpret_cast<uintptr_t>(ctx) % 16 || reinterpret_cast<uintptr_t>(ctxq) % 16 ||
      reinterpret_cast<uintptr_t>(qkv_out) % 16)
    return ZEN_ERR_UNSUPPORTED;
  QkvAttnParams p{};
  p.B = B; p.S = S; p.heads = heads; p.K = K;
  p.num_k_blocks = (K + 127) / 128;
  p.x_scale = x_scale; p.w_scale = w_scale; p.bias = bias; p.kv_lens = kv_lens;
  p.cu_seqlens = cu_seqlens; p.ctx = static_cast<__half*>(ctx); p.rows = int(rows);
  const SoftmaxScale sc = softmax_scale(scale);
  p.scale_log2 = sc.log2; p.qk_negate = sc.negate;
  p.ctxq = ctxq; p.ctx_scale = ctxq ? ctx_scale : 1.0f;
  p.qkv_out = static_cast<__half*>(qkv_out);
  p.early_b = (flags & ZEN_GEMM_CONST_WEIGHTS) ? 1 : 0;
  const void* next[2] = {next0, next1};
  const size_t next_bytes[2] = {next0_bytes, next1_bytes};
  for (int i = 0; i < 2; ++i) {
    const uintptr_t lo = (reinterpret_cast<uintptr_t>(next[i]) + 15u) & ~uintptr_t(15);
    const uintptr_t hi = (reinterpret_cast<uintptr_t>(next[i]) + next_bytes[i]) & ~uintptr_t(15);
    if (next_bytes[i] != 0 && hi > lo) {
      p.pf_ptr[i] = reinterpret_cast<const uint8_t*>(lo);
      p.pf_bytes[i] = uint64_t(hi - lo);
    }
  }
  CUtensorMap ta, tb, to, toq;
  if (packed) {
    // activations as (k, row of the packed batch): a tile starts at any row; rows past the end read as zero
    if (int st = encode_tmap_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, xq, uint64_t(K), uint64_t(rows), uint64_t(ldx), 128, 128);
        st != ZEN_OK)
      return st;
  } else {
    // activations as (k, token of the sequence, sequence): rows beyond S read as zero, so a tile never holds a
    // neighbouring sequence's tokens
    const uint64_t dims[3] = {uint64_t(K), uint64_t(S), uint64_t(B)};
    const uint64_t str[2] = {uint64_t(ldx), uint64_t(ldx) * uint64_t(S)};
    const uint32_t box[3] = {128u, 128u, 1u};
    if (int st = encode_tmap(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, xq, dims, str, box); st != ZEN_OK) return st;
  }
  if (int st = encode_tmap_2d(&tb, CU_TENSOR_MAP_DATA_TYPE_UINT8, wqkv, uint64_t(K), uint64_t(3) * hidden, uint64_t(ldw), 128, 64);
      st != ZEN_OK)
    return st;
  to = ta;  // the packed form stores without tensor maps
  toq = ta;
  if (!packed) {
    // outputs: ctx[b * S + s, h * 64 + d] seen as (d, seq, head, batch), 32-row boxes (one per softmax warp)
    int perm_q[3];
    if (int st = encode_qkv_map(&to, ctx, B, heads, S, 64, int64_t(S) * hidden, 64, hidden, p.o_perm, 32u, 2); st != ZEN_OK)
      return st;
    toq = to;
    if (ctxq)
      if (int st = encode_qkv_map(&toq, ctxq, B, heads, S, 64, int64_t(S) * hidden, 64, hidden, perm_q, 32u, 1); st != ZEN_OK)
        return st;
  }
  constexpr size_t smem = qkv_attn_smem_bytes();
  const int items = B * heads;
  const int grid = items < num_sms() ? items : num_sms();
  if (packed) {
    if (int st = ensure_dynamic_smem(reinterpret_cast<const void*>(qkv_attn_kernel<true>), smem); st != ZEN_OK) return st;
    return launch_pdl(PDL_GEMM, qkv_attn_kernel<true>, dim3(grid), dim3(QA_THREADS), smem, static_cast<cudaStream_t>(stream), ta,
                      tb, to, toq, p);
  }
  if (int st = ensure_dynamic_smem(reinterpret_cast<const void*>(qkv_attn_kernel<false>), smem); st != ZEN_OK) return st;
  return launch_pdl(PDL_GEMM, qkv_attn_kernel<false>, dim3(grid), dim3(QA_THREADS), smem, static_cast<cudaStream_t>(stream), ta,
                    tb, to, toq, p);
}

extern "C" int zen_qkv_attention_i8(const int8_t* xq, int64_t ldx, const int8_t* wqkv, int64_t ldw, int B, int S, int heads,
                                    int K, float x_scale, const float* w_scale, const float* bias,
                                    const int32_t* kv_lens, float scale, void* ctx, int8_t* ctxq, float ctx_scale,
                                    void* qkv_out, const void* next0, size_t next0_bytes, const void* next1,
                                    size_t next1_bytes, unsigned flags, void* stream) {
  return qkv_attention_launch(false, xq, ldx, wqkv, ldw, B, S, int64_t(B) * S, heads, K, x_scale, w_scale, bias, kv_lens,
                              nullptr, scale, ctx, ctxq, ctx_scale, qkv_out, next0, next0_bytes, next1, next1_bytes, flags,
                              stream);
}

extern "C" int zen_qkv_attention_unpadded_i8(const int8_t* xq, int64_t ldx, const int8_t* wqkv, int64_t ldw, int B,
                                             int64_t rows, const int32_t* cu_seqlens, int heads, int K, float x_scale,
                                             const float* w_scale, const float* bias, float scale, void* ctx, int8_t* ctxq,
                                             float ctx_scale, void* qkv_out, const void* next0, size_t next0_bytes,
                                             const void* next1, size_t next1_bytes, unsigned flags, void* stream) {
  return qkv_attention_launch(true, xq, ldx, wqkv, ldw, B, 128, rows, heads, K, x_scale, w_scale, bias, nullptr, cu_seqlens,
                              scale, ctx, ctxq, ctx_scale, qkv_out, next0, next0_bytes, next1, next1_bytes, flags, stream);
}
