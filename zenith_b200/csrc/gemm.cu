// Host side of the tcgen05 GEMMs: tile selection, tensor maps, launches, C ABI.
#include "gemm_tc.cuh"
#include "gemm_pair.cuh"
#include "gemm_small.h"
#include "tma_host.cuh"
#include <mutex>

namespace zen {

// Smallest estimated time: waves of persistent CTAs x (tile width + fixed per-tile cost).  `flags` may carry a
// forced width (ZEN_GEMM_TILE_N); a width the kernel family does not have is ignored.
static int pick_bn(int M, int N, const int* allowed, int n_allowed, unsigned flags) {
  const int forced = int((flags >> 8) & 0x3ffu);
  if (forced) {
    for (int i = 0; i < n_allowed; ++i)
      if (allowed[i] == forced) return forced;
  }
  const int sms = num_sms();
  const int tiles_m = (M + GEMM_BM - 1) / GEMM_BM;
  long best_cost = -1;
  int best = allowed[0];
  for (int i = 0; i < n_allowed; ++i) {
    const int bn = allowed[i];
    const long tiles = long(tiles_m) * ((N + bn - 1) / bn);
    const long waves = (tiles + sms - 1) / sms;
    const long cost = waves * (bn + 24);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = bn;
    }
  }
  return best;
}

template <int KIND, int BN, int STAGES, bool B_MN>
static int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, GemmParams p,
                       cudaStream_t stream) {
  auto kernel = gemm_tc_kernel<KIND, BN, STAGES, B_MN>;
  constexpr size_t smem = gemm_smem_bytes<BN, STAGES>();
  if (int st = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem); st != ZEN_OK) return st;
  p.tiles_m = (p.M + GEMM_BM - 1) / GEMM_BM;
  p.tiles_n = (p.N + BN - 1) / BN;
  const int tiles = p.tiles_m * p.tiles_n;
  const int grid = tiles < num_sms() ? tiles : num_sms();
  return launch_pdl(PDL_GEMM, kernel, dim3(grid), dim3(GEMM_THREADS), smem, stream, ta, tb, tc, p);
}

template <int KIND, int BN, int STAGES>
static int launch_gemm_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, GemmParams p,
                            cudaStream_t stream) {
  auto kernel = gemm_pair_kernel<KIND, BN, STAGES>;
  constexpr size_t smem = gemm_pair_smem_bytes<BN, STAGES>();
  if (int st = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem); st != ZEN_OK) return st;
  p.tiles_m = (p.M + 2 * GEMM_BM - 1) / (2 * GEMM_BM);  // 256-row blocks
  p.tiles_n = (p.N + BN - 1) / BN;
  const int tiles = p.tiles_m * p.tiles_n;
  const int resident = max_resident_clusters(reinterpret_cast<const void*>(kernel), smem, GEMM_THREADS, 2);
  const int pairs = tiles < resident ? tiles : resident;
  return launch_kernel(kernel, LaunchShape{dim3(unsigned(2 * pairs)), dim3(GEMM_THREADS), smem, (pdl_mask() & PDL_GEMM) != 0, 2}, stream,
                       ta, tb, tc, p);
}

template <int KIND>
static CUtensorMapDataType tmap_dtype() {
  return (KIND == KIND_I8 || KIND == KIND_F8) ? CU_TENSOR_MAP_DATA_TYPE_UINT8
         : KIND == KIND_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                            : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
}

// A [M,K] (row stride lda elements); B K-major [N,K] (ldb) or MN-major [K,N] (ldb).
// PAIR: the CTA-pair kernel (gemm_pair.cuh); each CTA then copies BN / 2 rows of B per k-block.
template <int KIND, int BN, int STAGES, bool B_MN, bool PAIR = false>
static int run_gemm(const void* A, int64_t lda, const void* B, int64_t ldb, GemmParams p, cudaStream_t stream) {
  static_assert(!(PAIR && B_MN), "the pair kernel takes K-major B only");
  constexpr int ELEM = GemmKind<KIND>::ELEM;
  constexpr int BK = 128 / ELEM;
  CUtensorMap ta, tb;
  int st = encode_tmap_2d(&ta, tmap_dtype<KIND>(), A, uint64_t(p.K), uint64_t(p.M), uint64_t(lda) * ELEM, BK, GEMM_BM);
  if (st != ZEN_OK) return st;
  if (!B_MN) st = encode_tmap_2d(&tb, tmap_dtype<KIND>(), B, uint64_t(p.K), uint64_t(p.N), uint64_t(ldb) * ELEM, BK, PAIR ? BN / 2 : BN);
  else st = encode_tmap_2d(&tb, tmap_dtype<KIND>(), B, uint64_t(p.N), uint64_t(p.K), uint64_t(ldb) * ELEM, BK, BK);
  if (st != ZEN_OK) return st;
  p.num_k_blocks = (p.K + BK - 1) / BK;
  // Outputs with 16-byte aligned rows leave through shared memory: fp16 / int8 by TMA stores of 32-row blocks, one slab
  // wide, 4-byte types as row pieces; anything else is stored by the epilogue threads directly
  CUtensorMap tc = ta;
  p.staged_store = 0;
  const int oelem = p.out_dtype == ZEN_DT_S8 ? 1 : p.out_dtype == ZEN_DT_F16 ? 2 : 4;
  // (a TMA store clips a row at N rounded up to 16 bytes: the rest of that unit may be the caller's next columns)
  if (reinterpret_cast<uintptr_t>(p.out) % 16 == 0 && (p.ldo * oelem) % 16 == 0 && (oelem == 4 || (int64_t(p.N) * oelem) % 16 == 0)) {
    p.staged_store = 1;
    if (oelem < 4) {
      constexpr int SLAB = gemm_slab_cols<BN>();
      const int row_bytes = SLAB * oelem;
      st = encode_tmap_2d(&tc, p.out_dtype == ZEN_DT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8,
                          p.out, uint64_t(p.N), uint64_t(p.M), uint64_t(p.ldo) * oelem, SLAB, 32,
                          row_bytes == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                          : row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                          : row_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                            : CU_TENSOR_MAP_SWIZZLE_NONE);
      if (st != ZEN_OK) return st;
    }
  }
  if constexpr (PAIR) return launch_gemm_pair<KIND, BN, STAGES>(ta, tb, tc, p, stream);
  else return launch_gemm<KIND, BN, STAGES, B_MN>(ta, tb, tc, p, stream);
}

// Whether a GEMM of this shape runs on CTA pairs.  ZEN_GEMM_PAIR / ZEN_GEMM_NO_PAIR force the choice.  A pair
// moves a third fewer operand bytes per operation but starts and ends more slowly (cluster scheduling, two
// cluster-wide rendezvous), and it does nothing for the epilogue: it pays when the main loop dominates, i.e. for
// large products, and for the GELU + requantisation epilogue only with a deep K (measured on 11 shapes: wins of
// 8 - 17 % above the thresholds, losses of 3 - 9 % below them).  fp16 operands are twice the bytes and twice the
// tensor work per element while the epilogue stays the same, and its threshold is lower: of 18 shapes of 2048 - 16384 rows
// those from 2^33 multiply-adds on gained 2 - 14 % (4096 x 3072 x 768: 21.6 -> 20.2 us, 12288 x 1024 x 1024: 24.4 -> 22.5,
// 3000 x 4096 x 1024: 28.3 -> 24.5), those below lost 1 - 8 %.  Deep int8 products
// with a light epilogue gain from 2^34.5 on (12288 x 768 x 3072: 27.8 -> 25.2 us, 6000 x 1024 x 4096: 22.1 -> 20.4), shallower
// ones gain alone but not between other kernels (8192 x 3072 x 1024: 24.4 -> 23.7, its encoder 4286 -> 4304 us).
static bool use_pair(int kind, int M, int N, int K, bool heavy_epilogue, unsigned flags) {
  if (flags & ZEN_GEMM_NO_PAIR) return false;
  if (flags & ZEN_GEMM_PAIR) return true;
  const double work = double(M) * double(N) * double(K);
  const double from = kind == KIND_F16                 ? 8589934592.0    // 2^33
                      : !heavy_epilogue && K >= 2048 ? 24296004000.0   // 2^34.5
                                                     : 34359738368.0;  // 2^35
  return M >= 1024 && work >= from && (!heavy_epilogue || K >= 4096);
}

// Pair tile width: fewest rounds of the resident pairs, wider tiles preferred on a tie (less traffic per operation).  A tile
// of 128 columns reads as much of A as one of 256 and is dearer than its columns (fp16 3700 x 3072 x 768: five rounds of 128
// 21.2 us, three of 256 19.8).
static int pick_bn_pair(int M, int N, unsigned flags) {
  static const int allowed[] = {256, 192, 128};
  const int forced = int((flags >> 8) & 0x3ffu);
  for (int bn : allowed)
    if (bn == forced) return bn;
  const int pairs = num_sms() / 2;
  const int tiles_m = (M + 2 * GEMM_BM - 1) / (2 * GEMM_BM);
  long best_cost = -1;
  int best = allowed[0];
  for (int bn : allowed) {
    const long tiles = long(tiles_m) * ((N + bn - 1) / bn);
    const long rounds = (tiles + pairs - 1) / pairs;
    const long cost = rounds * (bn + (bn == 128 ? 40 : 24));
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = bn;
    }
  }
  return best;
}

// K split of a product on the small-product kernel (0: not there), by shape or as the flags say.  A forced tile width or pair
// choice is about the large-tile kernels.
static int use_small(int kind, int M, int N, int K, unsigned flags) {
  const int elem = kind == KIND_F16 ? 2 : kind == KIND_TF32 ? 4 : 1;
  if (const int f = forced_split(flags); f != 0) return f == 15 ? 0 : nearest_split(f, (long(K) * elem + 127) / 128);
  if (flags & (ZEN_GEMM_PAIR | ZEN_GEMM_NO_PAIR | (0x3ffu << 8))) return 0;
  return small_rule(elem, M, N, K, false);
}

// out[c, r] = in[r, c] for a row-major [rows, cols] fp32 matrix, 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256) transpose_f32_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                            int rows, int cols) {
  grid_launch_dependents();  // the GEMM behind this kernel sets itself up meanwhile
  __shared__ float tile[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int i = ty; i < 32; i += 8) {
    const int r = r0 + i, c = c0 + tx;
    if (r < rows && c < cols) tile[i][tx] = in[size_t(r) * cols + c];
  }
  __syncthreads();
  for (int i = ty; i < 32; i += 8) {
    const int c = c0 + i, r = r0 + tx;
    if (r < rows && c < cols) out[size_t(c) * rows + r] = tile[tx][i];
  }
}

static int launch_transpose_f32(const float* in, float* out, int rows, int cols, cudaStream_t s) {
  dim3 grid((cols + 31) / 32, (rows + 31) / 32);
  if (grid.y > 65535) return ZEN_ERR_UNSUPPORTED;
  return launch_kernel(transpose_f32_kernel, LaunchShape{grid, dim3(256)}, s, in, out, rows, cols);
}

// int8 or fp16 operands, B K-major: the small-product kernel, CTA pairs or the one-CTA kernel by shape (or by `flags`).
int run_gemm_auto(int kind, const void* A, int64_t lda, const void* B, int64_t ldb, const GemmParams& p, unsigned flags, cudaStream_t s) {
  static const int allowed[] = {64, 128, 192, 256};
  if (const int ks = use_small(kind, p.M, p.N, p.K, flags); ks > 0) return launch_gemm_small(kind, ks, false, A, lda, B, ldb, p, s);
  if (kind == KIND_I8) {
    if (use_pair(kind, p.M, p.N, p.K, p.out_dtype == ZEN_DT_S8 && p.act == ZEN_ACT_GELU, flags)) {
      switch (pick_bn_pair(p.M, p.N, flags)) {
        case 128: return run_gemm<KIND_I8, 128, 6, false, true>(A, lda, B, ldb, p, s);
        case 192: return run_gemm<KIND_I8, 192, 5, false, true>(A, lda, B, ldb, p, s);
        default: return run_gemm<KIND_I8, 256, 4, false, true>(A, lda, B, ldb, p, s);
      }
    }
    switch (pick_bn(p.M, p.N, allowed, 4, flags)) {
      case 64: return run_gemm<KIND_I8, 64, 7, false>(A, lda, B, ldb, p, s);
      case 128: return run_gemm<KIND_I8, 128, 5, false>(A, lda, B, ldb, p, s);
      case 192: return run_gemm<KIND_I8, 192, 4, false>(A, lda, B, ldb, p, s);
      default: return run_gemm<KIND_I8, 256, 3, false>(A, lda, B, ldb, p, s);
    }
  }
  if (use_pair(kind, p.M, p.N, p.K, false, flags)) {
    switch (pick_bn_pair(p.M, p.N, flags)) {
      case 128: return run_gemm<KIND_F16, 128, 6, false, true>(A, lda, B, ldb, p, s);
      case 192: return run_gemm<KIND_F16, 192, 5, false, true>(A, lda, B, ldb, p, s);
      default: return run_gemm<KIND_F16, 256, 4, false, true>(A, lda, B, ldb, p, s);
    }
  }
  switch (pick_bn(p.M, p.N, allowed, 4, flags)) {
    case 64: return run_gemm<KIND_F16, 64, 7, false>(A, lda, B, ldb, p, s);
    case 128: return run_gemm<KIND_F16, 128, 5, false>(A, lda, B, ldb, p, s);
    case 192: return run_gemm<KIND_F16, 192, 4, false>(A, lda, B, ldb, p, s);
    default: return run_gemm<KIND_F16, 256, 3, false>(A, lda, B, ldb, p, s);
  }
}

}  // namespace zen

using namespace zen;

ZEN_DEFINE_TU_STATUS(gemm)

extern "C" {

int zen_version(void) { return ZEN_VERSION; }

unsigned zen_gemm_plan(int elem_bytes, int rows, int N, int K, int layernorm) {
  if ((elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4) || rows <= 0 || N <= 0 || K <= 0) return 0u;
  const int form = layernorm ? layernorm_rule(elem_bytes, rows, N, K) : small_rule(elem_bytes, rows, N, K, false);
  return ZEN_GEMM_SPLIT_K(form > 0 ? form : 15);
}

const char* zen_status_string(int s) {
  switch (s) {
    case ZEN_OK: return "ok";
    case ZEN_ERR_INVALID_ARG: return "invalid argument";
    case ZEN_ERR_UNSUPPORTED: return "unsupported shape, stride or alignment";
    case ZEN_ERR_LAUNCH: return "kernel launch failed";
    case ZEN_ERR_TIMEOUT: return "a bounded device-side wait ran out";
    case ZEN_ERR_DRIVER: return "tensor-map encoding unavailable or failed";
    case ZEN_ERR_TOO_LARGE: return "request exceeds a fixed capacity";
    case ZEN_ERR_NEEDS_WORKSPACE: return "this call needs the form with a workspace";
    default: return "unknown status";
  }
}

static bool flags_ok(unsigned flags) {
  const unsigned bn = (flags >> 8) & 0x3ffu;
  if (flags & ~(ZEN_GEMM_CONST_WEIGHTS | ZEN_GEMM_PAIR | ZEN_GEMM_NO_PAIR | ZEN_GEMM_NARROW | (0x3ffu << 8) | (0xfu << 20))) return false;
  const int ks = forced_split(flags);
  if (ks != 0 && ks != 1 && ks != 2 && ks != 4 && ks != 8 && ks != 15) return false;
  if ((flags & ZEN_GEMM_PAIR) && (flags & ZEN_GEMM_NO_PAIR)) return false;
  return bn == 0 || bn == 64 || bn == 128 || bn == 192 || bn == 256;
}

int zen_linear_i8(const int8_t* xq, int64_t ldx, const int8_t* wq, int64_t ldw, int M, int N, int K, float x_scale,
                  const float* w_scale, const float* bias, int act, int out_dtype, float out_scale, int round_mode,
                  void* out, int64_t ldo, void* stream) {
  return zen_linear_i8_ex(xq, ldx, wq, ldw, M, N, K, x_scale, w_scale, bias, act, out_dtype, out_scale, round_mode, out,
                          ldo, nullptr, 0, nullptr, 0, 0u, stream);
}

int zen_linear_i8_prefetch(const int8_t* xq, int64_t ldx, const int8_t* wq, int64_t ldw, int M, int N, int K,
                           float x_scale, const float* w_scale, const float* bias, int act, int out_dtype,
                           float out_scale, int round_mode, void* out, int64_t ldo, const void* next0,
                           size_t next0_bytes, const void* next1, size_t next1_bytes, void* stream) {
  return zen_linear_i8_ex(xq, ldx, wq, ldw, M, N, K, x_scale, w_scale, bias, act, out_dtype, out_scale, round_mode, out,
                          ldo, next0, next0_bytes, next1, next1_bytes, 0u, stream);
}

int zen_linear_i8_ex(const int8_t* xq, int64_t ldx, const int8_t* wq, int64_t ldw, int M, int N, int K, float x_scale,
                     const float* w_scale, const float* bias, int act, int out_dtype, float out_scale, int round_mode,
                     void* out, int64_t ldo, const void* next0, size_t next0_bytes, const void* next1,
                     size_t next1_bytes, unsigned flags, void* stream) {
  if (!xq || !wq || !out || M <= 0 || N <= 0 || K <= 0 || !flags_ok(flags)) return ZEN_ERR_INVALID_ARG;
  if ((next0_bytes != 0 && !next0) || (next1_bytes != 0 && !next1)) return ZEN_ERR_INVALID_ARG;
  if (out_dtype < ZEN_DT_S32 || out_dtype > ZEN_DT_S8 || act < ZEN_ACT_NONE || act > ZEN_ACT_RELU)
    return ZEN_ERR_INVALID_ARG;
  if (round_mode != ZEN_ROUND_NEAREST_EVEN && round_mode != ZEN_ROUND_TRUNC) return ZEN_ERR_INVALID_ARG;
  if (out_dtype == ZEN_DT_S8 && !(out_scale > 0.0f)) return ZEN_ERR_INVALID_ARG;
  if (K % 16 || ldx % 16 || ldw % 16 || ldx < K || ldw < K || ldo < N) return ZEN_ERR_UNSUPPORTED;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K;
  p.out = out; p.ldo = ldo; p.out_dtype = out_dtype; p.act = act; p.round_mode = round_mode;
  p.x_scale = x_scale; p.out_scale = out_scale; p.w_scale = w_scale; p.bias = bias;
  p.early_b = (flags & ZEN_GEMM_CONST_WEIGHTS) ? 1 : 0;
  const void* next[2] = {next0, next1};
  const size_t next_bytes[2] = {next0_bytes, next1_bytes};
  for (int i = 0; i < 2; ++i) {
    // whole 16-byte units only: a hint may skip the ragged ends
    const uintptr_t lo = (reinterpret_cast<uintptr_t>(next[i]) + 15u) & ~uintptr_t(15);
    const uintptr_t hi = (reinterpret_cast<uintptr_t>(next[i]) + next_bytes[i]) & ~uintptr_t(15);
    if (next_bytes[i] != 0 && hi > lo) {
      p.pf_ptr[i] = reinterpret_cast<const uint8_t*>(lo);
      p.pf_bytes[i] = uint64_t(hi - lo);
    }
  }
  return run_gemm_auto(KIND_I8, xq, ldx, wq, ldw, p, flags, static_cast<cudaStream_t>(stream));
}

int zen_linear_f16(const void* x, int64_t ldx, const void* w, int64_t ldw, int M, int N, int K, const float* bias,
                   int act, int out_dtype, void* out, int64_t ldo, void* stream) {
  return zen_linear_f16_ex(x, ldx, w, ldw, M, N, K, bias, act, out_dtype, out, ldo, 0u, stream);
}

int zen_linear_f16_ex(const void* x, int64_t ldx, const void* w, int64_t ldw, int M, int N, int K, const float* bias,
                      int act, int out_dtype, void* out, int64_t ldo, unsigned flags, void* stream) {
  if (!x || !w || !out || M <= 0 || N <= 0 || K <= 0 || !flags_ok(flags)) return ZEN_ERR_INVALID_ARG;
  if ((out_dtype != ZEN_DT_F32 && out_dtype != ZEN_DT_F16) || act < ZEN_ACT_NONE || act > ZEN_ACT_RELU)
    return ZEN_ERR_INVALID_ARG;
  if (K % 8 || ldx % 8 || ldw % 8 || ldx < K || ldw < K || ldo < N) return ZEN_ERR_UNSUPPORTED;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K;
  p.out = out; p.ldo = ldo; p.out_dtype = out_dtype; p.act = act;
  p.x_scale = 1.0f; p.out_scale = 1.0f; p.w_scale = nullptr; p.bias = bias;
  p.early_b = (flags & ZEN_GEMM_CONST_WEIGHTS) ? 1 : 0;
  return run_gemm_auto(KIND_F16, x, ldx, w, ldw, p, flags, static_cast<cudaStream_t>(stream));
}

int zen_linear_f8(const uint8_t* xq, int64_t ldx, const uint8_t* wq, int64_t ldw, int M, int N, int K, float x_scale,
                  const float* w_scale, const float* bias, int act, int out_dtype, void* out, int64_t ldo, unsigned flags,
                  void* stream) {
  if (!xq || !wq || !out || M <= 0 || N <= 0 || K <= 0) return ZEN_ERR_INVALID_ARG;
  if (!flags_ok(flags) || (flags & ZEN_GEMM_PAIR)) return ZEN_ERR_INVALID_ARG;
  if ((out_dtype != ZEN_DT_F32 && out_dtype != ZEN_DT_F16) || act < ZEN_ACT_NONE || act > ZEN_ACT_RELU)
    return ZEN_ERR_INVALID_ARG;
  if (K % 16 || ldx % 16 || ldw % 16 || ldx < K || ldw < K || ldo < N) return ZEN_ERR_UNSUPPORTED;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K;
  p.out = out; p.ldo = ldo; p.out_dtype = out_dtype; p.act = act;
  p.x_scale = x_scale; p.out_scale = 1.0f; p.w_scale = w_scale; p.bias = bias;
  p.early_b = (flags & ZEN_GEMM_CONST_WEIGHTS) ? 1 : 0;
  static const int allowed[] = {64, 128, 192, 256};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (const int ks = use_small(KIND_F8, M, N, K, flags); ks > 0) return launch_gemm_small(KIND_F8, ks, false, xq, ldx, wq, ldw, p, s);
  switch (pick_bn(M, N, allowed, 4, flags)) {
    case 64: return run_gemm<KIND_F8, 64, 7, false>(xq, ldx, wq, ldw, p, s);
    case 128: return run_gemm<KIND_F8, 128, 5, false>(xq, ldx, wq, ldw, p, s);
    case 192: return run_gemm<KIND_F8, 192, 4, false>(xq, ldx, wq, ldw, p, s);
    default: return run_gemm<KIND_F8, 256, 3, false>(xq, ldx, wq, ldw, p, s);
  }
}

int zen_linear_f32(const float* x, int64_t ldx, const float* w, int64_t ldw, int M, int N, int K, const float* bias,
                   int act, float* out, int64_t ldo, void* stream) {
  if (!x || !w || !out || M <= 0 || N <= 0 || K <= 0) return ZEN_ERR_INVALID_ARG;
  if (act < ZEN_ACT_NONE || act > ZEN_ACT_RELU) return ZEN_ERR_INVALID_ARG;
  if (K % 4 || ldx % 4 || ldw % 4 || ldx < K || ldw < K || ldo < N) return ZEN_ERR_UNSUPPORTED;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K;
  p.out = out; p.ldo = ldo; p.out_dtype = ZEN_DT_F32; p.act = act;
  p.x_scale = 1.0f; p.out_scale = 1.0f; p.w_scale = nullptr; p.bias = bias;
  static const int allowed[] = {64, 128, 256};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (const int ks = use_small(KIND_TF32, M, N, K, 0u); ks > 0) return launch_gemm_small(KIND_TF32, ks, false, x, ldx, w, ldw, p, s);
  switch (pick_bn(M, N, allowed, 3, 0u)) {
    case 64: return run_gemm<KIND_TF32, 64, 7, false>(x, ldx, w, ldw, p, s);
    case 128: return run_gemm<KIND_TF32, 128, 5, false>(x, ldx, w, ldw, p, s);
    default: return run_gemm<KIND_TF32, 256, 3, false>(x, ldx, w, ldw, p, s);
  }
}

int zen_wmma_matmul_f16(const void* A, const void* B, float* C, int M, int N, int K, void* stream) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return ZEN_ERR_INVALID_ARG;
  if (K % 8 || N % 8) return ZEN_ERR_UNSUPPORTED;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K;
  p.out = C; p.ldo = N; p.out_dtype = ZEN_DT_F32; p.act = ZEN_ACT_NONE;
  p.x_scale = 1.0f; p.out_scale = 1.0f;
  static const int allowed[] = {64, 128, 256};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (const int ks = small_rule_mn(M, N, K); ks > 0) return launch_gemm_small(KIND_F16, ks, true, A, K, B, N, p, s);
  switch (pick_bn(M, N, allowed, 3, 0u)) {
    case 64: return run_gemm<KIND_F16, 64, 7, true>(A, K, B, N, p, s);
    case 128: return run_gemm<KIND_F16, 128, 5, true>(A, K, B, N, p, s);
    default: return run_gemm<KIND_F16, 256, 3, true>(A, K, B, N, p, s);
  }
}

size_t zen_matmul_f32_workspace_bytes(int N, int K) {
  if (N <= 0 || K <= 0) return 0;
  return size_t(N) * size_t(K) * sizeof(float);
}

int zen_matmul_f32_direct(const float* A, const float* B, float* C, int M, int N, int K, void* stream) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return ZEN_ERR_INVALID_ARG;
  if (K % 4) return ZEN_ERR_UNSUPPORTED;
  const int ks = small_rule_f32_kn(M, N, K);
  if (ks <= 0) return ZEN_ERR_NEEDS_WORKSPACE;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K;
  p.out = C; p.ldo = N; p.out_dtype = ZEN_DT_F32; p.act = ZEN_ACT_NONE;
  p.x_scale = 1.0f; p.out_scale = 1.0f;
  return launch_gemm_small(KIND_TF32, ks, true, A, K, B, N, p, static_cast<cudaStream_t>(stream));
}

int zen_matmul_f32(const float* A, const float* B, float* C, int M, int N, int K, void* workspace,
                   size_t workspace_bytes, void* stream) {
  if (!A || !B || !C || !workspace || M <= 0 || N <= 0 || K <= 0) return ZEN_ERR_INVALID_ARG;
  if (K % 4) return ZEN_ERR_UNSUPPORTED;
  if (workspace_bytes < zen_matmul_f32_workspace_bytes(N, K) || reinterpret_cast<uintptr_t>(workspace) % 16)
    return ZEN_ERR_INVALID_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (const int st = zen_matmul_f32_direct(A, B, C, M, N, K, stream); st != ZEN_ERR_NEEDS_WORKSPACE) return st;
  float* Bt = static_cast<float*>(workspace);
  int st = launch_transpose_f32(B, Bt, K, N, s);
  if (st != ZEN_OK) return st;
  return zen_linear_f32(A, K, Bt, K, M, N, K, nullptr, ZEN_ACT_NONE, C, N, stream);
}

// ------------------------------------------------------------------------------------------------
// zen_matmul_f32 without a caller workspace
// ------------------------------------------------------------------------------------------------
// Scratch for the transposed B operand, resident in every device that loads this library for as long
// as the process lives.  In host code the NAME below is only a stand-in for the symbol: it is not a
// device address and must never be handed to a kernel.  The address valid on a given device is
// obtained once per device with cudaGetSymbolAddress (scratch_for_current_device) and that pointer is
// what the kernels receive.
static __device__ __align__(256) float g_matmul_static_scratch[ZEN_MATMUL_STATIC_MAX_ELEMS];

static int scratch_for_current_device(float** out) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static float* per_device[kMaxDevices] = {};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return ZEN_ERR_LAUNCH;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (per_device[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_matmul_static_scratch) != cudaSuccess || p == nullptr) {
      cudaGetLastError();
      return ZEN_ERR_LAUNCH;
    }
    per_device[dev] = static_cast<float*>(p);
  }
  *out = per_device[dev];
  return ZEN_OK;
}

int zen_matmul_f32_static(const float* A, const float* B, float* C, int M, int N, int K, void* stream) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return ZEN_ERR_INVALID_ARG;
  if (K % 4) return ZEN_ERR_UNSUPPORTED;
  if (size_t(N) * size_t(K) > size_t(ZEN_MATMUL_STATIC_MAX_ELEMS)) return ZEN_ERR_TOO_LARGE;
  if (const int st = zen_matmul_f32_direct(A, B, C, M, N, K, stream); st != ZEN_ERR_NEEDS_WORKSPACE) return st;
  float* Bt = nullptr;
  int st = scratch_for_current_device(&Bt);
  if (st != ZEN_OK) return st;
  // every element of Bt that the GEMM reads is written by the transpose first: nothing needs clearing
  st = launch_transpose_f32(B, Bt, K, N, static_cast<cudaStream_t>(stream));
  if (st != ZEN_OK) return st;
  return zen_linear_f32(A, K, Bt, K, M, N, K, nullptr, ZEN_ACT_NONE, C, N, stream);
}

}  // extern "C"
