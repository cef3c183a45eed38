// Host entry of the small-product GEMM (gemm_small.cu) and of the dispatch among all GEMM kernels (gemm.cu).
#pragma once
#include "gemm_small.cuh"

namespace zen {

// ZEN_GEMM_SPLIT_K field of a call's flags: K split of the small-product kernel (1, 2, 4, 8), 15 = never that kernel,
// 0 = chosen by shape; ZEN_GEMM_NARROW: its 32-column tile.
inline int forced_split(unsigned flags) { return int((flags >> 20) & 0xfu); }
inline int forced_small_bn(unsigned flags) { return (flags & ZEN_GEMM_NARROW) ? 32 : 64; }

struct SmallChoice {
  int bn, ks;  // ks 0: the product runs on the large-tile kernels
};

// When a product runs on the small-product kernel (measured per launch in a graph, N = 768 .. 4096, K = 768 .. 4096).
// 32-column tiles beat 64-column ones throughout (one exchange-and-epilogue step instead of two).  K is split while
// every CTA keeps three k-blocks (below that the exchange costs more than the blocks; before a LayerNorm one and a half,
// because the fp32 rows then also leave in narrower pieces), and while the CTAs fit the chip: 192 is where a second CTA
// on some SMs still pays, with a deep K two per SM everywhere.  Beyond, the persistent kernels win (3072 x 768 at 385
// rows: 6.1 us against 7.9).  Without a split they are within 5 % of each other.
//   2.4 MB of weights, 24 rows: K 3072 -> 768 9.5 -> 3.6 us; 128 rows: 9.7 -> 3.9; 512 rows 9.7 -> 5.2; 768 rows 9.8 -> 6.1.
inline SmallChoice small_rule(int elem_bytes, int M, int N, int K, bool layernorm) {
  const long kb = (long(K) * elem_bytes + 127) / 128;
  const long tiles = long((M + GEMM_BM - 1) / GEMM_BM) * ((N + 31) / 32);
  if (tiles * 4 <= 192 && kb >= (layernorm ? 6 : 12)) return {32, 4};
  if (tiles * 2 <= (kb >= 16 ? 296 : 192) && kb >= 4) return {32, 2};
  return {64, 0};
}

// Form of a projection + residual + LayerNorm: the value of the ZEN_GEMM_SPLIT_K field, 15 = one kernel (four-CTA clusters),
// 14 = large-tile GEMM with fp32 output and a LayerNorm of its rows, else the small-product kernel and that LayerNorm.  A
// round of the clusters (37 row blocks) takes 9.5 - 10.4 us (K 768) or 16.4 (K 3072) whatever it holds; the two launches
// take 7.4 / 10.5 us at 1024 rows, 10.3 / 14.1 at 2048, 12 / 17 at 4096, 18 / 25 at 4864 against 19.6 / 30.9, 25 / 32 at
// 7680 against 20 / 31: they win in a first round that is not full and where a further round would hold little.  At hidden
// 1024 a cluster CTA holds 256 columns in a two-stage ring and never wins.
inline SmallChoice layernorm_rule(int elem_bytes, int M, int N, int K) {
  const SmallChoice c = small_rule(elem_bytes, M, N, K, true);
  if (c.ks > 0) return c;
  const bool deep = (long(K) * elem_bytes + 127) / 128 >= 16;
  const int blocks = (M + GEMM_BM - 1) / GEMM_BM;
  const int last = (blocks - 1) % 37 + 1;  // row blocks of the last round
  const bool two = blocks <= 37 ? last <= (deep ? 24 : 12) : last <= (deep ? 18 : 5);
  return {64, N != 768 || two ? 14 : 15};
}

// kind: KIND_*; bn: 64 or 32; ks: 1, 2, 4 or (bn 64) 8; b_mn: B is [K, N] (fp16 only, bn 64).  num_k_blocks is filled in here.
__attribute__((visibility("hidden"))) int launch_gemm_small(int kind, int bn, int ks, bool b_mn, const void* A, int64_t lda, const void* B,
                                                            int64_t ldb, const GemmParams& g, cudaStream_t stream);

// int8 or fp16 operands, B [N, K]: picks among all GEMM kernels.
__attribute__((visibility("hidden"))) int run_gemm_auto(int kind, const void* A, int64_t lda, const void* B, int64_t ldb,
                                                        const GemmParams& p, unsigned flags, cudaStream_t s);

}  // namespace zen
