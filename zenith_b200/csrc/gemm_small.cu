// Launches of the small-product GEMM (gemm_small.cuh).
#include "gemm_small.h"
#include "tma_host.cuh"

ZEN_DEFINE_TU_STATUS(gemm_small)

namespace zen {

template <int KIND, int KS, bool B_MN>
static int launch_ks(const CUtensorMap& ta, const CUtensorMap& tb, const GemmSmallParams& sp, cudaStream_t stream) {
  constexpr int BN = gs_bn<B_MN>();
  auto kernel = gemm_small_kernel<KIND, BN, KS, B_MN>;
  constexpr size_t smem = gs_smem_bytes<BN, KS>();
  if (int st = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem); st != ZEN_OK) return st;
  const dim3 grid(unsigned((sp.g.N + BN - 1) / BN * KS), unsigned((sp.g.M + GEMM_BM - 1) / GEMM_BM));
  return launch_kernel(kernel, LaunchShape{grid, dim3(GS_THREADS), smem, (pdl_mask() & PDL_GEMM) != 0, KS}, stream, ta, tb, sp);
}

template <int KIND, bool B_MN>
static int launch_kind(int ks, const void* A, int64_t lda, const void* B, int64_t ldb, GemmSmallParams sp, cudaStream_t stream) {
  constexpr int ELEM = GemmKind<KIND>::ELEM;
  constexpr int BK = 128 / ELEM, BN = gs_bn<B_MN>();
  constexpr CUtensorMapDataType dt = ELEM == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : ELEM == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  GemmParams& p = sp.g;
  // a box of 128 rows of which most lie outside the tensor is filled at a fraction of the speed of one that is all inside
  sp.a_rows = p.M < GEMM_BM ? (p.M + 7) / 8 * 8 : GEMM_BM;
  CUtensorMap ta, tb;
  if (int st = encode_tmap_2d(&ta, dt, A, uint64_t(p.K), uint64_t(p.M), uint64_t(lda) * ELEM, BK, uint32_t(sp.a_rows)); st != ZEN_OK) return st;
  const int st = B_MN ? encode_tmap_2d(&tb, dt, B, uint64_t(p.N), uint64_t(p.K), uint64_t(ldb) * ELEM, BN, BK)
                      : encode_tmap_2d(&tb, dt, B, uint64_t(p.K), uint64_t(p.N), uint64_t(ldb) * ELEM, BK, BN);
  if (st != ZEN_OK) return st;
  p.num_k_blocks = (p.K + BK - 1) / BK;
  if (B_MN) p.early_b = 0;
  return ks == 4 ? launch_ks<KIND, 4, B_MN>(ta, tb, sp, stream) : launch_ks<KIND, 2, B_MN>(ta, tb, sp, stream);
}

int launch_gemm_small(int kind, int ks, bool b_mn, const void* A, int64_t lda, const void* B, int64_t ldb, const GemmParams& g, cudaStream_t stream) {
  const GemmSmallParams sp{g, 0};
  if ((g.M + GEMM_BM - 1) / GEMM_BM > 65535) return ZEN_ERR_UNSUPPORTED;
  switch (kind) {
    case KIND_I8: return launch_kind<KIND_I8, false>(ks, A, lda, B, ldb, sp, stream);
    case KIND_F8: return launch_kind<KIND_F8, false>(ks, A, lda, B, ldb, sp, stream);
    case KIND_TF32: return launch_kind<KIND_TF32, false>(ks, A, lda, B, ldb, sp, stream);
    default: return b_mn ? launch_kind<KIND_F16, true>(ks, A, lda, B, ldb, sp, stream) : launch_kind<KIND_F16, false>(ks, A, lda, B, ldb, sp, stream);
  }
}

}  // namespace zen
