// GEMM for products that leave the chip idle under 128 x 128 .. 256 tiles: few rows, or narrow outputs with a deep K.
//   D[M,N] = A[M,K] . B^T with the epilogues of gemm_tc.cuh, one 128 x BN tile (BN 32; 64 for B [K, N] in fp16, whose box of 64
//   columns is one swizzle span) per cluster of KS (2 or 4) CTAs.
//
// What bounds such a product is latency: with four to a few dozen CTAs each pulling its operands through a three-stage
// ring, a K = 3072 projection of 24 rows took 9.5 us, 16 us with the fused LayerNorm (weights 2.4 MB: 0.4 us of HBM
// time).  So the tile is narrow, K is split over the KS CTAs of a cluster (k-blocks rank * nkb / KS ..), and a CTA asks
// for all its operand tiles at once.  The partial accumulators meet through distributed shared memory: CTA r owns columns
// r * BN / KS .. of the tile, every peer sends its partials of those columns to r's exchange buffer with asynchronous
// stores that r's barrier counts, and r adds them up, so the epilogue arithmetic (the longest serial part of a small
// tile) is split KS ways too.  s32 sums are exact in any order; fp32 partials are added own first, then by rank.
//
//   warp 0     TMA producer          warp 1   TMEM owner, MMA issuer
//   warps 2..9 epilogue: two warps per 32-lane TMEM quadrant, each half of the columns
//
// fp32 B [K, N] (TF32): the load engine cannot transpose, so the epilogue warps, idle until the accumulator is complete, bring
// B in: a warp reads 32 columns of four rows (coalesced, at any alignment), each lane then holds four consecutive k of one
// column and stores them as one 16-byte unit of the K-major tile, eight k-blocks ahead (four of 64 columns).  With a transposition launch in front
// 500 x 1000 x 768 took 9.2 us (6.5 now), 456 x 514 x 24 9.1 (5.2), 24 x 3072 x 768 10.7 (5.7).  What bounds the larger ones is the
// operand traffic (288 KB an SM), the smaller ones one load's latency, the exchange and the launch.
//
// 92 to 112 KB of shared memory and 32 or 64 TMEM columns per CTA, so that two CTAs fit on an SM and a kernel's CTAs become
// resident (barriers, TMEM, constant weight tiles on their way) while the previous kernel in the stream still runs.  The two
// deeper rings for fp32 B [K, N] take 196 and 212 KB: one CTA per SM, which starts when the SM is free.
#pragma once
#include "gemm_tc.cuh"

namespace zen {

constexpr int GS_EPI_WARPS = 8;
constexpr int GS_THREADS = 64 + 32 * GS_EPI_WARPS;

template <int KIND, bool B_MN>
__host__ __device__ constexpr int gs_bn() { return B_MN && KIND == KIND_F16 ? 64 : 32; }
template <int BN>
__host__ __device__ constexpr int gs_stage_bytes() { return GEMM_BM * 128 + BN * 128; }
template <int BN, int KS>
__host__ __device__ constexpr int gs_stages() { return BN == 64 ? 3 : KS == 4 ? 4 : 5; }
// Rings for one CTA per SM (a load takes 1300 clocks, so with four stages in flight a k-block takes 325): 32 and 64 columns
constexpr int GS_DEEP_STAGES = 9, GS_WIDE_STAGES = 8;

template <int BN, int KS, int STAGES>
constexpr size_t gs_smem_bytes() {
  // ring + exchange buffer (KS - 1 peers x 128 rows x BN / KS columns) + per-warp scale / bias / fold rows + control + slack
  return size_t(STAGES) * gs_stage_bytes<BN>() + size_t(KS - 1) * 128 * (BN / KS) * 4 + size_t(GS_EPI_WARPS) * 3 * 32 * 4 + 256 + 1024;
}

struct GemmSmallParams {
  GemmParams g;
  const float* b;  // fp32 B [K, N], which no tensor map describes, and its row stride
  int64_t ldb;
  int a_rows;  // rows of the A box: 128, or the rows of the only row block rounded up to 8
};

// 16 bytes into a peer CTA's shared memory, counted on a barrier of that CTA: the peer waits for bytes, so the sender needs
// neither a fence nor an arrival (a cluster fence and remote arrivals per destination cost 0.7 us each here).
__device__ __forceinline__ void st_async_v4(uint32_t cluster_addr, uint32_t cluster_bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];" ::"r"(cluster_addr),
               "r"(cluster_bar), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}

template <int W>
__device__ __forceinline__ void gs_tmem_ld(uint32_t taddr, uint32_t (&r)[W]) {
  static_assert(W == 16 || W == 8 || W == 4, "width");
  if constexpr (W == 16) tmem_ld_32x16(taddr, r);
  else if constexpr (W == 8) tmem_ld_32x8(taddr, r);
  else tmem_ld_32x4(taddr, r);
}

// W consecutive outputs of one row to global memory; `words` holds them packed.
template <typename T, int W>
__device__ __forceinline__ void gs_store(void* out, int64_t off, const uint32_t* words, int nvalid, bool vec_ok) {
  T* o = static_cast<T*>(out) + off;
  constexpr int BYTES = W * int(sizeof(T));
  if (vec_ok && nvalid >= W) {
    if constexpr (BYTES >= 16) store_words<BYTES / 4>(o, words);
    else if constexpr (BYTES == 8) *reinterpret_cast<uint2*>(o) = make_uint2(words[0], words[1]);
    else *reinterpret_cast<uint32_t*>(o) = words[0];
  } else {
    constexpr int PER = 4 / int(sizeof(T));
#pragma unroll
    for (int j = 0; j < W; ++j)
      if (j < nvalid) {
        const uint32_t v = words[j / PER] >> (8 * int(sizeof(T)) * (j % PER));
        if constexpr (sizeof(T) == 4) reinterpret_cast<uint32_t*>(o)[j] = v;
        else if constexpr (sizeof(T) == 2) reinterpret_cast<uint16_t*>(o)[j] = uint16_t(v);
        else reinterpret_cast<uint8_t*>(o)[j] = uint8_t(v);
      }
  }
}

// The requantised value by the definition (out of line: rare, and long when inlined for every column).
template <int ACT>
__device__ __noinline__ int gs_exact_requant(int acc, float x_scale, float scale, float bias, float out_scale, int round_mode) {
  return zen_det_round_clamp_i8(ZEN_DIV(zen_det_act(zen_det_dequant(acc, x_scale, scale, bias), ACT), out_scale), round_mode);
}

// Epilogue of W columns of one row: the arithmetic of epilogue_chunk / epilogue_step_s8, from registers to global memory.
template <int KIND, int ACT, int W>
__device__ __forceinline__ void gs_epilogue(const uint32_t (&a)[W], const float* sc, const float* bi, const float* fo, float risk_thr,
                                            float inv_scale, const GemmParams& p, int row, int col0, bool vec_ok) {
  const int nvalid = p.N - col0;
  if (nvalid <= 0 || row >= p.M) return;
  const int64_t off = int64_t(row) * p.ldo + col0;
  if constexpr (KIND == KIND_I8) {
    if (p.out_dtype == ZEN_DT_S32) {
      gs_store<int32_t, W>(p.out, off, a, nvalid, vec_ok);
      return;
    }
    if (p.out_dtype == ZEN_DT_S8) {
      uint32_t w[W / 4];
      if (p.round_mode == 0) {
        const uint32_t redo = requant_i8_step<ACT>(a, fo, bi, risk_thr, inv_scale, w);
        if (redo) {
#pragma unroll
          for (int j = 0; j < W; ++j)
            if (redo & (1u << j))
              patch_q_byte(w, j, gs_exact_requant<ACT>(int32_t(a[j]), p.x_scale, sc[j], bi[j], p.out_scale, 0));
        }
      } else {
#pragma unroll
        for (int j4 = 0; j4 < W / 4; ++j4) w[j4] = 0;
#pragma unroll
        for (int j = 0; j < W; ++j)
          patch_q_byte(w, j, gs_exact_requant<ACT>(int32_t(a[j]), p.x_scale, sc[j], bi[j], p.out_scale, p.round_mode));
      }
      gs_store<int8_t, W>(p.out, off, w, nvalid, vec_ok);
      return;
    }
  }
  float y[W];
  if ((KIND == KIND_I8 || KIND == KIND_F8) && ACT == ZEN_ACT_NONE && p.fold) {
#pragma unroll
    for (int j = 0; j < W; j += 2) {
      const float2 af = KIND == KIND_I8 ? make_float2(float(int32_t(a[j])), float(int32_t(a[j + 1])))
                                        : make_float2(__uint_as_float(a[j]), __uint_as_float(a[j + 1]));
      const float2 v = f2fma(af, make_float2(fo[j], fo[j + 1]), make_float2(bi[j], bi[j + 1]));
      y[j] = v.x;
      y[j + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < W; j += 2) {
      if constexpr (KIND == KIND_I8 || KIND == KIND_F8) {
        const float2 af = KIND == KIND_I8 ? make_float2(float(int32_t(a[j])), float(int32_t(a[j + 1])))
                                          : make_float2(__uint_as_float(a[j]), __uint_as_float(a[j + 1]));
        const float2 v = f2mul_then_add(f2mul(af, make_float2(p.x_scale, p.x_scale)), make_float2(sc[j], sc[j + 1]), make_float2(bi[j], bi[j + 1]));
        y[j] = v.x;
        y[j + 1] = v.y;
      } else {
        y[j] = ZEN_ADD(__uint_as_float(a[j]), bi[j]);
        y[j + 1] = ZEN_ADD(__uint_as_float(a[j + 1]), bi[j + 1]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < W; ++j) {
    if constexpr (ACT == ZEN_ACT_GELU) y[j] = KIND == KIND_I8 ? zen_det_gelu(y[j]) : gelu_fast(y[j]);
    if constexpr (ACT == ZEN_ACT_RELU) y[j] = y[j] > 0.0f ? y[j] : 0.0f;
  }
  if (p.out_dtype == ZEN_DT_F32) {
    gs_store<float, W>(p.out, off, reinterpret_cast<const uint32_t*>(y), nvalid, vec_ok);
  } else {
    uint32_t w[W / 2];
#pragma unroll
    for (int j = 0; j < W / 2; ++j) {
      const __half2 h = __floats2half2_rn(y[2 * j], y[2 * j + 1]);
      w[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    gs_store<__half, W>(p.out, off, w, nvalid, vec_ok);
  }
}

// An epilogue warp's share of the B tiles of k-blocks kb0 .. kb0 + nkb - 1: rows 4 ew .. + 3 of each block's 32, columns
// n0 + lane (+ 32).  Two blocks are stored behind one proxy fence.
template <int BN, int STAGES, int STAGE_BYTES, int A_BYTES>
__device__ __forceinline__ void load_b_transposed(const GemmSmallParams& sp, uint8_t* smem, uint64_t* full_bar, uint64_t* empty_bar, int kb0, int nkb,
                                                  int n0, int ew, int lane, volatile int* abort_flag) {
  constexpr int COLS = BN / 32;
  constexpr int AHEAD = 8 / COLS;  // k-blocks on their way
  const GemmParams& p = sp.g;
  int k_next = kb0 * 32 + 4 * ew;  // first row of the next block to fetch
  const float* src = sp.b + int64_t(k_next) * sp.ldb + n0 + lane;
  const int k_end = min(p.K, (kb0 + nkb) * 32);
  float v[AHEAD][COLS][4];
  auto fetch = [&](float (&d)[COLS][4]) {
#pragma unroll
    for (int c = 0; c < COLS; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        d[c][e] = 0.0f;
        if (n0 + lane + 32 * c < p.N && k_next + e < k_end) d[c][e] = src[int64_t(e) * sp.ldb + 32 * c];
      }
    k_next += 32;
    src += 32 * sp.ldb;
  };
#pragma unroll
  for (int i = 0; i < AHEAD; ++i) fetch(v[i]);
  int st = 0;
  uint32_t phase = 1;
#pragma unroll 1
  for (int first = 0; first < nkb; first += AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; i += 2) {
      if (first + i >= nkb) return;
      uint64_t* bar[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        bar[u] = &full_bar[st];
        if (first + i + u < nkb) {
          if (!mbar_wait_warp(&empty_bar[st], phase, abort_flag)) return;
          uint8_t* tile = smem + size_t(st) * STAGE_BYTES + A_BYTES;
#pragma unroll
          for (int c = 0; c < COLS; ++c) {
            const float(&f)[4] = v[i + u][c];
            *reinterpret_cast<float4*>(tile + (lane + 32 * c) * 128 + ((ew ^ (lane & 7)) << 4)) = make_float4(f[0], f[1], f[2], f[3]);
          }
          fetch(v[i + u]);
        }
        if (++st == STAGES) {
          st = 0;
          phase ^= 1u;
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar[0]);
        if (first + i + 1 < nkb) mbar_arrive(bar[1]);
      }
    }
  }
}

template <int KIND, int BN, int KS, bool B_MN, int STAGES>
__global__ void __launch_bounds__(GS_THREADS, 2)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmSmallParams sp) {
  constexpr int ELEM = GemmKind<KIND>::ELEM;
  constexpr int BK = 128 / ELEM, UK = 32 / ELEM;
  constexpr int A_BYTES = GEMM_BM * 128;
  constexpr int STAGE_BYTES = gs_stage_bytes<BN>();
  constexpr bool LOAD_B = KIND == KIND_TF32 && B_MN;  // the epilogue warps bring B in, K-major
  constexpr bool MN_DESC = B_MN && !LOAD_B;
  constexpr int CO = BN / KS;                  // columns this CTA finishes
  constexpr int CWARP = CO / 2;                // ... and one epilogue warp
  constexpr int CH = CWARP < 16 ? CWARP : 16;  // ... in steps of
  constexpr uint32_t IDESC =
      KIND == KIND_I8 ? make_idesc(IDESC_C_S32, IDESC_S8, IDESC_S8, 0, MN_DESC ? 1 : 0, GEMM_BM, BN)
      : KIND == KIND_F16 ? make_idesc(IDESC_C_F32, IDESC_F16, IDESC_F16, 0, MN_DESC ? 1 : 0, GEMM_BM, BN)
      : KIND == KIND_F8  ? make_idesc(IDESC_C_F32, IDESC_E4M3, IDESC_E4M3, 0, MN_DESC ? 1 : 0, GEMM_BM, BN)
                         : make_idesc(IDESC_C_F32, IDESC_TF32, IDESC_TF32, 0, MN_DESC ? 1 : 0, GEMM_BM, BN);
  static_assert((BN == gs_bn<KIND, B_MN>() || (LOAD_B && BN == 64)) && (KS == 2 || KS == 4) && (!B_MN || KIND == KIND_F16 || KIND == KIND_TF32), "forms of the kernel");
  static_assert(CH >= 4, "an epilogue warp finishes at least four columns");
  const GemmParams& p = sp.g;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* xbuf = smem + size_t(STAGES) * STAGE_BYTES;  // [KS - 1 peers][CO / 4][128 rows] 16-byte units
  float* rows = reinterpret_cast<float*>(xbuf + size_t(KS - 1) * 128 * CO * 4);
  uint8_t* ctrl = reinterpret_cast<uint8_t*>(rows + GS_EPI_WARPS * 3 * 32);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(ctrl);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* xbar = tfull_bar + 1;  // the peers' partials have arrived
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xbar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int n0 = (int(blockIdx.x) / KS) * BN;
  const int m0 = int(blockIdx.y) * GEMM_BM;
  const int kb0 = int(rank) * p.num_k_blocks / KS;
  const int nkb = (int(rank) + 1) * p.num_k_blocks / KS - kb0;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_a);
    if (!LOAD_B) tma_prefetch_desc(&tmap_b);
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full_bar[i], LOAD_B ? 1 + GS_EPI_WARPS : 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(tfull_bar, 1);
    mbar_init(xbar, 1);
    *abort_flag = 0;
    mbar_fence_init();
    mbar_arrive_expect_tx(xbar, uint32_t(KS - 1) * 128 * CO * 4);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // every CTA's exchange barrier exists before a peer's bytes are counted on it
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  grid_launch_dependents();
  if (threadIdx.x == 64) {
    // constants of later kernels (a hint)
    const uint32_t cta = blockIdx.y * gridDim.x + blockIdx.x, ctas = gridDim.x * gridDim.y;
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (p.pf_bytes[i] != 0) prefetch_slice_l2(p.pf_ptr[i], p.pf_bytes[i], cta, ctas);
  }

  if (warp == 0) {
    if (elect_one()) {
      auto load_b = [&](int kb, uint8_t* sb, uint64_t* bar) {
        if constexpr (LOAD_B) return;
        else if constexpr (B_MN) tma_load_2d(sb, &tmap_b, bar, n0, (kb0 + kb) * BK);
        else tma_load_2d(sb, &tmap_b, bar, (kb0 + kb) * BK, n0);
      };
      const uint32_t stage_tx = uint32_t(sp.a_rows * 128 + (LOAD_B ? 0 : BN * 128));
      const int first = nkb < STAGES ? nkb : STAGES;
      for (int kb = 0; kb < first; ++kb) mbar_arrive_expect_tx(&full_bar[kb], stage_tx);
      // constant weights: asked for while the previous kernel may still be running
      if (p.early_b)
        for (int kb = 0; kb < first; ++kb) load_b(kb, smem + size_t(kb) * STAGE_BYTES + A_BYTES, &full_bar[kb]);
      grid_dependency_wait();
      for (int kb = 0; kb < first; ++kb) {
        uint8_t* sa = smem + size_t(kb) * STAGE_BYTES;
        tma_load_2d(sa, &tmap_a, &full_bar[kb], (kb0 + kb) * BK, m0);
        if (!p.early_b) load_b(kb, sa + A_BYTES, &full_bar[kb]);
      }
      bool ok = true;
      int st = 0;
      uint32_t phase = 0;
      for (int kb = first; kb < nkb; ++kb) {
        uint8_t* sa = smem + size_t(st) * STAGE_BYTES;
        if (!mbar_wait(&empty_bar[st], phase, abort_flag)) {
          ok = false;
          break;
        }
        mbar_arrive_expect_tx(&full_bar[st], stage_tx);
        tma_load_2d(sa, &tmap_a, &full_bar[st], (kb0 + kb) * BK, m0);
        load_b(kb, sa + A_BYTES, &full_bar[st]);
        if (++st == STAGES) {
          st = 0;
          phase ^= 1u;
        }
      }
      if (!ok)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);  // copies in flight land before the memory is released
    }
  } else if (warp == 1) {
    if (elect_one()) {
      bool ok = true;
      int st = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < nkb; ++kb) {
        if (!mbar_wait(&full_bar[st], phase, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t a_addr = smem_u32(smem + size_t(st) * STAGE_BYTES);
        const uint32_t b_addr = a_addr + A_BYTES;
#pragma unroll
        for (int k = 0; k < BK / UK; ++k)
          issue_mma<KIND>(tmem, make_smem_desc_sw128(a_addr + k * 32, 1024, 16),
                          MN_DESC ? make_smem_desc_sw128(b_addr + k * (UK * 128), 1024, BK * 128) : make_smem_desc_sw128(b_addr + k * 32, 1024, 16),
                          IDESC, (kb | k) != 0 ? 1u : 0u);
        tc_commit(&empty_bar[st]);
        if (++st == STAGES) {
          st = 0;
          phase ^= 1u;
        }
      }
      if (ok) tc_commit(tfull_bar);
    }
  } else {
    const int ew = warp - 2, quad = warp & 3, half = ew >> 2;
    const int row = quad * 32 + lane;
    const int c0 = int(rank) * CO + half * CWARP;  // first of this warp's columns in the tile
    float* s_scale = rows + ew * 3 * 32;
    float* s_bias = s_scale + 32;
    float* s_fold = s_bias + 32;
    grid_dependency_wait();
    float sv = 1.0f, bv = 0.0f;
    if (lane < CWARP && n0 + c0 + lane < p.N) {
      if (p.w_scale != nullptr) sv = __ldg(p.w_scale + n0 + c0 + lane);
      if (p.bias != nullptr) bv = __ldg(p.bias + n0 + c0 + lane);
    }
    s_scale[lane] = sv;
    s_bias[lane] = bv;
    s_fold[lane] = ZEN_MUL(p.x_scale, sv);
    const float inv_scale = ZEN_DIV(1.0f, p.out_scale);
    const float bmax = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(fabsf(bv))));
    const float risk_thr = 0.5f - 2e-6f - inv_scale * fmaf(4.2e-7f, bmax, 1.6e-7f);  // see requant_i8_step
    __syncwarp();
    if constexpr (LOAD_B) load_b_transposed<BN, STAGES, STAGE_BYTES, A_BYTES>(sp, smem, full_bar, empty_bar, kb0, nkb, n0, ew, lane, abort_flag);
    bool ok = mbar_wait_warp(tfull_bar, 0, abort_flag);
    tc_fence_after_sync();
    const uint32_t tacc = tmem + (uint32_t(quad * 32) << 16);
    if (ok) {
      // this CTA's partials of the columns that the peers finish
#pragma unroll 1
      for (int i = 1; i < KS; ++i) {
        const uint32_t dst = (rank + uint32_t(i)) % KS;
        const uint32_t slot = rank < dst ? rank : rank - 1;
        const uint32_t base = map_to_cta(smem_u32(xbuf), dst), bar = map_to_cta(smem_u32(xbar), dst);
#pragma unroll
        for (int s = 0; s < CWARP / CH; ++s) {
          uint32_t v[CH];
          __syncwarp();
          gs_tmem_ld<CH>(tacc + dst * CO + uint32_t(half * CWARP + s * CH), v);
          tmem_wait_ld();
#pragma unroll
          for (int u = 0; u < CH / 4; ++u) {
            const uint32_t unit = (slot * (CO / 4) + uint32_t((half * CWARP + s * CH) / 4 + u)) * 128 + uint32_t(row);
            st_async_v4(base + unit * 16, bar, v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
          }
        }
      }
      ok = mbar_wait_cluster_warp(xbar, 0, abort_flag);
    }
    if (ok) {
      const int elem = p.out_dtype == ZEN_DT_S8 ? 1 : p.out_dtype == ZEN_DT_F16 ? 2 : 4;
      const bool vec_ok = (reinterpret_cast<uintptr_t>(p.out) % 16 == 0) && ((p.ldo * elem) % 16 == 0);
#pragma unroll
      for (int s = 0; s < CWARP / CH; ++s) {
        uint32_t a[CH];
        __syncwarp();
        gs_tmem_ld<CH>(tacc + uint32_t(c0 + s * CH), a);
        tmem_wait_ld();
#pragma unroll
        for (int src = 0; src < KS - 1; ++src)
#pragma unroll
          for (int u = 0; u < CH / 4; ++u) {
            const uint4 v = reinterpret_cast<const uint4*>(xbuf)[(src * (CO / 4) + (half * CWARP + s * CH) / 4 + u) * 128 + row];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              a[4 * u + e] = KIND == KIND_I8 ? a[4 * u + e] + w[e] : __float_as_uint(__uint_as_float(a[4 * u + e]) + __uint_as_float(w[e]));
          }
        const int o = s * CH;
        const int col0 = n0 + c0 + o;
        if (p.act == ZEN_ACT_GELU)
          gs_epilogue<KIND, ZEN_ACT_GELU, CH>(a, s_scale + o, s_bias + o, s_fold + o, risk_thr, inv_scale, p, m0 + row, col0, vec_ok);
        else if (p.act == ZEN_ACT_RELU)
          gs_epilogue<KIND, ZEN_ACT_RELU, CH>(a, s_scale + o, s_bias + o, s_fold + o, risk_thr, inv_scale, p, m0 + row, col0, vec_ok);
        else
          gs_epilogue<KIND, ZEN_ACT_NONE, CH>(a, s_scale + o, s_bias + o, s_fold + o, risk_thr, inv_scale, p, m0 + row, col0, vec_ok);
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  // No rendezvous: a CTA has waited for everything its peers write here, unless a wait has run out.  (A pass of 24 tokens, 48 of
  // these products: 292.8 us without the check, 293.1 with it, 302 with an arrival before the exchange and a wait here.)
  if (warp == 1) {
    tmem_dealloc(tmem, BN);
    cluster_leave(abort_flag);
  }
}

}  // namespace zen
