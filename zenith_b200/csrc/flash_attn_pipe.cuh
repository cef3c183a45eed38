// Flash-attention forward for sequences longer than one key block: GROUPS tiles of 128 queries per CTA.
//
//   warp 0      : TMA producer — the Q tiles once, then K and V tiles of 128 keys (ring of KV_STAGES)
//   warps 1 ..  : tcgen05.mma issuers, one warp per query tile (warp 1 also owns TMEM)
//   the others  : one softmax group of four warps per query tile, one thread per row (GROUPS == 2: from warp 4 on, two
//                 warpgroups that take over the registers the first does not need)
//
// What bounds it is the softmax: at head size 64 a 128 x 128 tile is 656 clocks of tensor work, 1024 of the special-function
// unit (16 exponentials per clock) and, written carelessly, 1000 issue slots per scheduler.  So:
//  * a thread takes its whole row of S (128 values) into registers in one trip through tensor memory;
//  * blocks that are valid for all 32 rows of a warp run without any per-element test (the causal diagonal and the end of
//    the keys take the masked form); maxima are taken three at a time, scaling and sums on fp32 pairs.  (A quarter to
//    half of the exponentials as a polynomial on the FMA pipe lost 2 - 10 %: the special-function unit is 60 % busy);
//  * P goes back to tensor memory (packed fp16 pairs) and P V reads its A operand there: no shared-memory round trip, and at
//    head size 64 the product is no longer bound by shared-memory reads (32 instead of 50 clocks per instruction).
//  * every tile has its own issuing warp: its events come in a fixed order, so it blocks on one barrier at a time.  One thread
//    polling both tiles' barriers issued P V 500 clocks after P was ready and took issue slots from the softmax.
// Q K^T of the next block runs under the softmax of this one.  At head size 64 every tile has S columns of its own; at 128
// tensor memory holds O and P of both tiles and one set of S columns, which they fill and empty in turn (a tile's S waits
// there until its softmax is through with the block before; P in the S columns instead left 1200 of 3500 clocks per block
// to the round trip P ready -> P V -> Q K^T).
//
// GROUPS == 2 shares K and V between 256 queries (long sequences: operand traffic).  GROUPS == 1 runs two CTAs per SM
// instead (head size 64): set-up, tile loads and output of one hide behind the other, and a short sequence does not leave
// half of a CTA idle.
//
// O accumulates in TMEM across key blocks; the maximum used for scaling is only moved, and O rescaled in TMEM by
// tcgen05.ld / st, when the row maximum has grown by more than 2^8 since the last move.
#pragma once
#include "zen_common.cuh"

namespace zen {

template <int GROUPS>
__host__ __device__ constexpr int fap_lead_warps() { return GROUPS == 2 ? 4 : 2; }
// (fp32 operands: four warps more)
template <int GROUPS, bool F32 = false>
__host__ __device__ constexpr int fap_threads() { return 32 * fap_lead_warps<GROUPS>() + 128 * GROUPS + (F32 ? 128 : 0); }

template <int D, int GROUPS, int KV_STAGES>
__host__ __device__ constexpr size_t fap_smem_bytes() {
  // Q tiles (the outputs are staged there at the end) + KV_STAGES x (K + V) tiles (128 x D fp16 each) + control + slack
  return size_t(GROUPS + 2 * KV_STAGES) * 128 * D * 2 + 256 + 1024;
}

// D[tmem] (+)= A[tmem] * B[smem desc]: A is 128 lanes x 16 fp16, two to a 32-bit column
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Scores of 32 keys of which only those below `lim` (of the same 32) are this row's: the others become -inf, neither a maximum
// nor any probability.
__device__ __forceinline__ void mask_scores(uint32_t* v, int lim) {
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (i >= lim) v[i] = 0xff800000u;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// The query tile of a CTA.  Causal tiles start from the end of their sequence: the heaviest first.
__device__ __forceinline__ void fa_tile(const FaParams& p, int q_tiles, int& b, int& h, int& qt) {
  int idx = int(blockIdx.x);
  if (p.order == FA_ORDER_HEADS_BATCHES) {
    h = idx % p.H;
    idx /= p.H;
    b = idx % p.B;
    qt = idx / p.B;
  } else if (p.order == FA_ORDER_HEADS_TILES) {
    h = idx % p.H;
    idx /= p.H;
    qt = idx % q_tiles;
    b = idx / q_tiles;
  } else {
    qt = idx % q_tiles;
    idx /= q_tiles;
    h = idx % p.H;
    b = idx / p.H;
  }
  if (p.causal) qt = q_tiles - 1 - qt;
}

// The sequence of a tile: its keys and query rows, and where the tensor maps find them.
// Unpadded batches: the sequences lie back to back in one [rows, ...] tensor, sequence b in rows cu_seqlens[b] ..
// cu_seqlens[b + 1] - 1 (cut at the tensor's rows).  A tile then starts at the sequence's first row and may run on
// into the next sequence's rows: as keys they lie beyond the key length and are masked like padding, as queries
// their rows are not stored.  The tensor maps see one batch of `rows` tokens.
struct FaSequence {
  int kv_len;    // keys
  int q_len;     // query rows
  int row_base;  // first row in the packed tensors
  int tma_b;     // batch coordinate
};
__device__ __forceinline__ FaSequence fa_sequence(const FaParams& p, int b) {
  FaSequence s{p.kv_lens ? p.kv_lens[b] : p.S, p.S, 0, b};
  if (p.cu_seqlens != nullptr) {
    const int lo = p.cu_seqlens[b], hi = p.cu_seqlens[b + 1];
    s.kv_len = lo < 0 ? 0 : (hi < p.rows ? hi : p.rows) - lo;
    s.row_base = lo < 0 ? 0 : lo;
    s.tma_b = 0;
  }
  s.kv_len = s.kv_len < 0 ? 0 : (s.kv_len > p.S ? p.S : s.kv_len);
  if (p.cu_seqlens != nullptr) s.q_len = s.kv_len;
  return s;
}

// The warp's rows of O scaled by each thread's alpha (16 columns at a time: the row of S occupies most of a thread's registers).
// The stores are not waited for.
template <int D>
__device__ __forceinline__ void fa_rescale(uint32_t tmem_o, float alpha) {
#pragma unroll 1
  for (int c = 0; c < D; c += 16) {
    uint32_t ov[16];
    __syncwarp();
    tmem_ld_32x16(tmem_o + c, ov);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
    tmem_st_32x16(tmem_o + c, ov);
  }
}

// Output of one warp's 32 query rows (first row `qr0` of the sequence): O / l into the warp's part of the dead Q tile
// (`stage`, + dc * 16 KB per 64 columns: 32 rows x 128 bytes, 16-byte units swizzled), then to global memory as whole
// 128-byte lines, eight lanes per row piece, with the int8 copy beside it.  Only rows below q_len are stored.
template <int D>
__device__ __forceinline__ void fa_write_output(const FaParams& p, uint8_t* stage, uint32_t tmem_o, bool any, float l_run, int lane, int qr0,
                                                int q_len, int b, int h, int row_base) {
  constexpr int DC = D / 64;
  constexpr int CHUNK_BYTES = 128 * 128;
  const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
#pragma unroll 1
  for (int c = 0; c < D / 32; ++c) {
    uint32_t ov[32];
    __syncwarp();
    if (any) {
      tmem_ld_32x32(tmem_o + c * 32, ov);
      tmem_wait_ld();
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) ov[i] = 0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __half2 hh = __floats2half2_rn(__uint_as_float(ov[8 * u + 2 * i]) * inv, __uint_as_float(ov[8 * u + 2 * i + 1]) * inv);
        w[i] = *reinterpret_cast<const uint32_t*>(&hh);
      }
      *reinterpret_cast<uint4*>(stage + (c >> 1) * CHUNK_BYTES + lane * 128 + ((((c & 1) * 4 + u) ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  __syncwarp();
  const int64_t base = p.cu_seqlens != nullptr ? int64_t(h) * p.o_sh + int64_t(row_base) * p.o_ss : int64_t(b) * p.o_sb + int64_t(h) * p.o_sh;
  const int u = lane & 7;
  if (!p.o_f32 && p.oq == nullptr) {
    // eight pieces in flight (48 x 12 x 256 x 64: 29.6 -> 28.3 us)
#pragma unroll 1
    for (int dc = 0; dc < DC; ++dc) {
      uint4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int rr = k * 4 + (lane >> 3);
        v[k] = *reinterpret_cast<const uint4*>(stage + dc * CHUNK_BYTES + rr * 128 + ((u ^ (rr & 7)) << 4));
      }
      __half* at = static_cast<__half*>(p.o) + base + int64_t(qr0 + (lane >> 3)) * p.o_ss + dc * 64 + u * 8;
#pragma unroll
      for (int k = 0; k < 8; ++k, at += 4 * p.o_ss)
        if (qr0 + k * 4 + (lane >> 3) < q_len) *reinterpret_cast<uint4*>(at) = v[k];
    }
    return;
  }
#pragma unroll 1
  for (int k = 0; k < 8 * DC; ++k) {
    const int dc = k >> 3, rr = (k & 7) * 4 + (lane >> 3);
    const int qr = qr0 + rr;
    if (qr >= q_len) continue;
    const uint4 v = *reinterpret_cast<const uint4*>(stage + dc * CHUNK_BYTES + rr * 128 + ((u ^ (rr & 7)) << 4));
    const int64_t off = base + int64_t(qr) * p.o_ss + dc * 64 + u * 8;
    if (p.o_f32) {
      const __half2* hp = reinterpret_cast<const __half2*>(&v);
      const float2 a0 = __half22float2(hp[0]), a1 = __half22float2(hp[1]), a2 = __half22float2(hp[2]), a3 = __half22float2(hp[3]);
      float4* of = reinterpret_cast<float4*>(static_cast<float*>(p.o) + off);
      of[0] = make_float4(a0.x, a0.y, a1.x, a1.y);
      of[1] = make_float4(a2.x, a2.y, a3.x, a3.y);
      continue;
    }
    *reinterpret_cast<uint4*>(static_cast<__half*>(p.o) + off) = v;
    if (p.oq) {
      // the int8 copy quantizes the fp16 values that were stored (branch-free rounding, exact division only next to a
      // rounding boundary)
      const __half2* hp = reinterpret_cast<const __half2*>(&v);
      float2 val[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) val[e] = __half22float2(hp[e]);
      uint32_t qw[2];
      const uint32_t risky = quantize_pairs_rn<8>(val, p.inv_o_scale, qw);
      if (risky) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (risky & (1u << e))
            patch_q_byte(qw, e, exact_q8((e & 1) ? val[e >> 1].y : val[e >> 1].x, p.o_scale, 0));
      }
      *reinterpret_cast<uint2*>(p.oq + off) = make_uint2(qw[0], qw[1]);
    }
  }
}

// `rows` rows of an operand tile from fp32 rows at `src` (stride D), as 128 threads (`t`) convert them into the layout that a
// swizzled tensor load leaves: 64 columns x 128 bytes a row, 16-byte units XORed with the row.  Rows from `valid` on are zero.
template <int D>
__device__ __forceinline__ void fa_convert_tile(uint8_t* tile, const float* src, int valid, int rows, int t) {
  const int u = t & 7, r = t >> 3;
  uint8_t* to = tile + r * 128 + ((u ^ (r & 7)) << 4);
#pragma unroll 1
  for (int dc = 0; dc < D / 64; ++dc, to += 128 * 128) {
    const float* at = src + int64_t(r) * D + dc * 64 + u * 8;
    float4 v[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i][0] = v[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r + 16 * i < valid) {
        v[i][0] = *reinterpret_cast<const float4*>(at + i * 16 * D);
        v[i][1] = *reinterpret_cast<const float4*>(at + i * 16 * D + 4);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (16 * i >= rows) break;
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const __half2 lo = __floats2half2_rn(v[i][e].x, v[i][e].y), hi = __floats2half2_rn(v[i][e].z, v[i][e].w);
        w[2 * e] = *reinterpret_cast<const uint32_t*>(&lo);
        w[2 * e + 1] = *reinterpret_cast<const uint32_t*>(&hi);
      }
      *reinterpret_cast<uint4*>(to + i * 16 * 128) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}
// The warp's part of a tile is in shared memory, where the tensor core reads it: one arrival for the warp.
__device__ __forceinline__ void fa_tile_ready(uint64_t* bar, int lane) {
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// F32: fp32 operands ([B, H, S, D], 16-byte aligned, one tile per CTA), converted on their way in: Q by the softmax warps, which
// wait for S, K and V by four warps of their own.  The same arithmetic as on converted operands, hence the same bits.
template <int D, int GROUPS, int KV_STAGES, bool F32 = false>
__global__ void __launch_bounds__(fap_threads<GROUPS, F32>(), GROUPS == 1 && !F32 ? 2 : 1)
flash_attn_pipe_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, const FaParams p) {
  constexpr int DC = D / 64;
  constexpr int TILE_BYTES = 128 * D * 2;
  constexpr int CHUNK_BYTES = 128 * 128;
  constexpr bool S_SHARED = D == 128 && GROUPS == 2;  // one set of S columns for both tiles
  constexpr uint32_t P_OFF = S_SHARED ? 128 : GROUPS * 128;  // + g * 64
  constexpr uint32_t O_OFF = P_OFF + GROUPS * 64;            // + g * D
  constexpr uint32_t TMEM_COLS = O_OFF + GROUPS * D > 256 ? 512 : 256;
  static_assert(!F32 || GROUPS == 1, "one tile");
  constexpr int LOAD_WARP = fap_lead_warps<GROUPS>() + 4 * GROUPS;  // the first of the converting warps
  constexpr uint32_t TILE_ARRIVALS = F32 ? 4 : 1;
  static_assert(O_OFF + GROUPS * D <= TMEM_COLS, "tensor memory");
  constexpr uint32_t IDESC_QK = make_idesc(IDESC_C_F32, IDESC_F16, IDESC_F16, 0, 0, 128, 128);
  constexpr uint32_t IDESC_PV = make_idesc(IDESC_C_F32, IDESC_F16, IDESC_F16, 0, 1, 128, D);
  constexpr float RESCALE_THRESHOLD = 8.0f;  // log2 units

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem;                              // [GROUPS][TILE]
  uint8_t* sK = sQ + GROUPS * TILE_BYTES;          // [KV_STAGES][TILE]
  uint8_t* sV = sK + KV_STAGES * TILE_BYTES;       // [KV_STAGES][TILE]
  uint8_t* ctrl = sV + KV_STAGES * TILE_BYTES;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(ctrl);
  uint64_t* k_full = q_full + 1;                   // [KV_STAGES]
  uint64_t* k_empty = k_full + KV_STAGES;
  uint64_t* v_full = k_empty + KV_STAGES;
  uint64_t* v_empty = v_full + KV_STAGES;
  uint64_t* s_full = v_empty + KV_STAGES;          // [GROUPS]
  uint64_t* p_full = s_full + GROUPS;              // [GROUPS]
  uint64_t* o_full = p_full + GROUPS;              // [GROUPS]
  uint64_t* s_free = o_full + GROUPS;              // [GROUPS] the group has taken S into registers
  uint64_t* p_half = s_free + GROUPS;              // [GROUPS] the first 64 keys of P are in tensor memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(p_half + GROUPS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  int b, h, qt;
  fa_tile(p, (p.S + 128 * GROUPS - 1) / (128 * GROUPS), b, h, qt);
  const int q0 = qt * (128 * GROUPS);

  if (threadIdx.x == 0) {
    if constexpr (!F32) {
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_v);
    }
    mbar_init(q_full, TILE_ARRIVALS);
    for (int i = 0; i < KV_STAGES; ++i) {
      mbar_init(&k_full[i], TILE_ARRIVALS);
      mbar_init(&k_empty[i], GROUPS);
      mbar_init(&v_full[i], TILE_ARRIVALS);
      mbar_init(&v_empty[i], GROUPS);
    }
    for (int g = 0; g < GROUPS; ++g) {
      mbar_init(&s_full[g], 1);
      mbar_init(&p_full[g], 128);
      mbar_init(&o_full[g], 1);
      mbar_init(&s_free[g], 128);
      mbar_init(&p_half[g], 128);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_wait();  // Q, K, V, the key lengths and the output buffers may belong to the previous kernel until here
  grid_launch_dependents();
  const FaSequence seq = fa_sequence(p, b);
  const int kv_len = seq.kv_len, q_len = seq.q_len, row_base = seq.row_base, tma_b = seq.tma_b;
  // key blocks needed by each group (a group has none if the sequence ends before its tile)
  int nblk[GROUPS];
  int n_blocks = 0;
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    int end = kv_len;
    if (p.causal && q0 + g * 128 + 128 < end) end = q0 + g * 128 + 128;
    nblk[g] = (q0 + g * 128 < q_len) ? (end + 127) / 128 : 0;
    n_blocks = nblk[g] > n_blocks ? nblk[g] : n_blocks;
  }

  if constexpr (GROUPS == 2) {
    // 384 threads start with 168 registers; a softmax thread holds a row of 128 values and more
    if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
  }
  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (!F32 && n_blocks > 0 && elect_one()) {
      bool ok = true;
      mbar_arrive_expect_tx(q_full, GROUPS * TILE_BYTES);
#pragma unroll
      for (int g = 0; g < GROUPS; ++g)
#pragma unroll
        for (int dc = 0; dc < DC; ++dc)
          fa_tma_tile(sQ + g * TILE_BYTES + dc * CHUNK_BYTES, &tmap_q, q_full, p.q_perm, dc * 64, row_base + q0 + g * 128, h, tma_b);
      int st = 0;
      uint32_t ph = 1;
      for (int j = 0; j < n_blocks && ok; ++j) {
        if (!mbar_wait(&k_empty[st], ph, abort_flag)) { ok = false; break; }
        mbar_arrive_expect_tx(&k_full[st], TILE_BYTES);
#pragma unroll
        for (int dc = 0; dc < DC; ++dc)
          fa_tma_tile(sK + st * TILE_BYTES + dc * CHUNK_BYTES, &tmap_k, &k_full[st], p.k_perm, dc * 64, row_base + j * 128, h, tma_b);
        if (!mbar_wait(&v_empty[st], ph, abort_flag)) { ok = false; break; }
        mbar_arrive_expect_tx(&v_full[st], TILE_BYTES);
#pragma unroll
        for (int dc = 0; dc < DC; ++dc)
          fa_tma_tile(sV + st * TILE_BYTES + dc * CHUNK_BYTES, &tmap_v, &v_full[st], p.v_perm, dc * 64, row_base + j * 128, h, tma_b);
        if (++st == KV_STAGES) {
          st = 0;
          ph ^= 1u;
        }
      }
      if (!ok) {
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
      }
    }
  } else if (warp < fap_lead_warps<GROUPS>()) {
    // ---------------------------------------------------------------- MMA issuer of one query tile
    if (n_blocks > 0 && warp <= GROUPS && elect_one()) {
      const int g = warp - 1;
      int nb = 0;
#pragma unroll
      for (int i = 0; i < GROUPS; ++i) nb = i == g ? nblk[i] : nb;
      const uint32_t qa = smem_u32(sQ + g * TILE_BYTES);
      const uint32_t ts = tmem_base + (S_SHARED ? 0u : uint32_t(g * 128));
      const uint32_t tp = tmem_base + P_OFF + uint32_t(g * 64);
      const uint32_t to = tmem_base + O_OFF + uint32_t(g * D);
      const uint32_t idesc_qk = IDESC_QK | p.qk_negate;
      auto issue_qk = [&](int st) {
        const uint32_t ka = smem_u32(sK + st * TILE_BYTES);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t off = (ks / 4) * CHUNK_BYTES + (ks % 4) * 32;
          mma_f16_ss(ts, make_smem_desc_sw128(qa + off, 1024, 16), make_smem_desc_sw128(ka + off, 1024, 16), idesc_qk, ks != 0 ? 1u : 0u);
        }
        tc_commit(&s_full[g]);
        tc_commit(&k_empty[st]);  // this tile has used the K tile
      };
      auto issue_pv = [&](int st, int ks0, int ks1, bool first) {
        const uint32_t va = smem_u32(sV + st * TILE_BYTES);
#pragma unroll
        for (int ks = ks0; ks < ks1; ++ks)
          mma_f16_ts(to, tp + uint32_t(ks * 8), make_smem_desc_sw128(va + ks * (16 * 128), 1024, CHUNK_BYTES), IDESC_PV, first && ks == 0 ? 0u : 1u);
      };
      bool ok = mbar_wait(q_full, 0, abort_flag);
      // K tiles run one block ahead of V tiles
      int kst = 0, vst = 0;
      uint32_t kph = 0, vph = 0;
      auto next_k = [&](bool use) {
        if (ok) ok = mbar_wait(&k_full[kst], kph, abort_flag);
        if (ok) {
          tc_fence_after_sync();
          if (use) issue_qk(kst);
          else mbar_arrive(&k_empty[kst]);  // a block that only the other tile needs
        }
        if (++kst == KV_STAGES) {
          kst = 0;
          kph ^= 1u;
        }
      };
      // S columns free for Q K^T of block j: the S before it has been taken into registers
      auto s_columns_free = [&](int j) -> bool {
        if constexpr (S_SHARED) {
          // the tiles take turns, tile 0 first; where only one has a block left it follows itself
          const int other = nblk[g ^ 1];
          const int turn = g == 0 ? j - 1 : j;  // the other tile's block before this one
          if (turn >= 0 && turn < other) return mbar_wait(&s_free[g ^ 1], turn & 1, abort_flag);
        }
        return j == 0 || mbar_wait(&s_free[g], (j - 1) & 1, abort_flag);
      };
      if (nb > 0) ok = ok && s_columns_free(0);
      next_k(nb > 0);
      for (int j = 0; j < n_blocks && ok; ++j) {
        if (j + 1 < n_blocks) {
          // Q K^T of the next block runs under this block's softmax
          if (j + 1 < nb) ok = s_columns_free(j + 1);
          next_k(j + 1 < nb);
        }
        if (j < nb) {
          // the first half of P, then all of it, is in tensor memory; O has been rescaled if it had to be
          if (ok) ok = mbar_wait(&v_full[vst], vph, abort_flag) && mbar_wait(&p_half[g], j & 1, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          issue_pv(vst, 0, 4, j == 0);
          ok = mbar_wait(&p_full[g], j & 1, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          issue_pv(vst, 4, 8, false);
          tc_commit(&o_full[g]);
          tc_commit(&v_empty[vst]);
        } else {
          if (ok) ok = mbar_wait(&v_full[vst], vph, abort_flag);
          if (!ok) break;
          mbar_arrive(&v_empty[vst]);
        }
        if (++vst == KV_STAGES) {
          vst = 0;
          vph ^= 1u;
        }
      }
    }
  } else if (F32 && warp >= LOAD_WARP) {
    // ---------------------------------------------------------------- K and V tiles of fp32 operands
    const int t = int(threadIdx.x) - LOAD_WARP * 32;
    const int64_t base = (int64_t(b) * p.H + h) * p.S * D;
    int st = 0;
    uint32_t ph = 1;
    for (int j = 0; j < n_blocks; ++j) {
      const int64_t at = base + int64_t(j) * 128 * D;
      if (!mbar_wait_warp(&k_empty[st], ph, abort_flag)) break;
      fa_convert_tile<D>(sK + st * TILE_BYTES, p.k32 + at, p.S - j * 128, 128, t);
      fa_tile_ready(&k_full[st], lane);
      if (!mbar_wait_warp(&v_empty[st], ph, abort_flag)) break;
      fa_convert_tile<D>(sV + st * TILE_BYTES, p.v32 + at, p.S - j * 128, 128, t);
      fa_tile_ready(&v_full[st], lane);
      if (++st == KV_STAGES) {
        st = 0;
        ph ^= 1u;
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax groups
    const int g = (warp - fap_lead_warps<GROUPS>()) >> 2;
    if (F32 && n_blocks > 0) {
      fa_convert_tile<D>(sQ, p.q32 + ((int64_t(b) * p.H + h) * p.S + q0) * D, p.S - q0, 128, (warp - fap_lead_warps<GROUPS>()) * 32 + lane);
      fa_tile_ready(q_full, lane);
    }
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const int q = q0 + g * 128 + r;
    const uint32_t lane_sel = uint32_t(quad * 32) << 16;
    const uint32_t tmem_s = tmem_base + (S_SHARED ? 0u : uint32_t(g * 128)) + lane_sel;
    const uint32_t tmem_p = tmem_base + P_OFF + uint32_t(g * 64) + lane_sel;
    const uint32_t tmem_o = tmem_base + O_OFF + uint32_t(g * D) + lane_sel;
    int nb = 0;
#pragma unroll
    for (int i = 0; i < GROUPS; ++i) nb = i == g ? nblk[i] : nb;
    // blocks below this one are valid for every row of the warp: no per-element tests
    int n_plain = kv_len / 128;
    if (p.causal) n_plain = min(n_plain, (q0 + g * 128 + quad * 32 + 1) / 128);
    float m_ref = -INFINITY;  // the maximum the stored probabilities and O are scaled with (log2 units)
    float l_run = 0.f;
    bool ok = true;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);

    for (int j = 0; j < nb; ++j) {
      if (!mbar_wait_warp(&s_full[g], j & 1, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      uint32_t sv[4][32];
      __syncwarp();
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(tmem_s + c * 32, sv[c]);
      tmem_wait_ld();
      tc_fence_before_sync();
      mbar_arrive(&s_free[g]);
      if (j >= n_plain) {
        // (only 32 keys at a time in which a row of the warp has an end: a block with padding is mostly plain)
        int lim = kv_len - j * 128, lim_warp = lim;
        if (p.causal) {
          lim = min(lim, q + 1 - j * 128);
          lim_warp = min(lim_warp, q - lane + 1 - j * 128);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (lim_warp < 32 * (c + 1)) mask_scores(sv[c], lim - 32 * c);
      }
      auto s_at = [&](int i) { return __uint_as_float(sv[i >> 5][i & 31]); };
      float mx4[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        mx4[u] = max3(s_at(u), s_at(4 + u), s_at(8 + u));
#pragma unroll
        for (int i = 12; i + 8 <= 128; i += 8) mx4[u] = max3(mx4[u], s_at(i + u), s_at(i + 4 + u));
        mx4[u] = fmaxf(mx4[u], s_at(124 + u));
      }
      const float m_blk = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]) * p.scale_log2;
      // move the reference maximum only when this row has outgrown it by more than the threshold
      const bool grow = m_blk > m_ref + RESCALE_THRESHOLD || (m_ref == -INFINITY && m_blk != -INFINITY);
      const float m_new = grow ? m_blk : m_ref;
      const float alpha = (grow && m_ref != -INFINITY) ? fast_exp2(m_ref - m_new) : 1.0f;
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      m_ref = m_new;
      const bool rescale = j > 0 && __any_sync(0xffffffffu, alpha != 1.0f);
      // P V of the previous block has completed: P may be overwritten, O may be rescaled
      if (j > 0) {
        if (!mbar_wait_warp(&o_full[g], (j - 1) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
      }
      if (rescale) {
        fa_rescale<D>(tmem_o, alpha);
        tmem_wait_st();
        l_run *= alpha;
      }
      // probabilities -> tensor memory (fp16 pairs), row sum
      const float2 nm2 = make_float2(-m_use, -m_use);
      float2 rs[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {  // column pair 32 hc + i
          const float2 x = f2fma(make_float2(s_at(hc * 64 + 2 * i), s_at(hc * 64 + 2 * i + 1)), sc2, nm2);
          const float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
          rs[i & 1] = f2add(rs[i & 1], e);
          const __half2 hh = __floats2half2_rn(e.x, e.y);
          pk[i] = *reinterpret_cast<const uint32_t*>(&hh);
        }
        __syncwarp();
        tmem_st_32x32(tmem_p + hc * 32, pk);
        if (hc == 0) {
          tmem_wait_st();
          tc_fence_before_sync();
          mbar_arrive(&p_half[g]);
        }
      }
      l_run += (rs[0].x + rs[0].y) + (rs[1].x + rs[1].y);
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(&p_full[g]);
    }

    if (ok && nb > 0) {
      ok = mbar_wait_warp(&o_full[g], (nb - 1) & 1, abort_flag);
      tc_fence_after_sync();
    }
    if (ok) {
      // the Q tile has been read for the last time by Q K^T of the last block
      fa_write_output<D>(p, sQ + g * TILE_BYTES + quad * 4096, tmem_o, nb > 0, l_run, lane, q0 + g * 128 + quad * 32, q_len, b, h, row_base);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

}  // namespace zen
