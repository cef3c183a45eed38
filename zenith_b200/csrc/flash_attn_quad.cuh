// Flash-attention forward at head size 64 for sequences longer than one key block of flash_attn_short_kernel: one tile of 128
// queries per CTA, key blocks of 64, four CTAs per SM.
//
//   warp 0    : one thread issues the loads and the tensor-core instructions
//   warps 1-4 : softmax, one thread per query row
//
// What bounds it is the special-function unit: 64 exponentials a row and block, 512 clocks of each scheduler.  A softmax warp
// is one chain - S from tensor memory, maximum, exponentials, P to tensor memory, P V and Q K^T of the next block - of which
// the exponentials are a third, so a scheduler needs three or four such warps to keep the unit busy.  64 keys a block
// (64 values a thread instead of 128) and one issuing warp are what lets four tiles share an SM: 96 registers a thread, 48 KB
// of shared memory and 128 columns of tensor memory a CTA.  P lies over S (its thread has taken the row into registers), so
// Q K^T of block j + 1 follows P V of block j; the other three tiles work meanwhile.
//
// Measured against flash_attn_pipe_kernel in a stream of passes (short runs): 32 x 16 heads x 384 43.5 -> 39.7 us (43.8 -> 38.0),
// 48 x 12 x 256 24.7 -> 20.8, causal 23.0 -> 18.2, 40 x 12 x 160 22.7 -> 15.8, 8 x 16 x 2048 causal 118.5 -> 114.6 (110.7 -> 99.8),
// full 209 -> 210 (189 -> 186).  Slower were, where this took 37.6, 21.0 (causal 18.4) and 105.5 us: three CTAs with P in columns of its
// own, so that Q K^T runs under the softmax (39.4, 22.4 (28.8), 113 us); CTAs that take their next tile by cluster launch
// control and load ahead into it (39.8, 23.9 (26.0), 123 us: longer code per block, spilled registers).
//
// All of a tile's events form one cycle, so three kinds of barrier do: operands loaded, S complete (with it P V of the block
// before), P complete (with it S read, hence the K tile and the V tile of the block before are free).
//
// O accumulates in TMEM across key blocks; the maximum used for scaling is only moved, and O rescaled in TMEM by
// tcgen05.ld / st, when the row maximum has grown by more than 2^8 since the last move.
#pragma once
#include "flash_attn_pipe.cuh"

namespace zen {

constexpr int FAQ_THREADS = 160;
constexpr int FAQ_KEYS = 64;
constexpr int FAQ_CTAS = 4;  // per SM
__host__ __device__ constexpr size_t faq_smem_bytes() {
  // Q tile (the output is staged there at the end) + 2 x (K + V) tiles + control + slack
  return size_t(128 + 4 * FAQ_KEYS) * 128 + 128 + 1024;
}

__global__ void __launch_bounds__(FAQ_THREADS, FAQ_CTAS)
flash_attn_quad_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, const FaParams p) {
  constexpr int Q_BYTES = 128 * 128;
  constexpr int KV_BYTES = FAQ_KEYS * 128;
  constexpr uint32_t O_OFF = 64;  // S, then P, in columns 0 .. 63
  constexpr uint32_t TMEM_COLS = 128;
  constexpr uint32_t IDESC_QK = make_idesc(IDESC_C_F32, IDESC_F16, IDESC_F16, 0, 0, 128, FAQ_KEYS);
  constexpr uint32_t IDESC_PV = make_idesc(IDESC_C_F32, IDESC_F16, IDESC_F16, 0, 1, 128, 64);
  constexpr float RESCALE_THRESHOLD = 8.0f;  // log2 units

  extern __shared__ uint8_t smem_raw[];
  uint8_t* sQ = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sK = sQ + Q_BYTES;       // [2]
  uint8_t* sV = sK + 2 * KV_BYTES;  // [2]
  uint64_t* q_full = reinterpret_cast<uint64_t*>(sV + 2 * KV_BYTES);
  uint64_t* k_full = q_full + 1;  // [2]
  uint64_t* v_full = k_full + 2;  // [2]
  uint64_t* s_full = v_full + 2;
  uint64_t* p_full = s_full + 1;
  uint64_t* o_full = p_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  int b, h, qt;
  fa_tile(p, (p.S + 127) / 128, b, h, qt);
  const int q0 = qt * 128;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_v);
      mbar_init(q_full, 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(&k_full[i], 1);
        mbar_init(&v_full[i], 1);
      }
      mbar_init(s_full, 1);
      mbar_init(p_full, 4);
      mbar_init(o_full, 1);
      *abort_flag = 0;
      mbar_fence_init();
    }
    __syncwarp();
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
  const int key_end = p.causal && q0 + 128 < kv_len ? q0 + 128 : kv_len;
  const int nb = q0 < q_len ? (key_end + FAQ_KEYS - 1) / FAQ_KEYS : 0;

  if (warp == 0) {
    // ---------------------------------------------------------------- loads and tensor-core instructions
    if (nb > 0 && elect_one()) {
      auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, const int (&perm)[3], int row, uint32_t bytes) {
        mbar_arrive_expect_tx(bar, bytes);
        fa_tma_tile(dst, map, bar, perm, 0, row_base + row, h, tma_b);
      };
      auto load_k = [&](int j) { load(sK + (j & 1) * KV_BYTES, &tmap_k, &k_full[j & 1], p.k_perm, j * FAQ_KEYS, KV_BYTES); };
      auto load_v = [&](int j) { load(sV + (j & 1) * KV_BYTES, &tmap_v, &v_full[j & 1], p.v_perm, j * FAQ_KEYS, KV_BYTES); };
      const uint32_t qa = smem_u32(sQ), idesc_qk = IDESC_QK | p.qk_negate;
      auto issue_qk = [&](int j) -> bool {
        if (!mbar_wait(&k_full[j & 1], uint32_t(j >> 1) & 1u, abort_flag)) return false;
        tc_fence_after_sync();
        const uint32_t ka = smem_u32(sK) + uint32_t(j & 1) * KV_BYTES;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          mma_f16_ss(tmem_base, make_smem_desc_sw128(qa + ks * 32, 1024, 16), make_smem_desc_sw128(ka + ks * 32, 1024, 16), idesc_qk, ks != 0 ? 1u : 0u);
        tc_commit(s_full);
        return true;
      };
      load(sQ, &tmap_q, q_full, p.q_perm, q0, Q_BYTES);
      load_k(0);
      load_v(0);
      if (nb > 1) {
        load_k(1);
        load_v(1);
      }
      bool ok = mbar_wait(q_full, 0, abort_flag) && issue_qk(0);
      for (int j = 0; j < nb && ok; ++j) {
        ok = mbar_wait(&v_full[j & 1], uint32_t(j >> 1) & 1u, abort_flag) && mbar_wait(p_full, j & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t va = smem_u32(sV) + uint32_t(j & 1) * KV_BYTES;
#pragma unroll
        for (int ks = 0; ks < FAQ_KEYS / 16; ++ks)
          mma_f16_ts(tmem_base + O_OFF, tmem_base + uint32_t(ks * 8), make_smem_desc_sw128(va + ks * (16 * 128), 1024, Q_BYTES), IDESC_PV, j == 0 && ks == 0 ? 0u : 1u);
        if (j + 1 < nb) ok = issue_qk(j + 1);
        else tc_commit(o_full);
        // Q K^T of block j and P V of block j - 1 have read their tiles
        if (j + 2 < nb) load_k(j + 2);
        if (j > 0 && j + 1 < nb) load_v(j + 1);
      }
      if (!ok) {
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);  // the loads in flight end before the CTA does
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax
    const int quad = warp & 3;
    const uint32_t tmem_s = tmem_base + (uint32_t(quad * 32) << 16);
    const uint32_t tmem_o = tmem_s + O_OFF;
    const int qw = q0 + quad * 32;  // first row of the warp
    const int row_end = p.causal && qw + lane + 1 < kv_len ? qw + lane + 1 : kv_len;  // keys of this row
    const int warp_end = p.causal && qw + 32 < kv_len ? qw + 32 : kv_len;             // ... of any row of the warp
    // blocks below this one are valid for every row of the warp: no per-element tests
    const int n_plain = (p.causal && qw + 1 < kv_len ? qw + 1 : kv_len) / FAQ_KEYS;
    float m_ref = -INFINITY;  // the maximum the stored probabilities and O are scaled with (log2 units)
    float l_run = 0.f;
    bool ok = true;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);

    for (int j = 0; j < nb; ++j) {
      if (!mbar_wait_warp(s_full, j & 1, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      if (j * FAQ_KEYS < warp_end) {
        uint32_t sv[64];
        tmem_ld_32x64(tmem_s, sv);
        tmem_wait_ld();
        if (j >= n_plain) {
          const int lim = row_end - j * FAQ_KEYS, lim_warp = (p.causal ? min(qw + 1, kv_len) : kv_len) - j * FAQ_KEYS;
#pragma unroll
          for (int c = 0; c < 2; ++c)
            if (lim_warp < 32 * (c + 1)) mask_scores(sv + 32 * c, lim - 32 * c);
        }
        auto s_at = [&](int i) { return __uint_as_float(sv[i]); };
        float mx4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          mx4[u] = max3(s_at(u), s_at(4 + u), s_at(8 + u));
#pragma unroll
          for (int i = 12; i + 8 <= 64; i += 8) mx4[u] = max3(mx4[u], s_at(i + u), s_at(i + 4 + u));
          mx4[u] = fmaxf(mx4[u], s_at(60 + u));
        }
        const float m_blk = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]) * p.scale_log2;
        // Move the reference maximum only when this row has outgrown it by more than the threshold, except in the second block:
        // the largest of 128 keys is 1 exactly, as in the other kernel (else the results are 1 % further from those in 64 bits;
        // so they are 0.04 - 1.4 % nearer for normally distributed operands, and up to 7 % further where the last quarter of the
        // keys is four times as large, since a row's largest probability is then seldom in the block that moves the reference).
        const bool grow = m_blk > m_ref + (j == 1 ? 0.f : RESCALE_THRESHOLD) || (m_ref == -INFINITY && m_blk != -INFINITY);
        const float m_new = grow ? m_blk : m_ref;
        const float alpha = (grow && m_ref != -INFINITY) ? fast_exp2(m_ref - m_new) : 1.0f;
        const float m_use = m_new == -INFINITY ? 0.f : m_new;
        m_ref = m_new;
        if (j > 0 && __any_sync(0xffffffffu, alpha != 1.0f)) {
          // (P V of the previous block completed before S did)
          fa_rescale<64>(tmem_o, alpha);
          l_run *= alpha;
        }
        // probabilities -> tensor memory (fp16 pairs), row sum
        const float2 nm2 = make_float2(-m_use, -m_use);
        float2 rs[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {  // column pair 16 hc + i
            const float2 x = f2fma(make_float2(s_at(hc * 32 + 2 * i), s_at(hc * 32 + 2 * i + 1)), sc2, nm2);
            const float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
            rs[i & 1] = f2add(rs[i & 1], e);
            const __half2 hh = __floats2half2_rn(e.x, e.y);
            pk[i] = *reinterpret_cast<const uint32_t*>(&hh);
          }
          __syncwarp();
          tmem_st_32x16(tmem_s + hc * 16, pk);
        }
        l_run += (rs[0].x + rs[0].y) + (rs[1].x + rs[1].y);
      } else {
        // keys that lie behind every row of the warp (the causal diagonal)
        uint32_t zero[16] = {};
        tmem_st_32x16(tmem_s, zero);
        tmem_st_32x16(tmem_s + 16, zero);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }

    if (ok && nb > 0) {
      ok = mbar_wait_warp(o_full, 0, abort_flag);
      tc_fence_after_sync();
    }
    if (ok) {
      // the Q tile has been read for the last time by Q K^T of the last block
      fa_write_output<64>(p, sQ + quad * 4096, tmem_o, nb > 0, l_run, lane, qw, q_len, b, h, row_base);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, TMEM_COLS);
}

}  // namespace zen
