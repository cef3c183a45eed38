// Flash-attention forward at head size 64 with the bits of flash_attn_pipe_kernel: one tile of 128 queries per CTA, key blocks
// of 128 taken in halves, three CTAs per SM.
//
//   warp 0    : one thread issues the loads and the tensor-core instructions
//   warps 1-4 : softmax, one thread per query row
//
// What bounds it is the chain of a key block, as in flash_attn_quad_kernel, and the ends of a tile.  For the same bits the
// maximum that scales a probability is that of all 128 keys, and row sums add in the same order.  Two CTAs an SM is what a row
// of 128 scores in registers allows (flash_attn_pipe_kernel); here a thread holds the first 64, passes over the second half
// for its maximum, packs the first half's probabilities and reads the second half again: 124 registers.  P (64 columns) lies
// over S (64), so that a CTA takes 128 columns of tensor memory, and 64 KB of shared memory, with one V tile.
// Measured with int8 copy and key lengths against flash_attn_pipe_kernel in a stream of passes: 48 x 12 x 256 33.2 -> 29.5 us,
// 32 x 16 x 384 53.5 -> 49.3 (causal 48.1 -> 40.9), 40 x 12 x 160 28.9 -> 26.0.
//
// The events of a tile form one cycle: S of the first half complete (with it P V of the block before, hence the V tile is
// free), taken into registers, S of the second half complete, P complete (with it S read, hence the K tile is free).
#pragma once
#include "flash_attn_pipe.cuh"

namespace zen {

constexpr int FAT_THREADS = 160;
constexpr int FAT_KEYS = 128;
constexpr int FAT_CTAS = 3;  // per SM
__host__ __device__ constexpr size_t fat_smem_bytes() {
  // Q tile (the output is staged there at the end) + 2 K tiles + V tile + control + slack
  return size_t(128 + 3 * FAT_KEYS) * 128 + 128 + 1024;
}

__global__ void __launch_bounds__(FAT_THREADS, FAT_CTAS)
flash_attn_tri_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, const FaParams p) {
  constexpr int Q_BYTES = 128 * 128;
  constexpr int KV_BYTES = FAT_KEYS * 128;
  constexpr uint32_t O_OFF = 64;  // S, then P, in columns 0 .. 63
  constexpr uint32_t TMEM_COLS = 128;
  constexpr uint32_t IDESC_QK = make_idesc(IDESC_C_F32, IDESC_F16, IDESC_F16, 0, 0, 128, 64);
  constexpr uint32_t IDESC_PV = make_idesc(IDESC_C_F32, IDESC_F16, IDESC_F16, 0, 1, 128, 64);
  constexpr float RESCALE_THRESHOLD = 8.0f;  // log2 units

  extern __shared__ uint8_t smem_raw[];
  uint8_t* sQ = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sK = sQ + Q_BYTES;       // [2]
  uint8_t* sV = sK + 2 * KV_BYTES;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(sV + KV_BYTES);
  uint64_t* k_full = q_full + 1;  // [2]
  uint64_t* v_full = k_full + 2;
  uint64_t* s_full = v_full + 1;  // twice a block: keys 0 .. 63, 64 .. 127
  uint64_t* p_full = s_full + 1;
  uint64_t* o_full = p_full + 1;
  uint64_t* s_free = o_full + 1;  // the first half of S has been taken into registers
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_free + 1);
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
      mbar_init(&k_full[0], 1);
      mbar_init(&k_full[1], 1);
      mbar_init(v_full, 1);
      mbar_init(s_free, 4);
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
  const int nb = q0 < q_len ? (key_end + FAT_KEYS - 1) / FAT_KEYS : 0;

  if (warp == 0) {
    // ---------------------------------------------------------------- loads and tensor-core instructions
    if (nb > 0 && elect_one()) {
      auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, const int (&perm)[3], int row, uint32_t bytes) {
        mbar_arrive_expect_tx(bar, bytes);
        fa_tma_tile(dst, map, bar, perm, 0, row_base + row, h, tma_b);
      };
      auto load_k = [&](int j) { load(sK + (j & 1) * KV_BYTES, &tmap_k, &k_full[j & 1], p.k_perm, j * FAT_KEYS, KV_BYTES); };
      auto load_v = [&](int j) { load(sV, &tmap_v, v_full, p.v_perm, j * FAT_KEYS, KV_BYTES); };
      const uint32_t qa = smem_u32(sQ), va = smem_u32(sV), idesc_qk = IDESC_QK | p.qk_negate;
      auto issue_qk = [&](int j, uint32_t half) {
        const uint32_t ka = smem_u32(sK) + uint32_t(j & 1) * KV_BYTES + half * (64 * 128);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          mma_f16_ss(tmem_base, make_smem_desc_sw128(qa + ks * 32, 1024, 16), make_smem_desc_sw128(ka + ks * 32, 1024, 16), idesc_qk, ks != 0 ? 1u : 0u);
        tc_commit(s_full);
      };
      load(sQ, &tmap_q, q_full, p.q_perm, q0, Q_BYTES);
      load_k(0);
      load_v(0);
      if (nb > 1) load_k(1);
      bool ok = mbar_wait(q_full, 0, abort_flag) && mbar_wait(&k_full[0], 0, abort_flag);
      tc_fence_after_sync();
      if (ok) issue_qk(0, 0);
      for (int j = 0; j < nb && ok; ++j) {
        ok = mbar_wait(s_free, j & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        issue_qk(j, 1);
        if (j > 0) load_v(j);  // (P V of the block before completed before S did)
        ok = mbar_wait(v_full, j & 1, abort_flag) && mbar_wait(p_full, j & 1, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < FAT_KEYS / 16; ++ks)
          mma_f16_ts(tmem_base + O_OFF, tmem_base + uint32_t(ks * 8), make_smem_desc_sw128(va + ks * (16 * 128), 1024, Q_BYTES), IDESC_PV, j == 0 && ks == 0 ? 0u : 1u);
        if (j + 1 < nb) {
          ok = mbar_wait(&k_full[(j + 1) & 1], uint32_t((j + 1) >> 1) & 1u, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          issue_qk(j + 1, 0);
        } else {
          tc_commit(o_full);
        }
        if (j + 2 < nb) load_k(j + 2);
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
    float m_ref = -INFINITY;  // the maximum the stored probabilities and O are scaled with (log2 units)
    float l_run = 0.f;
    bool ok = true;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);

    for (int j = 0; j < nb; ++j) {
      // keys of the block below the end of this row, of the first row of the warp
      int lim = kv_len - j * FAT_KEYS, lim_warp = lim;
      if (p.causal) {
        lim = min(lim, qw + lane + 1 - j * FAT_KEYS);
        lim_warp = min(lim_warp, qw + 1 - j * FAT_KEYS);
      }
      auto max32 = [](const uint32_t* v) {
        auto at = [&](int i) { return __uint_as_float(v[i]); };
        float m0 = max3(at(0), at(1), at(2)), m1 = max3(at(3), at(4), at(5));
#pragma unroll
        for (int i = 6; i < 30; i += 4) {
          m0 = max3(m0, at(i), at(i + 1));
          m1 = max3(m1, at(i + 2), at(i + 3));
        }
        return fmaxf(max3(m0, at(30), at(31)), m1);
      };
      auto arrive = [&](uint64_t* bar) {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
      };
      if (!mbar_wait_warp(s_full, 0, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      uint32_t sv[64];
      tmem_ld_32x64(tmem_s, sv);
      tmem_wait_ld();
      arrive(s_free);
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (lim_warp < 32 * (c + 1)) mask_scores(sv + 32 * c, lim - 32 * c);
      float mx = fmaxf(max32(sv), max32(sv + 32));
      if (!mbar_wait_warp(s_full, 1, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t t[32];
        __syncwarp();
        tmem_ld_32x32(tmem_s + c * 32, t);
        tmem_wait_ld();
        if (lim_warp < 64 + 32 * (c + 1)) mask_scores(t, lim - 64 - 32 * c);
        mx = fmaxf(mx, max32(t));
      }
      const float m_blk = mx * p.scale_log2;
      // move the reference maximum only when this row has outgrown it by more than the threshold
      const bool grow = m_blk > m_ref + RESCALE_THRESHOLD || (m_ref == -INFINITY && m_blk != -INFINITY);
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
      uint32_t pk[2][32];
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        if (hc == 1) {
          __syncwarp();
          tmem_ld_32x64(tmem_s, sv);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 2; ++c)
            if (lim_warp < 64 + 32 * (c + 1)) mask_scores(sv + 32 * c, lim - 64 - 32 * c);
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float2 x = f2fma(make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sc2, nm2);
          const float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
          rs[i & 1] = f2add(rs[i & 1], e);
          const __half2 hh = __floats2half2_rn(e.x, e.y);
          pk[hc][i] = *reinterpret_cast<const uint32_t*>(&hh);
        }
      }
      __syncwarp();
      tmem_st_32x32(tmem_s, pk[0]);
      tmem_st_32x32(tmem_s + 32, pk[1]);
      l_run += (rs[0].x + rs[0].y) + (rs[1].x + rs[1].y);
      tmem_wait_st();
      arrive(p_full);
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
