// Flash-attention forward for sequences of one key block (S <= 128): one (head, batch) item per softmax group, GROUPS
// groups per CTA, persistent CTAs.
//
//   warp 0           : TMA producer of every group's Q, K and V tile
//   warps 1 .. GROUPS: tcgen05.mma issuer of one group each (warp 1 also owns TMEM)
//   warps 4 ..       : the softmax groups, four warps each, one thread per query row
//
// What bounds it is the chain of one item - set-up and loads 1.4 us, Q K^T 0.2, softmax 0.6 (alone on its SM) to 1.6 (three
// items, the special-function unit), P V 0.3, output 0.6 - and not any unit.  So an SM works on three items at a time (two at
// head size 128); the softmax fetches a chunk of S while it works on the one before (two trips: a row of 128 values in
// registers would spill beside three groups), takes maxima three at a time, scales and sums pairs; P goes back to tensor
// memory, where P V reads it, into columns of S that have been read, O into the ones behind.  With one item per CTA, four
// CTAs per SM, unpaired arithmetic and P through shared memory an fp16 encoder of 16 x 100 tokens took 721 us, with this 714
// (703 launched early), 32 x 128: 993 -> 984, 1 x 24: 293 -> 288.
// Products and softmax stop at the 16 or 32 keys that the key length fills.
#pragma once
#include "zen_common.cuh"

namespace zen {

template <int D>
__host__ __device__ constexpr int fas_groups() { return D == 64 ? 3 : 2; }
template <int D>
__host__ __device__ constexpr int fas_threads() { return 128 + 128 * fas_groups<D>(); }
template <int D>
__host__ __device__ constexpr size_t fas_smem_bytes() { return size_t(fas_groups<D>()) * 3 * 128 * D * 2 + 256 + 1024; }

// keys at and beyond `lim` of the chunk: neither a maximum nor any probability
__device__ __forceinline__ void mask_chunk(uint32_t (&v)[32], int lim) {
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (i >= lim) v[i] = 0xff800000u;  // -inf
}

__device__ __forceinline__ float chunk_max(const uint32_t (&v)[32]) {
  auto at = [&](int i) { return __uint_as_float(v[i]); };
  float m0 = max3(at(0), at(1), at(2)), m1 = max3(at(3), at(4), at(5));
#pragma unroll
  for (int i = 6; i < 30; i += 4) {
    m0 = max3(m0, at(i), at(i + 1));
    m1 = max3(m1, at(i + 2), at(i + 3));
  }
  return fmaxf(max3(m0, at(30), at(31)), m1);
}

// F32: fp32 operands ([B, H, S, D], 16-byte aligned), which a group converts on their way in while it has nothing else to do.
// The same arithmetic as on converted operands, hence the same bits.
template <int D, bool F32 = false>
__global__ void __launch_bounds__(fas_threads<D>(), 1)
flash_attn_short_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                        const __grid_constant__ CUtensorMap tmap_v, const FaParams p) {
  constexpr int GROUPS = fas_groups<D>();
  constexpr int DC = D / 64;
  constexpr int TILE_BYTES = 128 * D * 2;
  constexpr int CHUNK_BYTES = 128 * 128;
  constexpr uint32_t GROUP_COLS = D == 64 ? 128 : 256;  // S; P in columns 0 .. 63 of it
  constexpr uint32_t O_OFF = D == 64 ? 64 : 128;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t IDESC_PV = make_idesc(IDESC_C_F32, IDESC_F16, IDESC_F16, 0, 1, 128, D);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* tiles = smem;  // [GROUPS][Q, K, V]
  uint64_t* qk_full = reinterpret_cast<uint64_t*>(tiles + GROUPS * 3 * TILE_BYTES);  // [GROUPS] each
  uint64_t* v_full = qk_full + GROUPS;
  uint64_t* s_full = v_full + GROUPS;
  uint64_t* p_full = s_full + GROUPS;
  uint64_t* o_full = p_full + GROUPS;
  uint64_t* free_bar = o_full + GROUPS;  // the group is through with the item's tiles and columns
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(free_bar + GROUPS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    if constexpr (!F32) {
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_v);
    }
    for (int g = 0; g < GROUPS; ++g) {
      mbar_init(&qk_full[g], F32 ? 4 : 1);
      mbar_init(&v_full[g], F32 ? 4 : 1);
      mbar_init(&s_full[g], 1);
      mbar_init(&p_full[g], 128);
      mbar_init(&o_full[g], 1);
      mbar_init(&free_bar[g], 128);
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

  // Items are dealt over the CTAs first, then over the groups: few items get an SM each.
  const int items = p.B * p.H;
  const int stride = int(gridDim.x) * GROUPS;
  auto keys_of = [&](int b) {
    const int n = p.kv_lens ? p.kv_lens[b] : p.S;
    return n < 0 ? 0 : (n > p.S ? p.S : n);
  };
  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (!F32 && elect_one()) {
      bool ok = true;
      uint32_t parity = 1;
      const uint32_t bytes = uint32_t(p.box_rows) * (D * 2);
      for (int base = int(blockIdx.x); base < items && ok; base += stride, parity ^= 1u) {
#pragma unroll 1
        for (int g = 0; g < GROUPS && ok; ++g) {
          const int item = base + g * int(gridDim.x);
          if (item >= items) break;
          const int b = item / p.H, h = item - b * p.H;
          if (!mbar_wait(&free_bar[g], parity, abort_flag)) { ok = false; break; }
          uint8_t* t = tiles + g * 3 * TILE_BYTES;
          mbar_arrive_expect_tx(&qk_full[g], 2 * bytes);
#pragma unroll
          for (int dc = 0; dc < DC; ++dc) {
            fa_tma_tile(t + dc * CHUNK_BYTES, &tmap_q, &qk_full[g], p.q_perm, dc * 64, 0, h, b);
            fa_tma_tile(t + TILE_BYTES + dc * CHUNK_BYTES, &tmap_k, &qk_full[g], p.k_perm, dc * 64, 0, h, b);
          }
          mbar_arrive_expect_tx(&v_full[g], bytes);
#pragma unroll
          for (int dc = 0; dc < DC; ++dc)
            fa_tma_tile(t + 2 * TILE_BYTES + dc * CHUNK_BYTES, &tmap_v, &v_full[g], p.v_perm, dc * 64, 0, h, b);
        }
      }
      if (!ok) {
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);  // the loads in flight end before the CTA does
      }
    }
  } else if (warp < 4) {
    // ---------------------------------------------------------------- MMA issuer of one group
    const int g = warp - 1;
    if (g < GROUPS && elect_one()) {
      const uint32_t qa = smem_u32(tiles + g * 3 * TILE_BYTES);
      const uint32_t ka = qa + TILE_BYTES, va = ka + TILE_BYTES;
      const uint32_t ts = tmem_base + uint32_t(g) * GROUP_COLS;
      uint32_t ph = 0;
      for (int item = int(blockIdx.x) + g * int(gridDim.x); item < items; item += stride) {
        const int kv_len = keys_of(item / p.H);
        const int steps = (kv_len + 15) / 16;
        const uint32_t idesc_qk = make_idesc(IDESC_C_F32, IDESC_F16, IDESC_F16, 0, 0, 128, steps * 16) | p.qk_negate;
        if (!mbar_wait(&qk_full[g], ph, abort_flag)) break;
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          if (steps == 0) break;
          const uint32_t off = (ks / 4) * CHUNK_BYTES + (ks % 4) * 32;
          mma_f16_ss(ts, make_smem_desc_sw128(qa + off, 1024, 16), make_smem_desc_sw128(ka + off, 1024, 16), idesc_qk, ks != 0 ? 1u : 0u);
        }
        tc_commit(&s_full[g]);
        // P is in tensor memory, so S has been read by every thread of the group
        if (!mbar_wait(&v_full[g], ph, abort_flag) || !mbar_wait(&p_full[g], ph, abort_flag)) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int ks = 0; ks < steps; ++ks)
          mma_f16_ts(ts + O_OFF, ts + uint32_t(ks * 8), make_smem_desc_sw128(va + ks * (16 * 128), 1024, CHUNK_BYTES), IDESC_PV, ks != 0 ? 1u : 0u);
        tc_commit(&o_full[g]);
        ph ^= 1u;
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax groups
    const int g = (warp - 4) >> 2;
    const int quad = warp & 3;
    const int q = quad * 32 + lane;
    const uint32_t tmem_s = tmem_base + uint32_t(g) * GROUP_COLS + (uint32_t(quad * 32) << 16);
    const uint32_t tmem_o = tmem_s + O_OFF;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    uint32_t ph = 0;
    for (int item = int(blockIdx.x) + g * int(gridDim.x); item < items; item += stride) {
      const int b = item / p.H, h = item - b * p.H;
      const int kv_len = keys_of(b);
      float l_sum = 0.f;
      if constexpr (F32) {
        // The output of the item before is staged in its Q tile, by every warp.  (A bounded wait, unlike bar.sync: a warp whose
        // wait for S or O has run out never comes here.)
        if (item != int(blockIdx.x) + g * int(gridDim.x) && !mbar_wait_warp(&free_bar[g], ph ^ 1u, abort_flag)) break;
        uint8_t* tile = tiles + g * 3 * TILE_BYTES;
        const int t = int(threadIdx.x) - 128 - g * 128;
        const int64_t at = int64_t(item) * p.S * D;
        fa_convert_tile<D>(tile, p.q32 + at, p.S, p.box_rows, t);
        fa_convert_tile<D>(tile + TILE_BYTES, p.k32 + at, p.S, p.box_rows, t);
        fa_tile_ready(&qk_full[g], lane);
        fa_convert_tile<D>(tile + 2 * TILE_BYTES, p.v32 + at, p.S, p.box_rows, t);
        fa_tile_ready(&v_full[g], lane);
      }
      const int p_chunks = (kv_len + 31) / 32;  // 32-key chunks of P that P V reads
      // chunks with a key of any row of this warp, and those whose keys are valid for all its rows
      int n_chunks = p_chunks, n_plain = kv_len / 32, lim = kv_len;
      if (p.causal) {
        n_chunks = min(n_chunks, quad + 1);
        n_plain = min(n_plain, quad);
        lim = min(lim, q + 1);
      }
      if (!mbar_wait_warp(&s_full[g], ph, abort_flag)) break;
      tc_fence_after_sync();
      // the row maximum, 64 columns a step
      float mx = -INFINITY;
      uint32_t sv[2][32];
#pragma unroll
      for (int c2 = 0; c2 < 2; ++c2) {
        if (2 * c2 < n_chunks) {
          __syncwarp();
          tmem_ld_32x32(tmem_s + c2 * 64, sv[0]);
          tmem_ld_32x32(tmem_s + c2 * 64 + 32, sv[1]);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (2 * c2 + c < n_chunks) {
              if (2 * c2 + c >= n_plain) mask_chunk(sv[c], lim - (2 * c2 + c) * 32);
              mx = fmaxf(mx, chunk_max(sv[c]));
            }
          }
        }
      }
      const float m_use = mx == -INFINITY ? 0.f : mx * p.scale_log2;
      const float2 nm2 = make_float2(-m_use, -m_use);
      // probabilities -> tensor memory (fp16 pairs); row sum by chunks: even keys, odd keys, both, chunks in order.
      // A chunk is fetched again while the one before it is worked on; P of a chunk lies in columns of earlier chunks.
      __syncwarp();
      if (n_chunks > 0) tmem_ld_32x32(tmem_s, sv[0]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (c < p_chunks) {
          uint32_t pk[16];
          tmem_wait_ld();
          __syncwarp();
          if (c < 3 && c + 1 < n_chunks) tmem_ld_32x32(tmem_s + (c + 1) * 32, sv[(c + 1) & 1]);
          if (c < n_chunks) {
            if (c >= n_plain) mask_chunk(sv[c & 1], lim - c * 32);
            float2 rs = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float2 x = f2fma(make_float2(__uint_as_float(sv[c & 1][2 * i]), __uint_as_float(sv[c & 1][2 * i + 1])), sc2, nm2);
              const float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
              rs = f2add(rs, e);
              const __half2 hh = __floats2half2_rn(e.x, e.y);
              pk[i] = *reinterpret_cast<const uint32_t*>(&hh);
            }
            l_sum += rs.x + rs.y;
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) pk[i] = 0u;
          }
          tmem_st_32x16(tmem_s + c * 16, pk);
        }
      }
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(&p_full[g]);
      if (!mbar_wait_warp(&o_full[g], ph, abort_flag)) break;
      tc_fence_after_sync();
      fa_write_output<D>(p, tiles + g * 3 * TILE_BYTES + quad * 4096, tmem_o, kv_len > 0, l_sum, lane, quad * 32, p.S, b, h, 0);
      tc_fence_before_sync();
      fence_proxy_async_smem();  // the next item's Q tile is loaded (or converted) over the staged rows
      mbar_arrive(&free_bar[g]);
      ph ^= 1u;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

}  // namespace zen
