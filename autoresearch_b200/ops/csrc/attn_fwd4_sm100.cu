// Flash attention forward for head_dim = 128: one 128-query tile per CTA, half an SM's shared memory and TMEM per CTA, so
// that two CTAs run on every SM.
//
// The chain of a query tile is serial (scores -> softmax -> probabilities -> P V -> next scores), and the tensor pipe idles
// through most of it.  attn_fwd3_sm100.cu fills the gaps with a second query tile of the same CTA, served by one issuing
// thread in a fixed order; here the second tile belongs to another CTA.  Its issuing thread puts its products into the pipe
// whenever they are ready, its start (TMEM, barriers, first loads: several us) and its epilogue run under the other CTA's
// loop - what counts where a tile sees three key tiles, as in a sliding window of 256 - and the last wave is half as coarse.
//
//   shared memory  Q 32 KB | K 32 KB | V 32 KB.  One slot each: K(t+1) is fetched while the softmax of tile t runs, V(t+1)
//                  while S(t+1) and its softmax do.
//   TMEM           S 128 columns | O 128 columns.  P (bf16 pairs, 64 columns) overwrites the upper half of S, whose scores the
//                  thread holds in registers by then; S(t+1) is issued behind P V(t), and one thread's MMAs run in order.
//   registers      168 per thread (two CTAs of 192): the row maximum is taken over the whole score row, of which the upper
//                  64 columns stay in registers; the lower 64 are read from TMEM again for their exponentials.
//
// Mask semantics: key j is visible to query i iff i - window <= j <= i (brain/src/forward.rs:1134-1138); the reference calls
// a Hopper-only FlashAttention-3 build here (brain/src/forward.rs:1124-1177).
#include "attn_common.cuh"

namespace arb {

struct Fwd4Smem {
  static constexpr int Q = 0, K = 32768, V = 65536;
  static constexpr int BAR = 3 * 32768;
  static constexpr int TOTAL = BAR + 128 + 1024;      // + alignment slack
};
static_assert(2 * (Fwd4Smem::TOTAL + 1024) <= 233472, "two CTAs must fit the 228 KB of an SM");

// Exponentials of 32 scores of a row: e = 2^(s*c - mc), bf16 pairs into pk[16], row sum into the packed accumulator
template <bool MASK>
__device__ __forceinline__ void exp32_mufu(const uint32_t (&s)[32], uint32_t* pk, unsigned long long c2, unsigned long long nmc2,
                                           int col0, int mlo, unsigned span, unsigned long long& rs2) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float x0, x1;
    unpk2(fma2(pk2(__uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1])), c2, nmc2), x0, x1);
    float e0 = fast_exp2(x0), e1 = fast_exp2(x1);
    if constexpr (MASK) {
      e0 = (unsigned(col0 + 2 * j - mlo) <= span) ? e0 : 0.f;
      e1 = (unsigned(col0 + 2 * j + 1 - mlo) <= span) ? e1 : 0.f;
    }
    rs2 = add2(rs2, pk2(e0, e1));
    pk[j] = pack_bf16(e0, e1);
  }
}

__global__ void __launch_bounds__(ATT_THREADS, 2)
attn_fwd4_k(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
            const __grid_constant__ CUtensorMap tmV, const AttnArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Fwd4Smem::BAR);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* v_full = bars + 2;
  uint64_t* s_full = bars + 3;        // S(t) complete: scores readable, K slot free
  uint64_t* p_full = bars + 4;        // [2] P(t) of keys 64..127, then of keys 0..63, written (4 arrivals)
  uint64_t* pv_done = bars + 6;       // P V(t) complete: V slot free, after the last one O is final
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 7);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_mt = (p.T + 127) / 128;
  const AttnTile tile = attn_tile(p, n_mt);
  const int mt = n_mt - 1 - tile.rank, h = tile.h, b = tile.b;      // later query tiles see more keys
  const int m0 = mt * 128;
  const int j_lo = (p.window >= p.T) ? 0 : max(0, (m0 - p.window) / 128);
  const int n_tiles = min((p.T - 1) / 128, (m0 + 127) / 128) - j_lo + 1;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1); mbar_init(k_full, 1); mbar_init(v_full, 1);
    mbar_init(s_full, 1); mbar_init(&p_full[0], 4); mbar_init(&p_full[1], 4); mbar_init(pv_done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_enter();                 // global memory is not touched above
  const uint32_t TM_S = tmem, TM_P = tmem + 64, TM_O = tmem + 128;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
      mbar_expect_tx(q_full, 32768);                 // rows past the end of the sequence are zero-filled
      tma_load_4d(smem + Fwd4Smem::Q, &tmQ, q_full, 0, h, m0, b);
      tma_load_4d(smem + Fwd4Smem::Q + 16384, &tmQ, q_full, 64, h, m0, b);
      for (int t = 0; t < n_tiles; ++t) {
        const int n0 = (j_lo + t) * 128;
        if (t > 0 && !mbar_wait(s_full, uint32_t(t - 1) & 1u, abort_flag)) break;
        mbar_expect_tx(k_full, 32768);
        tma_load_4d(smem + Fwd4Smem::K, &tmK, k_full, 0, h, n0, b);
        tma_load_4d(smem + Fwd4Smem::K + 16384, &tmK, k_full, 64, h, n0, b);
        if (t > 0 && !mbar_wait(pv_done, uint32_t(t - 1) & 1u, abort_flag)) break;
        mbar_expect_tx(v_full, 32768);
        tma_load_4d(smem + Fwd4Smem::V, &tmV, v_full, 0, h, n0, b);
        tma_load_4d(smem + Fwd4Smem::V + 16384, &tmV, v_full, 64, h, n0, b);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
      constexpr uint32_t idesc_o = make_idesc_bf16(128, 128, false, true);
      // descriptor words once; a K slice is a 32-bit add on the low word (start address >> 4)
      const uint32_t hi_k = uint32_t(make_smem_desc(0, 0, 1024) >> 32), hi_v = uint32_t(make_smem_desc(0, 16384, 1024) >> 32);
      const uint32_t q_lo = uint32_t(make_smem_desc(smem_u32(smem + Fwd4Smem::Q), 0, 1024));
      const uint32_t k_lo = uint32_t(make_smem_desc(smem_u32(smem + Fwd4Smem::K), 0, 1024));
      const uint32_t v_lo = uint32_t(make_smem_desc(smem_u32(smem + Fwd4Smem::V), 16384, 1024));
      bool ok = mbar_wait(q_full, 0, abort_flag);
      auto issue_s = [&](int t) {
        if (!mbar_wait(k_full, uint32_t(t) & 1u, abort_flag)) { ok = false; return; }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t off = uint32_t(k >> 2) * 1024u + uint32_t(k & 3) * 2u;     // (16 KB half, 32 B slice) >> 4
          tc_mma_ss_lh(TM_S, q_lo + off, hi_k, k_lo + off, hi_k, idesc_s, k > 0);
        }
        tc_commit(s_full);
      };
      if (ok) issue_s(0);
      for (int t = 0; t < n_tiles && ok; ++t) {
        if (!mbar_wait(v_full, uint32_t(t) & 1u, abort_flag)) { ok = false; break; }
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {              // the upper keys' products run under the lower keys' exponentials
          if (!mbar_wait(&p_full[hf], uint32_t(t) & 1u, abort_flag)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t k = uint32_t(hf ? i : 4 + i);
            tc_mma_ts_lh(TM_O, TM_P + k * 8u, v_lo + k * 128u, hi_v, idesc_o, (t > 0 || hf > 0 || i > 0) ? 1u : 0u);
          }
        }
        if (!ok) break;
        tc_commit(pv_done);
        if (t + 1 < n_tiles) issue_s(t + 1);          // behind P V(t), which reads columns of the tile it overwrites
      }
    }
  } else {
    // ---------------- softmax / epilogue: thread <-> query row ----------------
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const int row = m0 + r;
    const uint32_t lane_addr = uint32_t(q * 32) << 16;
    const float c = p.scale * LOG2E;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int t = 0; t < n_tiles; ++t) {
      const int n0 = (j_lo + t) * 128;
      if (!mbar_wait(s_full, uint32_t(t) & 1u, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const bool need_mask = (n0 + 127 > m0) || (p.window < p.T && n0 < m0 + 127 - p.window) || (n0 + 127 >= p.T);
      // visible keys of this row inside the tile: column indices [mlo, mlo + span]
      const int mlo = (row < p.T) ? row - p.window - n0 : 128;
      const unsigned span = (row < p.T) ? unsigned(p.window) : 0u;
      uint32_t sc[32], sd[32];                           // columns 64..127 stay in registers
      float mx;
      {
        uint32_t sa[32], sb[32];
        tmem_ld32(TM_S + lane_addr, sa);
        tmem_ld32(TM_S + lane_addr + 32u, sb);
        tmem_wait_ld();
        tmem_ld32(TM_S + lane_addr + 64u, sc);
        tmem_ld32(TM_S + lane_addr + 96u, sd);
        if (need_mask) mx = max32<true>(sb, 32, mlo, span, max32<true>(sa, 0, mlo, span, -INFINITY));
        else mx = max32<false>(sb, 32, mlo, span, max32<false>(sa, 0, mlo, span, -INFINITY));
        tmem_wait_ld();
      }
      if (need_mask) mx = max32<true>(sd, 96, mlo, span, max32<true>(sc, 64, mlo, span, mx));
      else mx = max32<false>(sd, 96, mlo, span, max32<false>(sc, 64, mlo, span, mx));
      const float m_new = fmaxf(m_used, mx);
      bool resc = false;
      if (m_used == -INFINITY) m_used = m_new;            // nothing accumulated for this row yet
      else resc = (m_new - m_used) * c > 8.f;
      if (t > 0 && __any_sync(0xffffffffu, resc)) {
        // S(t) complete implies P V(t-1) complete: O is not in flight
        const float alpha = resc ? fast_exp2((m_used - m_new) * c) : 1.f;
        if (resc) { l *= alpha; m_used = m_new; }
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t v[32];
          tmem_ld32(TM_O + lane_addr + uint32_t(cc * 32), v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
          tmem_st32(TM_O + lane_addr + uint32_t(cc * 32), v);
        }
        tmem_wait_st();
      }
      const float mc = (m_used == -INFINITY) ? 0.f : m_used * c;
      const unsigned long long c2 = pk2(c, c), nmc2 = pk2(-mc, -mc);
      unsigned long long rs2 = pk2(0.f, 0.f);
      {
        uint32_t pk[32];
        if (need_mask) {
          exp32_mufu<true>(sc, pk, c2, nmc2, 64, mlo, span, rs2);
          exp32_mufu<true>(sd, pk + 16, c2, nmc2, 96, mlo, span, rs2);
        } else {
          exp32_mufu<false>(sc, pk, c2, nmc2, 64, mlo, span, rs2);
          exp32_mufu<false>(sd, pk + 16, c2, nmc2, 96, mlo, span, rs2);
        }
        tmem_st32(TM_P + lane_addr + 32u, pk);           // over scores that have been read
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[0]);
      {
        uint32_t sa[32], sb[32], pk[32];
        tmem_ld32(TM_S + lane_addr, sa);
        tmem_ld32(TM_S + lane_addr + 32u, sb);
        tmem_wait_ld();
        if (need_mask) {
          exp32_mufu<true>(sa, pk, c2, nmc2, 0, mlo, span, rs2);
          exp32_mufu<true>(sb, pk + 16, c2, nmc2, 32, mlo, span, rs2);
        } else {
          exp32_mufu<false>(sa, pk, c2, nmc2, 0, mlo, span, rs2);
          exp32_mufu<false>(sb, pk + 16, c2, nmc2, 32, mlo, span, rs2);
        }
        tmem_st32(TM_P + lane_addr, pk);
      }
      float r0, r1;
      unpk2(rs2, r0, r1);
      l += r0 + r1;
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[1]);
    }
    if (ok && mbar_wait(pv_done, uint32_t(n_tiles - 1) & 1u, abort_flag)) {
      tc_fence_after();
      const float inv_l = (l > 0.f) ? 1.f / l : 0.f;
      __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(p.o) + ((long long)b * p.T + row) * p.ldo + h * HD;
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        uint32_t v[32];
        tmem_ld32(TM_O + lane_addr + uint32_t(cc * 32), v);
        tmem_wait_ld();
        if (row < p.T) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            uint4 u;
            u.x = pack_bf16(__uint_as_float(v[j]) * inv_l, __uint_as_float(v[j + 1]) * inv_l);
            u.y = pack_bf16(__uint_as_float(v[j + 2]) * inv_l, __uint_as_float(v[j + 3]) * inv_l);
            u.z = pack_bf16(__uint_as_float(v[j + 4]) * inv_l, __uint_as_float(v[j + 5]) * inv_l);
            u.w = pack_bf16(__uint_as_float(v[j + 6]) * inv_l, __uint_as_float(v[j + 7]) * inv_l);
            *reinterpret_cast<uint4*>(orow + cc * 32 + j) = u;
          }
        }
      }
      if (row < p.T) p.lse[((long long)b * p.H + h) * p.T + row] = (l > 0.f) ? (m_used * p.scale + __logf(l)) : -INFINITY;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag && p.err) atomicExch(p.err, ERR_ATTN_TIMEOUT);
  if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, 256); }
}

int attn_fwd4_launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnArgs& a, cudaStream_t stream) {
  static PerDeviceOnce cfg;
  if (cfg.first()) { if (int r = set_smem(attn_fwd4_k, Fwd4Smem::TOTAL)) return r; }
  const unsigned grid = attn_grid(a.B, a.H, a.T, 128);
  if (!grid) return -3;
  return launch_dependent(true, attn_fwd4_k, grid, ATT_THREADS, Fwd4Smem::TOTAL, stream, tq, tk, tv, a);
}

}  // namespace arb
