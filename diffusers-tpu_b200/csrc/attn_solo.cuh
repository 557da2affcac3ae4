// Joint-attention forward for sm_100a on 128-row query blocks: the kernel of attn_kernel.cuh on one query tile.
//
// The two softmax groups take alternate key tiles, S(e) = Q K_e^T for group e % 2, each with its own (O_t, m, l); warp
// roles, tensor memory and barriers are those of the two-tile kernel, and group 0 merges (O_0, m, l) with
// (O_1, m, l) at the end.  A block is through its keys in half as many periods of the loop.  Taken for launches whose
// 256-row blocks leave SMs idle or hold empty query tiles (solo_blocks in attn_api.cu).  It reads K and V once per 128
// rows, through a ring of six slots: with long keys the loads bound it, 8 TB/s out of L2.
//
// The issuers wait for the loads.  While each group had an S of its own, one of its threads did, in the time that it waited for
// S; with one S those checks stand between the arrival of S and its read, in the chain that sets the pace.  Device time of
// calls in short loops, P over S / one S, checks in the groups / checks in the issuers: 1 x 3 heads x 1280 rows against 32 key
// tiles 33.8 / 32.1 / 30.1 us, with bounded logits 32.4 / 32.4 / 28.7, as a partial state 34.5 / 37.4 / 30.8, by a table 35.6 /
// 37.0 / 31.3; 2 x 24 x 333 queries against 16731 keys 158.3 / 144.4 / 135.7.
//
// A kernel of its own rather than a case of the other: the two-tile kernel's loop is sensitive to its neighbourhood,
// and as a template parameter of that body this form cost long sequences 2%.
// Measured in loops of half a second, 256-row blocks -> this: 1 x 6 heads x 2304 rows (54 -> 108 blocks) 31.3 -> 20.3 us; 2 x 24
// heads x 333 queries against 16731 keys (96 blocks, a third of their rows empty -> 144 blocks) 213 -> 151 us.
#pragma once

#include "attn_kernel.cuh"

namespace dtb {

constexpr int kSoloStages = 6;               // K/V ring slots
constexpr int kSiteSoloReady = 70;           // beside WaitSite, reported in status[1] when a wait runs out

struct __align__(8) SoloBarriers {
  uint64_t q_full[1];
  uint64_t kv_full[kSoloStages];
  uint64_t kv_empty[kSoloStages];
  uint64_t s_full[2];
  uint64_t p_lo[2];         // first 64 keys of P_t written
  uint64_t p_hi[2];         // last 64 keys of P_t written
  uint64_t pv_done[2];      // P_t V of a tile has run
  uint64_t s_free;          // S has been read into registers
  uint64_t solo_ready;      // ml holds group 1's (m, l)
  float2 ml[kBlockM];
  uint32_t tmem_base;
  int abort_flag;
};

constexpr size_t kSoloSmemBytes = 1024 /* alignment slack */ + kTileBytes + kSoloStages * kTileBytes + sizeof(SoloBarriers);

template <bool kResidual, bool kQkFp8>
__global__ void __launch_bounds__(kNumThreads, 1) attn_solo_kernel(const __grid_constant__ AttnKernelParams p) {
  constexpr uint32_t kQkTileBytes = kQkFp8 ? kPanelBytes : kTileBytes;   // bytes of one 128-row Q or K tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem;
  {
    const uint32_t a = smem_u32(smem_raw);
    smem = smem_raw + (((a + 1023u) & ~1023u) - a);
  }
  uint8_t* smem_q = smem;
  uint8_t* smem_kv = smem + kTileBytes;
  SoloBarriers* bars = reinterpret_cast<SoloBarriers*>(smem_kv + kSoloStages * kTileBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int b = blockIdx.z, h = blockIdx.y;
  const int hk = h / (p.Hq / p.Hkv);
  const int q0 = blockIdx.x * kBlockM;

  // Valid keys of this call: global indices [kv_offset, kv_offset + Skv) below kv_len[b].
  const int kv_len_b = (p.kv_len != nullptr) ? max(p.kv_len[b], 0) : 0x7fffffff;
  const int kv_eff = max(min(kv_len_b - p.kv_offset, p.Skv), 0);
  // Key tiles this query block visits: all of [0, ceil(kv_eff / 128)) or, for a block-sparse call, the
  // entries of its table row that start below kv_eff (the row is ascending: binary search).
  const int32_t* tile_list = nullptr;
  int n_tiles = (kv_eff + kBlockN - 1) / kBlockN;
  if (p.kv_table != nullptr) {
    const int cls = p.head_class != nullptr ? p.head_class[h] : 0;
    const int64_t trow = static_cast<int64_t>(cls) * p.table_qblocks + q0 / (kQTiles * kBlockM);
    tile_list = p.kv_table + trow * p.table_width;
    int lo = 0, hi = p.kv_count[trow];
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (tile_list[mid] * kBlockN < kv_eff) lo = mid + 1; else hi = mid;
    }
    n_tiles = lo;
  }
  const bool block_padded = p.zero_padded_rows && (p.q_offset + q0 >= kv_len_b);

  const int64_t acc_base = (static_cast<int64_t>(b) * p.Hq + h) * p.Sq;   // row of the state arrays of query row 0

  if (n_tiles <= 0 || block_padded) {
    // Nothing to attend to: emit zeros (normal) or the empty state (residual, when initialising).
    if (threadIdx.x < kBlockM) {
      const int row = q0 + threadIdx.x;
      if (row < p.Sq) {
        if (!kResidual) {
          uint4* dst;
          if (p.o_shard_rows > 0) {
            const int dest = row / p.o_shard_rows;
            dst = reinterpret_cast<uint4*>(
                p.o_peer[dest] + ((static_cast<int64_t>(b) * p.o_total_heads + p.o_head_offset + h) * p.o_shard_rows +
                                  (row - dest * p.o_shard_rows)) * kHeadDim);
          } else {
            dst = reinterpret_cast<uint4*>(p.o + b * p.o_stride_b + h * p.o_stride_h + row * p.o_stride_s);
          }
#pragma unroll
          for (int i = 0; i < kHeadDim * 2 / 16; ++i) dst[i] = make_uint4(0, 0, 0, 0);
        } else if (p.acc_init) {
          float4* dst = reinterpret_cast<float4*>(p.acc_o + (acc_base + row) * kHeadDim);
#pragma unroll
          for (int i = 0; i < kHeadDim / 4; ++i) dst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          p.acc_m[acc_base + row] = -INFINITY;
          p.acc_l[acc_base + row] = 0.f;
        }
      }
    }
    return;
  }

  AbortCtx ctx{&bars->abort_flag, p.status};

  if (threadIdx.x == kMmaWarp * 32) {
    bars->abort_flag = 0;
    mbar_init(smem_u32(&bars->q_full[0]), 1);
    for (int i = 0; i < kQTiles; ++i) {
      mbar_init(smem_u32(&bars->s_full[i]), 1);
      mbar_init(smem_u32(&bars->p_lo[i]), kBlockM);
      mbar_init(smem_u32(&bars->p_hi[i]), kBlockM);
      mbar_init(smem_u32(&bars->pv_done[i]), 1);
    }
    mbar_init(smem_u32(&bars->s_free), kBlockM);
    mbar_init(smem_u32(&bars->solo_ready), kBlockM);
    for (int i = 0; i < kSoloStages; ++i) {
      mbar_init(smem_u32(&bars->kv_full[i]), 1);
      mbar_init(smem_u32(&bars->kv_empty[i]), 1);
    }
    mbar_fence_init();
  }
  if (warp == kLoadWarp && lane == 0) {
    tma_prefetch_desc(&p.tmap_q);
    tma_prefetch_desc(&p.tmap_k);
    tma_prefetch_desc(&p.tmap_v);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&bars->tmem_base), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  // Places in the K/V ring: K_0 K_1 V_0 K_2 V_1 ... K_{n-1} V_{n-2} V_{n-1}.
  auto place_k = [&](int e) { return e == 0 ? 0 : 2 * e - 1; };
  auto place_v = [&](int e) { return e == n_tiles - 1 ? 2 * n_tiles - 1 : 2 * e + 2; };
  auto reloaded = [&](int i) { return i + kSoloStages < 2 * n_tiles; };   // as in the two-tile kernel

  if (warp == kLoadWarp) {
    // ------------------------------------------------------------------ TMA producer
    setmaxnreg_dec<kRegsService>();
    bool ok = true;
    if (lane == 0) {
      {
        const uint32_t bar = smem_u32(&bars->q_full[0]);
        mbar_expect_tx(bar, kQkTileBytes);
        const uint32_t dst = smem_u32(smem_q);
        tma_load_4d(dst, &p.tmap_q, bar, 0, q0, h, b);
        if (!kQkFp8) tma_load_4d(dst + kPanelBytes, &p.tmap_q, bar, 64, q0, h, b);
      }
      for (int i = 0; i < 2 * n_tiles && ok; ++i) {
        const int slot = i % kSoloStages;
        const int use = i / kSoloStages;
        if (use > 0) ok = mbar_wait(smem_u32(&bars->kv_empty[slot]), (use - 1) & 1, ctx, SITE_KV_EMPTY + slot);
        if (!ok) break;
        const uint32_t bar = smem_u32(&bars->kv_full[slot]);
        const bool last = i == 2 * n_tiles - 1;
        const bool is_v = last || (i > 0 && (i & 1) == 0);
        const int entry = last ? n_tiles - 1 : is_v ? (i - 2) >> 1 : (i + 1) >> 1;
        mbar_expect_tx(bar, is_v ? kTileBytes : kQkTileBytes);
        const uint32_t dst = smem_u32(smem_kv + slot * kTileBytes);
        const int row = (tile_list != nullptr ? tile_list[entry] : entry) * kBlockN;
        const CUtensorMap* tm = is_v ? &p.tmap_v : &p.tmap_k;
        tma_load_4d(dst, tm, bar, 0, row, hk, b);
        if (is_v || !kQkFp8) tma_load_4d(dst + kPanelBytes, tm, bar, 64, row, hk, b);
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------------ issuer of S(e) = Q K_e^T
    setmaxnreg_dec<kRegsService>();
    constexpr uint32_t idesc_qk = kQkFp8 ? make_idesc_e4m3(kBlockM, kBlockN) : make_idesc_bf16(kBlockM, kBlockN, false, false);
    const uint64_t q_desc0 = make_smem_desc_sw128(smem_u32(smem_q), 16, 1024);
    const uint64_t k_desc0 = make_smem_desc_sw128(smem_u32(smem_kv), 16, 1024);

    auto issue_qk = [&](int t, int slot) {
      if (elect_one()) {
        const uint64_t b0 = k_desc0 + static_cast<uint64_t>((slot * kTileBytes) >> 4);
        if (kQkFp8) {
#pragma unroll
          for (int kk = 0; kk < kHeadDim / 32; ++kk) {   // 32 one-byte elements = 32 bytes of the swizzled row
            const uint64_t off = static_cast<uint64_t>((kk * 32) >> 4);
            mma_ss_f8(tmem_base, q_desc0 + off, b0 + off, idesc_qk, kk > 0 ? 1u : 0u);
          }
        } else {
#pragma unroll
          for (int kk = 0; kk < kHeadDim / 16; ++kk) {
            const uint64_t off = static_cast<uint64_t>(((kk & 3) * 32 + (kk >> 2) * kPanelBytes) >> 4);
            mma_ss(tmem_base, q_desc0 + off, b0 + off, idesc_qk, kk > 0 ? 1u : 0u);
          }
        }
        mma_commit(smem_u32(&bars->s_full[t]));
      }
      __syncwarp();
    };
    auto commit_to = [&](uint64_t* bar) {
      if (elect_one()) mma_commit(smem_u32(bar));
      __syncwarp();
    };

    bool ok = warp_wait(&bars->q_full[0], 0, ctx, SITE_Q_FULL);
    for (int e = 0; e < n_tiles && ok; ++e) {
      const int i = place_k(e), slot = i % kSoloStages;
      ok = warp_wait(&bars->kv_full[slot], (i / kSoloStages) & 1, ctx, SITE_KV_FULL + slot);
      if (ok && e > 0) ok = warp_wait(&bars->s_free, (e - 1) & 1, ctx, SITE_S_FREE);
      if (!ok) break;
      tc_fence_after();
      issue_qk(e & 1, slot);
      if (reloaded(i)) commit_to(&bars->kv_empty[slot]);
    }
  } else if (warp == kPvWarp) {
    // ------------------------------------------------------------------ issuer of O_t += P_t(e) V_e
    setmaxnreg_dec<kRegsService>();
    constexpr uint32_t idesc_pv = make_idesc_bf16(kBlockM, kHeadDim, false, true);
    const uint64_t v_desc0 = make_smem_desc_sw128(smem_u32(smem_kv), kPanelBytes, 1024);
    bool ok = true;

    auto issue_pv = [&](int t, int slot, int half, bool accumulate) {
      if (elect_one()) {
        const uint64_t b0 = v_desc0 + static_cast<uint64_t>((slot * kTileBytes) >> 4);
        const uint32_t d_tmem = tmem_base + (kQTiles + t) * kBlockN;
        const uint32_t a_tmem = tmem_base + kBlockN + t * (kBlockN / 2);
#pragma unroll
        for (int kk = half * 4; kk < half * 4 + 4; ++kk) {
          const uint64_t off = static_cast<uint64_t>((kk * 16 * 128) >> 4);
          mma_ts(d_tmem, a_tmem + kk * 8, b0 + off, idesc_pv, (accumulate || kk > 0) ? 1u : 0u);
        }
      }
      __syncwarp();
    };
    auto commit_to = [&](uint64_t* bar) {
      if (elect_one()) mma_commit(smem_u32(bar));
      __syncwarp();
    };
    const bool o_preloaded = kResidual && !p.acc_init;
    for (int e = 0; e < n_tiles && ok; ++e) {
      const int t = e & 1, j = e >> 1, i = place_v(e), slot = i % kSoloStages;
      ok = warp_wait(&bars->kv_full[slot], (i / kSoloStages) & 1, ctx, SITE_KV_FULL + slot);
      if (ok) ok = warp_wait(&bars->p_lo[t], j & 1, ctx, SITE_P_FULL + t);
      if (!ok) break;
      tc_fence_after();
      issue_pv(t, slot, 0, j > 0 || (o_preloaded && t == 0));
      ok = warp_wait(&bars->p_hi[t], j & 1, ctx, SITE_P_HI + t);
      if (!ok) break;
      tc_fence_after();
      issue_pv(t, slot, 1, true);
      commit_to(&bars->pv_done[t]);
      if (reloaded(i)) commit_to(&bars->kv_empty[slot]);
    }
  } else if (warp < kMmaWarp) {
    // ------------------------------------------------------------------ softmax groups
    setmaxnreg_inc<kRegsSoftmax>();
    const int t = warp >> 2;                       // group: key tiles e with e % 2 == t
    const int row_in_tile = threadIdx.x & (kBlockM - 1);
    const int row = q0 + row_in_tile;  // query row within this call
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_tmem = tmem_base + lane_off;
    const uint32_t p_tmem = tmem_base + lane_off + kBlockN + t * (kBlockN / 2);
    const uint32_t o_tmem = tmem_base + lane_off + (kQTiles + t) * kBlockN;
    const float scale_log2 = p.scale_log2;
    const bool row_in_range = row < p.Sq;
    const int64_t acc_row = acc_base + row;
    const uint32_t bar_s_free = smem_u32(&bars->s_free);
    const uint32_t bar_p_lo = smem_u32(&bars->p_lo[t]);
    const uint32_t bar_p_hi = smem_u32(&bars->p_hi[t]);

    // A state, and group 1, start from a finite offset.  Group 1's first tile is not the first tile of the row: where all
    // its logits are -inf, they weigh 0 beside those of tile 0, and -inf - (-inf) would make them NaN.
    float m_used = kResidual || t == 1 ? kLowestOffset : -INFINITY;
    float l_sum = 0.f;
    bool fixed_m = false;
    if (p.mk != nullptr && p.mk[p.Hq + h] > 0.5f) {
      fixed_m = true;
      m_used = p.mk[h] - kFixedMRecenter;
    }
    bool o_live = false;
    if (kResidual && !p.acc_init && t == 0) {
      // Bring the running state of this row into registers / tensor memory.
      float m_in = -INFINITY, l_in = 0.f;
      if (row_in_range) {
        m_in = p.acc_m[acc_row];
        l_in = p.acc_l[acc_row];
      }
      // S is not read before, and with one S the other group waits for that too, so the load is in the way until it is over.
      // What it takes is a cycle per row and load instruction of a warp (32 rows lie in 32 lines), hence loads of 32 bytes
      // where the state allows them: 1 x 3 heads x 1280 rows against 4 / 10 key tiles 12.8 / 17.4 us with 16 bytes, 11.8 / 16.3
      // with 32.  (Two S, 16 bytes: 12.0 / 17.4.)
      const float* src = p.acc_o + acc_row * kHeadDim;
      const bool wide = (reinterpret_cast<uintptr_t>(p.acc_o) & 31) == 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = 0;
        if (row_in_range && wide) {
#pragma unroll
          for (int i = 0; i < 4; ++i) ld_global8(src + c * 32 + 8 * i, r + 8 * i);
        } else if (row_in_range) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 v = reinterpret_cast<const float4*>(src)[c * 8 + i];
            r[4 * i] = __float_as_uint(v.x);
            r[4 * i + 1] = __float_as_uint(v.y);
            r[4 * i + 2] = __float_as_uint(v.z);
            r[4 * i + 3] = __float_as_uint(v.w);
          }
        }
        tmem_st32(o_tmem + c * 32, r);
      }
      tmem_wait_st();
      o_live = true;
      if (fixed_m) {
        // The incoming state is expressed relative to m_in; re-express it relative to the fixed offset.
        // (Callers that use the bounded-logit mode keep one offset for the whole ring, so this is a no-op.)
        const bool shift = (m_in != m_used) && (l_in > 0.f);
        if (__any_sync(0xffffffffu, shift)) {
          const float alpha = shift ? ex2(m_in - m_used) : 1.0f;
          l_in *= alpha;
          uint32_t r[32];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            tmem_ld32_sync(o_tmem + c * 32, r);
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st32(o_tmem + c * 32, r);
          }
          tmem_wait_st();
        }
      } else {
        m_used = fmaxf(m_in, kLowestOffset);   // -inf: no key yet
      }
      l_sum = l_in;
    }

    bool ok = true;
    const int n_own = (n_tiles + 1 - t) >> 1;   // key tiles of this group
    for (int j = 0; j < n_own && ok; ++j) {
      const int e = 2 * j + t;
      ok = warp_wait(&bars->s_full[t], j & 1, ctx, SITE_S_FULL + t);
      if (!ok) break;
      tc_fence_after();
      const int tile = tile_list != nullptr ? tile_list[e] : e;
      const int valid_cols = min(kv_eff - tile * kBlockN, kBlockN);
      auto wait_pv = [&]() {
        if (j == 0) return true;
        const bool done = warp_wait(&bars->pv_done[t], (j - 1) & 1, ctx, SITE_O_FULL + t);
        tc_fence_after();
        return done;
      };
      if (fixed_m) {
        ok = softmax_tile<true, false>(s_tmem, p_tmem, o_tmem, scale_log2, valid_cols, o_live, m_used, l_sum, bar_s_free, bar_p_lo, bar_p_hi, wait_pv);
      } else {
        ok = softmax_tile<false, false>(s_tmem, p_tmem, o_tmem, scale_log2, valid_cols, o_live, m_used, l_sum, bar_s_free, bar_p_lo, bar_p_hi, wait_pv);
      }
      o_live = true;
    }
    if (ok && n_own > 0) ok = warp_wait(&bars->pv_done[t], (n_own - 1) & 1, ctx, SITE_O_FULL + t);
    // Group 1 hands over its (m, l); its O is read by group 0's warps, which see the same lanes.
    float w_own = 1.f, w_other = 1.f;      // factors of O_0 and O_1
    const bool merge = n_tiles > 1;
    if (merge && ok) {
      float2* ml = &bars->ml[row_in_tile];
      if (t == 1) {
        *ml = make_float2(m_used, l_sum);
        mbar_arrive(smem_u32(&bars->solo_ready));
      } else {
        ok = warp_wait(&bars->solo_ready, 0, ctx, kSiteSoloReady) && warp_wait(&bars->pv_done[1], ((n_tiles >> 1) - 1) & 1, ctx, SITE_O_FULL + 1);
        if (ok) {
          // A group whose sum is 0 has no say in the offset.  Any other sum has, NaN included, and both accumulators are
          // always taken: what is not finite in either half of the keys shows in the output, as with one group.
          const float2 other = *ml;
          const float m = other.y == 0.f ? m_used : l_sum == 0.f ? other.x : fmaxf(m_used, other.x);
          w_own = l_sum == 0.f || m_used == m ? 1.f : ex2(m_used - m);
          w_other = other.y == 0.f || other.x == m ? 1.f : ex2(other.x - m);
          l_sum = l_sum * w_own + other.y * w_other;
          m_used = m;
        }
      }
    }
    if (ok && t == 0) {
      tc_fence_after();
      // 32 columns of the row's finished O.
      auto load_o = [&](int c, uint32_t (&r)[32]) {
        tmem_ld32_sync(o_tmem + c * 32, r);
        if (merge) {
          uint32_t r1[32];
          tmem_ld32_sync(o_tmem + kBlockN + c * 32, r1);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            r[i] = __float_as_uint(fmaf(__uint_as_float(r1[i]), w_other, __uint_as_float(r[i]) * w_own));
        }
      };
      if (kResidual) {
        float4* dst = reinterpret_cast<float4*>(p.acc_o + acc_row * kHeadDim);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          load_o(c, r);
          if (row_in_range) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              dst[c * 8 + i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                           __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
          }
        }
        if (row_in_range) {
          p.acc_m[acc_row] = m_used;
          p.acc_l[acc_row] = l_sum;
        }
      } else {
        // Normalise, round to bf16 and stage the 32 rows of this warp in the (now dead) Q tile of
        // this group, 16-byte chunks XOR-swizzled by row so neither side bank-conflicts; then the warp
        // writes whole 256-byte rows, two per store instruction, to this GPU's output or, for a
        // head-parallel call whose output is sequence-sharded, straight into the owning peer's buffer.
        const bool padded = p.zero_padded_rows && (p.q_offset + row >= kv_len_b);
        const float inv = (l_sum > 0.f && !padded) ? (1.0f / l_sum) : 0.f;
        uint8_t* stage = smem_q + (warp & 3) * (32 * kHeadDim * 2);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          load_o(c, r);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 v;
            v.x = pack_bf16x2(__uint_as_float(r[8 * i]) * inv, __uint_as_float(r[8 * i + 1]) * inv);
            v.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]) * inv, __uint_as_float(r[8 * i + 3]) * inv);
            v.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]) * inv, __uint_as_float(r[8 * i + 5]) * inv);
            v.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]) * inv, __uint_as_float(r[8 * i + 7]) * inv);
            const int chunk = c * 4 + i;
            *reinterpret_cast<uint4*>(stage + lane * 256 + ((chunk ^ (lane & 15)) << 4)) = v;
          }
        }
        __syncwarp();
        const int row0 = q0 + (warp & 3) * 32;   // first query row of this warp
        const int sub = lane >> 4;                              // which of the two rows of a store
        const int chunk = lane & 15;
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
          const int rl = 2 * i + sub;
          const int grow = row0 + rl;
          if (grow < p.Sq) {
            const uint4 v = *reinterpret_cast<const uint4*>(stage + rl * 256 + ((chunk ^ (rl & 15)) << 4));
            __nv_bfloat16* dst_row;
            if (p.o_shard_rows > 0) {
              const int dest = grow / p.o_shard_rows;
              dst_row = p.o_peer[dest] +
                        ((static_cast<int64_t>(b) * p.o_total_heads + p.o_head_offset + h) * p.o_shard_rows +
                         (grow - dest * p.o_shard_rows)) * kHeadDim;
            } else {
              dst_row = p.o + b * p.o_stride_b + h * p.o_stride_h + grow * p.o_stride_s;
            }
            reinterpret_cast<uint4*>(dst_row)[chunk] = v;
          }
        }
      }
    }
  }

  else {
    setmaxnreg_dec<kRegsService>();  // idle warps of the service warpgroup
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (bars->abort_flag) {
    // Give copies and MMAs that are still in flight time to land before the
    // shared and tensor memory they target is released.
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 0) tmem_dealloc(tmem_base, kTmemCols);
}

}  // namespace dtb
