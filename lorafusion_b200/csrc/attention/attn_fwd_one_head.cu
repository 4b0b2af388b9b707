// Attention forward (see attn_fwd.cu) where every query head has its own KV head: there is no second
// head to pair with, so one CTA handles one 128-row query tile of one head, and two threads share
// a query row.
//   warp 0      TMA producer: Q, then K and V tiles through two 2-stage rings of their own (a K slot is
//               free as soon as its S = Q K^T has completed, one whole softmax before the V slot)
//   warp 1      tcgen05.mma issuer: S into one of two TMEM buffers, O += P V with P in shared memory
//   warps 2..9  softmax: 64 key columns of a row each; the two threads of a row trade their maxima
//               through shared memory once a tile, keep partial sums of their own and rescale / write
//               their own 64 columns of O
// Its chain from tile to tile is the shorter one; the kernel for pairs overlaps two longer ones and, with one
// head of every pair missing, is left with one of those.  Forward, us, here / there: 1 x 8192 tokens of 1, 8,
// 32 heads 95 / 125, 182 / 236, 745 / 939; 4 x 4096 of 32 796 / 1012; 64 x 256 of 32 219 / 225; 32 x 128 of 32
// 56.2 / 54.5 (one key tile each: set-up alone).
#include <stdio.h>

#include "../common/launch.h"
#include "../common/tensormap.h"
#include "attn_common.cuh"
#include "attn_fwd.h"

namespace lf {

constexpr int ONE_COLS = ATT_TILE / 2;   // key columns of a softmax thread
constexpr int ONE_SOFTMAX_WARPS = 8;
constexpr int ONE_THREADS = 64 + 32 * ONE_SOFTMAX_WARPS;
constexpr int ONE_XCHG_BYTES = 3 * 2 * 128 * 4;   // row maxima (two parities), row sums
constexpr int ONE_SMEM = ATT_TILE_BYTES * (1 + 4 + 1) + 256 + ONE_XCHG_BYTES + 1024;

__global__ void __launch_bounds__(ONE_THREADS, 1)
attn_fwd_one_head_kernel(const AttnFwdParams p, const __grid_constant__ CUtensorMap tm) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + ATT_TILE_BYTES;            // stage s: K at s * 64 KB, V at s * 64 KB + 32 KB
  uint8_t* sP = smem + ATT_TILE_BYTES * 5;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + ATT_TILE_BYTES * 6);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;    // [2]
  uint64_t* k_empty = bars + 3;   // [2]
  uint64_t* v_full = bars + 5;    // [2]
  uint64_t* v_empty = bars + 7;   // [2]
  uint64_t* s_full = bars + 9;    // [2]
  uint64_t* s_empty = bars + 11;  // [2]
  uint64_t* p_full = bars + 13;
  uint64_t* pv_done = bars + 14;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* xchg = reinterpret_cast<float*>(smem + ATT_TILE_BYTES * 6 + 256);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  AbortCtx ctx{p.err, abort_flag};
  // Longest tiles first (the list's order).  Up to eight waves the heads vary fastest, so that the long
  // tiles of the last heads don't start last (1 x 8192 of 8 heads 232 -> 190 us, while a CTA still walked a
  // group); beyond, the tiles do: then a head's K and V stay in L2 (4 x 4096 of 32 heads 886 -> 839 us).
  const bool heads_fastest = p.num_tiles * p.Hkv <= 8 * 148;
  const int h = heads_fastest ? blockIdx.x % p.Hkv : blockIdx.x / p.num_tiles;
  const int4 tile = p.tiles[heads_fastest ? blockIdx.x / p.Hkv : blockIdx.x % p.num_tiles];
  const int row0 = tile.x, rows = tile.y, seq_row0 = tile.z;
  const int n_kv = (row0 - seq_row0) / ATT_TILE + 1;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&s_empty[i], ONE_SOFTMAX_WARPS);  // one arrival per softmax warp
    }
    mbar_init(p_full, ONE_SOFTMAX_WARPS);
    mbar_init(pv_done, 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tm);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS[2] = {tmem_base, tmem_base + 128};
  const uint32_t tO = tmem_base + 256;

  if (warp == 0) {
    if (lane == 0) {
      for (int j = 0; j < n_kv; ++j) {
        const int s = j & 1;
        uint8_t* sK = sKV + s * 2 * ATT_TILE_BYTES;
        if (!mbar_wait<false>(&k_empty[s], ((j >> 1) & 1) ^ 1, ctx, ERR_WAIT_EMPTY)) break;
        mbar_expect_tx(&k_full[s], ATT_TILE_BYTES);
        att_load_tile(sK, &tm, &k_full[s], p.k_col0 + h * ATT_D, seq_row0 + j * ATT_TILE);
        if (j == 0) {
          mbar_expect_tx(q_full, ATT_TILE_BYTES);
          att_load_tile(sQ, &tm, q_full, p.q_col0 + h * ATT_D, row0);
        }
        if (!mbar_wait<false>(&v_empty[s], ((j >> 1) & 1) ^ 1, ctx, ERR_WAIT_EMPTY)) break;
        mbar_expect_tx(&v_full[s], ATT_TILE_BYTES);
        att_load_tile(sK + ATT_TILE_BYTES, &tm, &v_full[s], p.v_col0 + h * ATT_D, seq_row0 + j * ATT_TILE);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      auto issue_s = [&](int j) -> bool {
        const int s = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (!mbar_wait<false>(&k_full[s], ph, ctx, ERR_WAIT_FULL) ||
            !mbar_wait<false>(&s_empty[s], ph ^ 1, ctx, ERR_WAIT_TMEM_EMPTY))
          return false;
        tc_fence_after_sync();
        att_mma_kk(tS[s], smem_u32(sQ), smem_u32(sKV + s * 2 * ATT_TILE_BYTES), false);
        tc_commit(&s_full[s]);
        tc_commit(&k_empty[s]);
        return true;
      };
      bool ok = mbar_wait<false>(q_full, 0, ctx, ERR_WAIT_FULL) && issue_s(0);
      for (int j = 0; ok && j < n_kv; ++j) {
        // S of the next tile goes out before this tile's P V, so that the softmax warps always have a
        // tile waiting (two S buffers in TMEM)
        if (j + 1 < n_kv && !issue_s(j + 1)) break;
        ok = mbar_wait<false>(p_full, j & 1, ctx, ERR_WAIT_READY) &&
             mbar_wait<false>(&v_full[j & 1], (j >> 1) & 1, ctx, ERR_WAIT_FULL);
        if (!ok) break;
        tc_fence_after_sync();
        att_mma_kmn(tO, smem_u32(sP), smem_u32(sKV + (j & 1) * 2 * ATT_TILE_BYTES + ATT_TILE_BYTES), j > 0);
        tc_commit(&v_empty[j & 1]);
        tc_commit(pv_done);
      }
    }
  } else {
    const int q = warp & 3;            // TMEM lane quarter this warp may access
    const int part = (warp - 2) >> 2;  // half of the key columns, and of the columns of O
    const int r = q * 32 + lane;       // row inside the tile
    const int c0 = part * ONE_COLS;
    const uint32_t lane_addr = uint32_t(q * 32) << 16;
    const float c = p.scale_log2e;
    constexpr uint32_t FULL = 0xffffffffu;
    // The two warps that share a row quarter meet in a hardware named barrier (id 1 + q, 64 threads) for
    // the exchange.  `good` is warp-uniform (the tcgen05.ld / st below are .sync.aligned); a failed wait
    // is carried to the next named barrier, whose vote lets both warps leave together (`ok`).
    bool good = true, ok = true;
    float m_ref = -INFINITY, l = 0.f;
    for (int j = 0; j < n_kv; ++j) {
      const int b = j & 1;
      good = __all_sync(FULL, good && mbar_wait<false>(&s_full[b], (j >> 1) & 1, ctx, ERR_WAIT_TMEM_FULL));
      float s[ONE_COLS];
      if (good) {
        tc_fence_after_sync();
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t(&dst)[32] = *reinterpret_cast<uint32_t(*)[32]>(&s[cc * 32]);
          tmem_ld_32x32b_x32(tS[b] + lane_addr + c0 + cc * 32, dst);
        }
        tmem_ld_wait();
        tc_fence_before_sync();
      } else {
#pragma unroll
        for (int col = 0; col < ONE_COLS; ++col) s[col] = 0.f;
      }
      __syncwarp();
      if (lane == 0 && good) mbar_arrive(&s_empty[b]);
      if (j == n_kv - 1) {
#pragma unroll
        for (int col = 0; col < ONE_COLS; ++col)
          if (c0 + col > r) s[col] = -INFINITY;
      }
      // four independent chains each for the maximum and the sum
      float mx4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int col = 4; col < ONE_COLS; ++col) mx4[col & 3] = fmaxf(mx4[col & 3], s[col]);
      float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      xchg[(b * 2 + part) * 128 + r] = mx;
      ok = good = named_bar_and_id(1 + q, 64, good);
      if (!ok) break;
      mx = fmaxf(mx, xchg[(b * 2 + (part ^ 1)) * 128 + r]);
      float alpha = 1.f;
      bool need = false;
      if (j == 0) {
        m_ref = mx;
      } else {
        need = (mx - m_ref) * c > 8.f;
        if (need) {
          alpha = fast_exp2((m_ref - mx) * c);
          m_ref = mx;
          l *= alpha;
        }
      }
      const bool warp_need = __any_sync(FULL, need);
      const float mc = m_ref * c;
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int col = 0; col < ONE_COLS; ++col) {
        s[col] = fast_exp2(s[col] * c - mc);
        sum4[col & 3] += s[col];
      }
      l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
      // P and O belong to the previous tile's P V until it is done
      if (j > 0) good = __all_sync(FULL, mbar_wait<false>(pv_done, (j - 1) & 1, ctx, ERR_WAIT_MISC));
      if (good) {
        tc_fence_after_sync();
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          float(&src)[32] = *reinterpret_cast<float(*)[32]>(&s[cc * 32]);
          att_store_row_chunk(sP, r, c0 + cc * 32, src);
        }
        if (warp_need) {
#pragma unroll 1
          for (int cc = 0; cc < 2; ++cc) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(tO + lane_addr + c0 + cc * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32b_x32(tO + lane_addr + c0 + cc * 32, o);
          }
          tmem_st_wait();
        }
        fence_proxy_async_smem();
        tc_fence_before_sync();
      }
      __syncwarp();
      if (lane == 0 && good) mbar_arrive(p_full);
    }
    // combine the two partial row sums (both relative to the same m_ref), normalise, store
    if (ok) {   // the same for both warps, also where one's last wait has failed
      xchg[(2 * 2 + part) * 128 + r] = l;
      good = named_bar_and_id(1 + q, 64, good);
    }
    if (good) {
      l = xchg[(2 * 2 + 0) * 128 + r] + xchg[(2 * 2 + 1) * 128 + r];   // in the same order for both
      good = __all_sync(FULL, mbar_wait<false>(pv_done, (n_kv - 1) & 1, ctx, ERR_WAIT_MISC));
    }
    if (good) {
      tc_fence_after_sync();
      const float inv_l = 1.f / l;
      const long long grow = (long long)row0 + r;
      __nv_bfloat16* orow = p.out + grow * p.ldo + h * ATT_D + c0;
#pragma unroll 1
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(tO + lane_addr + c0 + cc * 32, o);
        tmem_ld_wait();
        if (r < rows) {
#pragma unroll
          for (int gq = 0; gq < 4; ++gq) {
            st_global_v4(orow + cc * 32 + gq * 8,
                         pack_bf16x2(__uint_as_float(o[gq * 8 + 0]) * inv_l, __uint_as_float(o[gq * 8 + 1]) * inv_l),
                         pack_bf16x2(__uint_as_float(o[gq * 8 + 2]) * inv_l, __uint_as_float(o[gq * 8 + 3]) * inv_l),
                         pack_bf16x2(__uint_as_float(o[gq * 8 + 4]) * inv_l, __uint_as_float(o[gq * 8 + 5]) * inv_l),
                         pack_bf16x2(__uint_as_float(o[gq * 8 + 6]) * inv_l, __uint_as_float(o[gq * 8 + 7]) * inv_l));
          }
        }
        __syncwarp();   // the TMEM load above is .sync.aligned
      }
      if (part == 0 && r < rows) p.lse[(long long)h * p.M_total + grow] = m_ref * p.scale + __logf(l);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

int launch_attn_fwd_one_head(const AttnFwdParams& p, const CUtensorMap& tm, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (ensure_max_dynamic_smem(configured, attn_fwd_one_head_kernel, ONE_SMEM) != cudaSuccess) return -10;
  attn_fwd_one_head_kernel<<<p.num_tiles * p.Hkv, ONE_THREADS, ONE_SMEM, stream>>>(p, tm);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // namespace lf
