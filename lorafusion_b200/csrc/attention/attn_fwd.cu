// Causal, variable-length, grouped-query attention forward for head_dim 128 on sm_100a.
// Replaces the FlashAttention-2 varlen call of the reference
// (lorafusion/patch/patch_transformers.py:150-159).
//
// One CTA handles one 128-row query tile of one sequence for one KV head and walks the query
// heads of that head's group two at a time: the two heads see the same key tiles, so each K / V tile
// is loaded once for both, and while the softmax warps of one head work on their scores the tensor
// pipe runs the products of the other.  (One head at a time, with two threads per row that traded
// row maxima through shared memory and P going through shared memory too, ran at 3.3K cycles
// per key tile: the two sides took turns.  Groups of one head have no pairs and still go that way,
// attn_fwd_one_head.cu.)
//   warp 0      TMA producer: Q of both heads, K and V tiles through two 2-stage rings
//   warp 1      tcgen05.mma issuer: S = Q K^T, then O += P V with P read from tensor memory
//   warps 2..5  softmax of the first head of the pair, one thread per query row; warps 6..9 of the second:
//               read S from TMEM, online max / sum with lazy rescaling of O (only when the running
//               max grows by more than 2^8), write bf16 P over S in TMEM in two halves (the first
//               half of P V starts while the second half is still being exponentiated), normalise.
// TMEM: S / P of both heads (2 x 128 columns), O of both heads (2 x 128).  Tensor instructions of a
// CTA complete in issue order, so "S of the next tile is there" also says "P V of this one is done".
// Q/K/V are read straight out of the packed, RoPE-rotated QKV projection with one tensor
// map; O is written token-major [M, Hq * 128]; the log-sum-exp is kept for the backward.
#include <stdio.h>

#include "../common/launch.h"
#include "../common/tensormap.h"
#include "attn_common.cuh"
#include "attn_fwd.h"

namespace lf {

constexpr int FWD_THREADS = 64 + 256;  // TMA warp, MMA warp, four softmax warps per head of the pair
constexpr int FWD_SMEM = ATT_TILE_BYTES * (2 + 4) + 256 + 1024;

__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_kernel(const AttnFwdParams p, const __grid_constant__ CUtensorMap tm) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint8_t* sQ = smem;                              // head i of the pair at i * 32 KB
  uint8_t* sKV = smem + 2 * ATT_TILE_BYTES;        // stage s: K at s * 64 KB, V at s * 64 KB + 32 KB
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + ATT_TILE_BYTES * 6);
  uint64_t* q_full = bars;          // [2] per head of the pair
  uint64_t* q_empty = bars + 2;     // [2] every S = Q K^T of the head has completed: its Q may be replaced
  uint64_t* k_full = bars + 4;      // [2] per stage
  uint64_t* k_empty = bars + 6;     // [2]
  uint64_t* v_full = bars + 8;      // [2]
  uint64_t* v_empty = bars + 10;    // [2]
  uint64_t* s_full = bars + 12;     // [2] per head of the pair
  uint64_t* p_full = bars + 14;     // [2 heads][2 halves of the key columns]
  uint64_t* o_full = bars + 18;     // [2] the last P V of the head has completed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  AbortCtx ctx{p.err, abort_flag};
  const int4 tile = p.tiles[blockIdx.x / p.Hkv];
  const int row0 = tile.x, rows = tile.y, seq_row0 = tile.z;
  const int g = blockIdx.x % p.Hkv;            // KV head
  const int group = p.Hq / p.Hkv;      // query heads that share it
  const int first_head = 2 * p.pairs_per_cta * int(blockIdx.y);
  const int heads = min(group - first_head, 2 * p.pairs_per_cta);  // of this CTA
  const int h0 = g * group + first_head;
  const int n_pairs = (heads + 1) / 2;
  const int n_kv = (row0 - seq_row0) / ATT_TILE + 1;
  const int total = n_pairs * n_kv;    // the flat (pair, key tile) sequence J = pair * n_kv + j

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[2 * i], 4);      // one arrival per softmax warp of the head
      mbar_init(&p_full[2 * i + 1], 4);
      mbar_init(&o_full[i], 1);
    }
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
  const uint32_t tmem_base = *tmem_slot;   // S / P of head i at 128 i, O at 256 + 128 i

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      for (int pr = 0; ok && pr < n_pairs; ++pr) {
        const int active = min(2, heads - 2 * pr);
        for (int j = 0; j < n_kv; ++j) {
          const int J = pr * n_kv + j;
          const int s = J & 1;
          if (!mbar_wait<false>(&k_empty[s], ((J >> 1) & 1) ^ 1, ctx, ERR_WAIT_EMPTY)) {
            ok = false;
            break;
          }
          uint8_t* sK = sKV + s * 2 * ATT_TILE_BYTES;
          mbar_expect_tx(&k_full[s], ATT_TILE_BYTES);
          att_load_tile(sK, &tm, &k_full[s], p.k_col0 + g * ATT_D, seq_row0 + j * ATT_TILE);
          if (j == 0) {
            for (int i = 0; i < active; ++i) {
              // a head's Q buffer is free once the previous pair's last S product has read it
              if (pr > 0 && !mbar_wait<false>(&q_empty[i], (pr - 1) & 1, ctx, ERR_WAIT_EMPTY)) {
                ok = false;
                break;
              }
              mbar_expect_tx(&q_full[i], ATT_TILE_BYTES);
              att_load_tile(sQ + i * ATT_TILE_BYTES, &tm, &q_full[i], p.q_col0 + (h0 + 2 * pr + i) * ATT_D, row0);
            }
            if (!ok) break;
          }
          if (!mbar_wait<false>(&v_empty[s], ((J >> 1) & 1) ^ 1, ctx, ERR_WAIT_EMPTY)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&v_full[s], ATT_TILE_BYTES);
          att_load_tile(sK + ATT_TILE_BYTES, &tm, &v_full[s], p.v_col0 + g * ATT_D, seq_row0 + j * ATT_TILE);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      auto issue_s = [&](int i, int J) -> bool {   // S of head i for element J of the sequence
        const int pr = J / n_kv, j = J - pr * n_kv;
        if ((j == 0 && !mbar_wait<false>(&q_full[i], pr & 1, ctx, ERR_WAIT_FULL)) ||
            !mbar_wait<false>(&k_full[J & 1], (J >> 1) & 1, ctx, ERR_WAIT_FULL))
          return false;
        tc_fence_after_sync();
        att_mma_kk(tmem_base + 128 * i, smem_u32(sQ + i * ATT_TILE_BYTES), smem_u32(sKV + (J & 1) * 2 * ATT_TILE_BYTES),
                   false);
        tc_commit(&s_full[i]);
        if (i == min(2, heads - 2 * pr) - 1) tc_commit(&k_empty[J & 1]);   // both heads have read this K
        if (j == n_kv - 1) tc_commit(&q_empty[i]);
        return true;
      };
      bool ok = true;
      for (int i = 0; ok && i < min(2, heads); ++i) ok = issue_s(i, 0);
      for (int J = 0; ok && J < total; ++J) {
        const int pr = J / n_kv, j = J - pr * n_kv;
        const int active = min(2, heads - 2 * pr);
        const int active_next = J + 1 < total ? min(2, heads - 2 * ((J + 1) / n_kv)) : 0;
        const uint32_t sV = smem_u32(sKV + (J & 1) * 2 * ATT_TILE_BYTES + ATT_TILE_BYTES);
        for (int i = 0; i < active; ++i) {
          const uint32_t tP = tmem_base + 128 * i, tO = tmem_base + 256 + 128 * i;
          if (!mbar_wait<false>(&p_full[2 * i], J & 1, ctx, ERR_WAIT_READY) ||
              !mbar_wait<false>(&v_full[J & 1], (J >> 1) & 1, ctx, ERR_WAIT_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          att_mma_ts_half(tO, tP, sV, 0, j > 0);
          if (!mbar_wait<false>(&p_full[2 * i + 1], J & 1, ctx, ERR_WAIT_READY)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          att_mma_ts_half(tO, tP, sV, 1, j > 0);
          if (i == active - 1) tc_commit(&v_empty[J & 1]);
          if (j == n_kv - 1) tc_commit(&o_full[i]);
          // S of the next element overwrites P, which the product just issued reads first
          if (i < active_next && !issue_s(i, J + 1)) {
            ok = false;
            break;
          }
        }
      }
    }
  } else {
    const int i = (warp - 2) >> 2;     // head of the pair
    const int q = warp & 3;            // TMEM lane quarter this warp may access
    const int r = q * 32 + lane;       // row inside the tile
    const uint32_t lane_addr = uint32_t(q * 32) << 16;
    const uint32_t tS = tmem_base + 128 * i + lane_addr, tO = tmem_base + 256 + 128 * i + lane_addr;
    const float c = p.scale_log2e;
    constexpr uint32_t FULL = 0xffffffffu;
    // every answer is warp-uniform: the tcgen05.ld / st below are .sync.aligned
    bool ok = true;
    for (int pr = 0; ok && 2 * pr + i < heads; ++pr) {
      const int h = h0 + 2 * pr + i;
      float m_ref = -INFINITY, l = 0.f;
      for (int j = 0; j < n_kv; ++j) {
        const int J = pr * n_kv + j;
        ok = __all_sync(FULL, mbar_wait<false>(&s_full[i], J & 1, ctx, ERR_WAIT_TMEM_FULL));
        if (!ok) break;
        tc_fence_after_sync();
        float s[128];
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t(&dst)[32] = *reinterpret_cast<uint32_t(*)[32]>(&s[cc * 32]);
          tmem_ld_32x32b_x32(tS + cc * 32, dst);
        }
        tmem_ld_wait();
        if (j == n_kv - 1) {
#pragma unroll
          for (int col = 0; col < 128; ++col)
            if (col > r) s[col] = -INFINITY;
        }
        // independent chains for the maximum and the sum: one chain of 128 dependent operations per
        // row would leave the scheduler waiting on fixed latencies
        float mx4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
        for (int col = 4; col < 128; col += 8) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mx4[k] = col + 4 + k < 128 ? fmaxf(fmaxf(mx4[k], s[col + k]), s[col + 4 + k]) : fmaxf(mx4[k], s[col + k]);
        }
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
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
        if (__any_sync(FULL, need)) {
          // (P V of the previous tile is complete: S of this one was issued after it)
#pragma unroll 1
          for (int cc = 0; cc < 4; ++cc) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(tO + cc * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
            tmem_st_32x32b_x32(tO + cc * 32, o);
          }
        }
        const unsigned long long c2 = f32x2(c, c), mc2 = f32x2(-m_ref * c, -m_ref * c);
        unsigned long long sum2[2] = {0ull, 0ull};
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t pk[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            float e0, e1;
            unpack_f32x2(fma_f32x2(f32x2(s[cc * 32 + 2 * k], s[cc * 32 + 2 * k + 1]), c2, mc2), e0, e1);
            e0 = fast_exp2(e0);
            e1 = fast_exp2(e1);
            sum2[k & 1] = add_f32x2(sum2[k & 1], f32x2(e0, e1));
            pk[k] = pack_bf16x2(e0, e1);
          }
          tmem_st_32x32b_x16(tS + cc * 16, pk);
          if (cc & 1) {   // half of P (and the rescaled O) is in place
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[2 * i + (cc >> 1)]);
          }
        }
        float s0, s1;
        unpack_f32x2(add_f32x2(sum2[0], sum2[1]), s0, s1);
        l += s0 + s1;
      }
      if (!ok) break;
      // ---- this head is complete: normalise and store.  The next P V into this O waits for a P that
      // these same warps write afterwards.
      ok = __all_sync(FULL, mbar_wait<false>(&o_full[i], pr & 1, ctx, ERR_WAIT_MISC));
      if (!ok) break;
      tc_fence_after_sync();
      const float inv_l = 1.f / l;
      const long long grow = (long long)row0 + r;
      __nv_bfloat16* orow = p.out + grow * p.ldo + h * ATT_D;
#pragma unroll 1
      for (int cc = 0; cc < 4; ++cc) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(tO + cc * 32, o);
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
      if (r < rows) p.lse[(long long)h * p.M_total + grow] = m_ref * p.scale + __logf(l);
      tc_fence_before_sync();
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

}  // namespace lf

using namespace lf;

// qkv: packed [M, ld_qkv] bf16 (q heads, then k heads, then v heads at the given column
// offsets); tiles: device int32 [num_tiles, 4]; out [M, Hq*128]; lse fp32 [Hq, M].
extern "C" int lf_attn_fwd(const void* qkv, long long M, long long ld_qkv, int q_col0, int k_col0,
                           int v_col0, int Hq, int Hkv, const void* tiles, int num_tiles, void* out,
                           long long ldo, float* lse, float scale, int* err, void* stream) {
  if (num_tiles <= 0) return 0;
  if (Hq % Hkv != 0 || (q_col0 | k_col0 | v_col0) % 64 != 0) return -1;
  CUtensorMap tm;
  int rc = make_tmap_2d_b16(&tm, qkv, (uint64_t)M, (uint64_t)ld_qkv, (uint64_t)ld_qkv, 128, 64, true);
  if (rc != 0) return -20 + rc;
  AttnFwdParams p;
  p.tiles = (const int4*)tiles;
  p.num_tiles = num_tiles;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.q_col0 = q_col0;
  p.k_col0 = k_col0;
  p.v_col0 = v_col0;
  p.out = (__nv_bfloat16*)out;
  p.ldo = ldo;
  p.lse = lse;
  p.M_total = M;
  p.scale = scale;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.err = err;
  if (Hq == Hkv) return launch_attn_fwd_one_head(p, tm, (cudaStream_t)stream);   // no second head to pair with
  static PerDeviceOnce configured;
  if (ensure_max_dynamic_smem(configured, attn_fwd_kernel, FWD_SMEM) != cudaSuccess) return -10;
  // One CTA per (query tile, KV head) walks all head pairs of the group, which pays for its set-up
  // once, unless the launch would leave SMs idle: then the pairs of a group go to CTAs of their own.
  const int pairs = (Hq / Hkv + 1) / 2;
  int parts = 1;
  while (parts < pairs && (long long)num_tiles * Hkv * (parts + 1) <= 148) ++parts;
  p.pairs_per_cta = (pairs + parts - 1) / parts;
  // KV heads vary fastest: the tile list starts with the longest key ranges, and so does the launch.
  dim3 grid(num_tiles * Hkv, (pairs + p.pairs_per_cta - 1) / p.pairs_per_cta);
  attn_fwd_kernel<<<grid, FWD_THREADS, FWD_SMEM, (cudaStream_t)stream>>>(p, tm);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
