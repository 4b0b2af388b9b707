// The four skinny products of a LoRA linear layer, each one pass over a token-sized matrix:
//   S'  = a * drop(X) A_a^T      rows of X      x  rank      (bf16 out)     -- reference K1-K3
//   dS  = a * dY B_a             rows of dY     x  rank      (bf16 out)     -- reference K8, K11
//   dB += dY^T S'                columns of dY  x  rank      (fp32 accumulate)
//   dA += dS^T drop(X)           rank x columns of X         (fp32 accumulate)
// (file:line citations of the reference live in lorafusion_b200/ops/lora.py).
//
// The rank is 64 to 256 wide, so the tensor cores are idle most of the time whatever the tiling;
// what bounds these kernels is (a) how many SMs stream the big operand, (b) the Philox rounds of
// the dropout mask (one call per eight elements) and (c) for small batches latency.
//   * Split over the reduction: the C CTAs of a cluster (C = 1, 2, 4 or 8, chosen by the caller)
//     share one 128-row output tile, each sums a slice of the reduction in its own TMEM, and the
//     partial tiles meet over distributed shared memory, every CTA finishing 1 / C of the tile.  The
//     partials are added in rank order, so results do not depend on timing.
//   * Two CTAs per SM (about 100 KB of stages each, at most 256 TMEM columns): one's prologue and
//     epilogue hide behind the other's loads.  One tile per CTA, no persistence: the hardware
//     scheduler evens out segments of different lengths.
//   * The mask warps keep a row (or a column) of the counter fixed while they walk the other
//     index, which leaves nine to ten of the fourteen multiplies of a Philox call, and apply the
//     mask two elements at a time.  After the main loop the same warps are the epilogue.
//   * The fp32 accumulators are read and written 16 bytes (or, transposed, 128 bytes a warp) at a
//     time with all loads of a chunk in flight before the first store.
//
// Roles: warp 0 = TMA producer, warp 1 = TMEM allocator and MMA issuer, warps 2..9 = dropout mask
// on the A stage (MASK only), then epilogue.
#include <stdio.h>

#include "../common/launch.h"
#include "../common/philox.cuh"
#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "gemm_api.h"

namespace lf {
namespace skinny {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int WARPS = 8;                 // mask / epilogue warps
constexpr int THREADS = 64 + 32 * WARPS;
constexpr int PITCH = 68;                // floats per row of a 64-column partial tile: 16-byte
                                         // accesses of eight neighbouring rows hit distinct banks

struct Params {
  int M, K;                    // output rows (tokens, or features with SEG); reduction length (rows mode)
  int tiles_per_seg;           // SEG: 128-feature tiles of one segment
  const int* tile_adapter;     // rows mode: adapter of each 128-row tile, may be null (= 0)
  const int4* segs;            // SEG: {adapter, first token, end token, 0}; null = one segment of all K tokens
  int b_adapter_rows;          // rows mode: rows of B per adapter
  void* out;
  long long ldo, out_adapter_stride;
  int out_vec;                 // SEG, not transposed: whether rows of the output are read and written 16 bytes at a time
  const float* adapter_scale;
  float scale;
  const uint32_t* adapter_thresh16;
  const float* adapter_inv_keep;
  uint32_t thresh16;
  float inv_keep;
  uint32_t seed_lo, seed_hi, stream_id;
  int row_offset, col_offset8;  // col_offset in units of eight columns
  int* err;
};

template <int R>
struct Plan {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = R * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  // as many stages as leave room for two CTAs per SM (227 KB)
  static constexpr int STAGES = R == 64 ? 4 : (R == 128 ? 3 : 2);
  // Mask warps work in groups on different stages: a stage's rewrite is a chain of latencies (barrier,
  // shared-memory load, Philox rounds, store, proxy fence).  The groups divide the stages, so that a
  // group always meets the same ones: it must have seen a stage's previous fill before it waits
  // for the next, or the barrier's parity, two fills back, would let it pass.
  static constexpr int GROUPS = STAGES == 4 ? 4 : (STAGES == 2 ? 2 : 1);
  static_assert(STAGES % GROUPS == 0, "a group would skip fills of a stage");
  static constexpr int GROUP_THREADS = 32 * WARPS / GROUPS;
  static constexpr int TOTAL = STAGES * STAGE_BYTES + 256 + 1024;
  static_assert(BM * PITCH * 4 <= STAGES * STAGE_BYTES, "the partial tile reuses the stages");
  static constexpr uint32_t TMEM = R == 64 ? 64 : (R == 128 ? 128 : 256);
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

// Eight bf16 values times inv_keep, zero where the mask drops them.
__device__ __forceinline__ uint4 mask8(uint4 x, const Philox4& o, uint32_t thresh2, float inv_keep) {
  const uint32_t rnd[4] = {o.x, o.y, o.z, o.w};
  uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16x2(w[j]);
    w[j] = pack_bf16x2(f.x * inv_keep, f.y * inv_keep) & keep_lanes2(rnd[j], thresh2);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// SEG = false: out[M, R] bf16, A K-major [rows, K], B K-major (B_MN = false) or MN-major.
// SEG = true : out fp32 += A^T B over the tokens of a segment, both operands MN-major; TRANS stores
//              out[r][row] instead of out[row][r].
template <int R, bool SEG, bool B_MN, bool MASK, bool TRANS>
__global__ void __launch_bounds__(THREADS, 2)
lora_skinny_kernel(const Params p, const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB) {
  static_assert(!SEG || B_MN, "segment mode reads both operands token-major");
  using P = Plan<R>;
  constexpr int STAGES = P::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * P::STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* ready = empty + STAGES;
  uint64_t* tfull = ready + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  AbortCtx ctx{p.err, abort_flag};
  uint32_t csize, crank;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));

  // ---- which tile, which slice of its reduction ----
  const int tile = blockIdx.x / int(csize);
  int m0, adapter, k_first = 0, nkb;
  if (SEG) {
    const int sgi = tile / p.tiles_per_seg;
    const int4 sg = p.segs != nullptr ? p.segs[sgi] : make_int4(0, 0, p.K, 0);
    m0 = (tile - sgi * p.tiles_per_seg) * BM;
    adapter = sg.x;
    k_first = sg.y;
    nkb = (sg.z - sg.y + BK - 1) / BK;
  } else {
    m0 = tile * BM;
    adapter = p.tile_adapter != nullptr ? p.tile_adapter[tile] : 0;
    nkb = adapter >= 0 ? (p.K + BK - 1) / BK : 0;
  }
  const int kb0 = int((long long)nkb * crank / csize), kb1 = int((long long)nkb * (crank + 1) / csize);
  const int n = kb1 - kb0;
  const int kbase = k_first + kb0 * BK;
  const int b_row0 = (!SEG && adapter >= 0) ? adapter * p.b_adapter_rows : 0;
  float scale = p.scale;
  if (!SEG && p.adapter_scale != nullptr) scale = adapter >= 0 ? p.adapter_scale[adapter] : 0.f;
  uint32_t thresh = p.thresh16;
  float inv_keep = p.inv_keep;
  if (MASK && adapter >= 0 && p.adapter_thresh16 != nullptr) {
    thresh = p.adapter_thresh16[adapter];
    inv_keep = p.adapter_inv_keep[adapter];
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
      mbar_init(&ready[s], WARPS / P::GROUPS);
    }
    mbar_init(tfull, 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, P::TMEM);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      for (int it = 0; it < n; ++it) {
        const int s = it % STAGES;
        if (!mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, ctx, ERR_WAIT_EMPTY)) break;
        uint8_t* sA = smem + s * P::STAGE_BYTES;
        uint8_t* sB = sA + P::A_BYTES;
        const int kk = kbase + it * BK;
        mbar_expect_tx(&full[s], P::STAGE_BYTES);
        if (SEG) {
          tma_load_2d(sA, &tmA, &full[s], m0, kk);
          tma_load_2d(sA + 8192, &tmA, &full[s], m0 + 64, kk);
        } else {
          tma_load_2d(sA, &tmA, &full[s], kk, m0);
        }
        if (B_MN) {
#pragma unroll
          for (int h = 0; h < R / 64; ++h) tma_load_2d(sB + h * 8192, &tmB, &full[s], 64 * h, b_row0 + kk);
        } else {
          tma_load_2d(sB, &tmB, &full[s], kk, b_row0);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t IDESC = make_idesc_bf16(BM, R, SEG ? 1 : 0, B_MN ? 1 : 0);
      bool good = true;
      for (int it = 0; it < n; ++it) {
        const int s = it % STAGES;
        good = mbar_wait(MASK ? &ready[s] : &full[s], (it / STAGES) & 1, ctx, MASK ? ERR_WAIT_READY : ERR_WAIT_FULL);
        if (!good) break;
        tc_fence_after_sync();
        const uint32_t sA = smem_u32(smem + s * P::STAGE_BYTES);
        const uint32_t sB = sA + P::A_BYTES;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) {
          const uint64_t da = SEG ? make_smem_desc_sw128(sA + kk * 2048, 8192, 1024)
                                  : make_smem_desc_sw128(sA + kk * 32, 16, 1024);
          const uint64_t db = B_MN ? make_smem_desc_sw128(sB + kk * 2048, 8192, 1024)
                                   : make_smem_desc_sw128(sB + kk * 32, 16, 1024);
          umma_bf16_ss(tmem_base, da, db, IDESC, uint32_t(it > 0 || kk > 0));
        }
        tc_commit(&empty[s]);
      }
      if (good && n > 0) tc_commit(tfull);
    }
  } else {
    if (MASK) {
      constexpr int GT = P::GROUP_THREADS, CHUNKS = 1024 / GT;   // 16-byte chunks of a stage per thread
      const int grp = (threadIdx.x - 64) / GT;
      const int mt = (threadIdx.x - 64) % GT;
      const uint32_t thresh2 = thresh | (thresh << 16);
      // Rows mode: with 64 threads a thread owns tile rows mt and mt + 64 for the whole reduction, with
      // more it owns (part of) row mt % 128.  SEG: (part of) token row mt % 64 of a stage.
      constexpr int ROWS = SEG || GT > 64 ? 1 : 2;
      const int own = SEG ? mt & 63 : mt & 127;
      const int first = SEG ? (mt >> 6) * CHUNKS : (mt >> 7) * CHUNKS;   // of the own row's chunks
      PhiloxRow pr[ROWS];
      if (!SEG) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
          pr[i] = philox_row(uint32_t(m0 + own + 64 * i + p.row_offset), p.stream_id, p.seed_lo, p.seed_hi);
      }
      for (int it = grp; it < n; it += P::GROUPS) {
        const int s = it % STAGES;
        // one answer per warp: its lanes meet again in __syncwarp below
        ok = __all_sync(0xffffffffu, mbar_wait(&full[s], (it / STAGES) & 1, ctx, ERR_WAIT_FULL));
        if (!ok) break;
        if (thresh != 0) {
          uint8_t* sA = smem + s * P::STAGE_BYTES;
          const int kk = kbase + it * BK;
          if (SEG) pr[0] = philox_row(uint32_t(kk + own + p.row_offset), p.stream_id, p.seed_lo, p.seed_hi);
          const uint32_t col0 = uint32_t(((SEG ? m0 : kk) >> 3) + p.col_offset8);
#pragma unroll 4
          for (int j = 0; j < CHUNKS; ++j) {
            const int i = j % ROWS;                 // which of the own rows
            const int c = first + j / ROWS;         // chunk of that row; SEG: 0..15 over both panels
            const int panel = SEG ? c >> 3 : 0, row = own + 64 * i;
            uint4* ptr = reinterpret_cast<uint4*>(sA + panel * 8192 + row * 128 + (((c & 7) ^ (row & 7)) << 4));
            const Philox4 o = philox_rest(pr[i], philox_col(col0 + uint32_t(c), p.stream_id, p.seed_lo), p.seed_lo,
                                          p.seed_hi);
            // a threshold past 16 bits drops every element
            *ptr = thresh > 0xffffu ? make_uint4(0u, 0u, 0u, 0u) : mask8(*ptr, o, thresh2, inv_keep);
          }
          fence_proxy_async_smem();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ready[s]);
      }
    }
    if (n > 0) {
      ok = __all_sync(0xffffffffu, ok && mbar_wait(tfull, 0, ctx, ERR_WAIT_TMEM_FULL));
      tc_fence_after_sync();
    }
  }
  __syncwarp();

  // ---- epilogue: 64 columns at a time; warp w reads TMEM lane quarter w % 4, and of the 64 columns
  // the first half (warps 2..5) or the second ----
  const int q = warp & 3, half = (warp - 2) >> 2;
  const int trow = q * 32 + lane;
  const uint32_t taddr = tmem_base + (uint32_t(q * 32) << 16) + half * 32;
  float* out_f32 = reinterpret_cast<float*>(p.out) + (adapter >= 0 ? adapter * p.out_adapter_stride : 0);
  __nv_bfloat16* out_bf16 = reinterpret_cast<__nv_bfloat16*>(p.out);
  const uint32_t stage_addr = smem_u32(smem);
  if (csize == 1) {
    if (warp >= 2 && ok) {
#pragma unroll 1
      for (int c = 0; c < R / 64; ++c) {
        uint32_t r[32];
        if (n > 0) {
          tmem_ld_32x32b_x32(taddr + c * 64, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
        const int row = m0 + trow, col0 = c * 64 + half * 32;
        if (row < p.M) {
          if (!SEG) {
            __nv_bfloat16* dst = out_bf16 + (long long)row * p.ldo + col0;
#pragma unroll
            for (int g = 0; g < 4; ++g)
              st_global_v4(dst + g * 8,
                           pack_bf16x2(__uint_as_float(r[g * 8 + 0]) * scale, __uint_as_float(r[g * 8 + 1]) * scale),
                           pack_bf16x2(__uint_as_float(r[g * 8 + 2]) * scale, __uint_as_float(r[g * 8 + 3]) * scale),
                           pack_bf16x2(__uint_as_float(r[g * 8 + 4]) * scale, __uint_as_float(r[g * 8 + 5]) * scale),
                           pack_bf16x2(__uint_as_float(r[g * 8 + 6]) * scale, __uint_as_float(r[g * 8 + 7]) * scale));
          } else if (!TRANS && !p.out_vec) {
            float* dst = out_f32 + (long long)row * p.ldo + col0;
#pragma unroll
            for (int j = 0; j < 32; ++j) dst[j] = fmaf(scale, __uint_as_float(r[j]), dst[j]);
          } else if (!TRANS) {
            float4* dst = reinterpret_cast<float4*>(out_f32 + (long long)row * p.ldo + col0);
            float4 old[8];
#pragma unroll
            for (int g = 0; g < 8; ++g) old[g] = dst[g];
#pragma unroll
            for (int g = 0; g < 8; ++g)
              dst[g] = make_float4(fmaf(scale, __uint_as_float(r[g * 4 + 0]), old[g].x),
                                   fmaf(scale, __uint_as_float(r[g * 4 + 1]), old[g].y),
                                   fmaf(scale, __uint_as_float(r[g * 4 + 2]), old[g].z),
                                   fmaf(scale, __uint_as_float(r[g * 4 + 3]), old[g].w));
          } else {
            float* dst = out_f32 + (long long)col0 * p.ldo + row;
#pragma unroll
            for (int g = 0; g < 2; ++g) {   // sixteen loads in flight: thirty-two did not fit the registers
              float old[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) old[j] = dst[(long long)(g * 16 + j) * p.ldo];
#pragma unroll
              for (int j = 0; j < 16; ++j)
                dst[(long long)(g * 16 + j) * p.ldo] = fmaf(scale, __uint_as_float(r[g * 16 + j]), old[j]);
            }
          }
        }
        // whole again before the next chunk: the TMEM load is .sync.aligned
        __syncwarp();
      }
    }
  } else {
#pragma unroll 1
    for (int c = 0; c < R / 64; ++c) {
      if (warp >= 2) {
        uint32_t r[32];
        if (n > 0 && ok) {
          tmem_ld_32x32b_x32(taddr + c * 64, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
        // every load into the stages and every MMA that reads them has completed (tfull)
        float4* st = reinterpret_cast<float4*>(smem) + (trow * PITCH + half * 32) / 4;
#pragma unroll
        for (int g = 0; g < 8; ++g)
          st[g] = make_float4(__uint_as_float(r[g * 4]), __uint_as_float(r[g * 4 + 1]), __uint_as_float(r[g * 4 + 2]),
                              __uint_as_float(r[g * 4 + 3]));
      }
      __syncwarp();
      cluster_arrive();
      cluster_wait();
      if (warp >= 2 && !aborted(ctx)) {
        // this CTA finishes 128 / C rows of the 64 columns, or (TRANS) 64 / C columns of all rows
        const int t = threadIdx.x - 64;
        const int items = BM * 16 / int(csize);
        for (int i = t; i < items; i += 32 * WARPS) {
          int srow, c4;
          if (!TRANS) {
            srow = int(crank) * (BM / int(csize)) + i / 16;
            c4 = i % 16;
          } else {
            srow = i % BM;
            c4 = int(crank) * (16 / int(csize)) + i / BM;
          }
          const uint32_t off = stage_addr + uint32_t(srow * PITCH + c4 * 4) * 4u;
          float4 part[8];
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) {
            if (k < csize) {
              uint32_t addr;
              asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(off), "r"(k));
              part[k] = ld_cluster_f4(addr);
            }
          }
          float4 v = part[0];
#pragma unroll
          for (uint32_t k = 1; k < 8; ++k) {
            if (k < csize) {
              v.x += part[k].x;
              v.y += part[k].y;
              v.z += part[k].z;
              v.w += part[k].w;
            }
          }
          const int row = m0 + srow, col = c * 64 + c4 * 4;
          if (row >= p.M) continue;
          if (!SEG) {
            uint2 w;
            w.x = pack_bf16x2(v.x * scale, v.y * scale);
            w.y = pack_bf16x2(v.z * scale, v.w * scale);
            *reinterpret_cast<uint2*>(out_bf16 + (long long)row * p.ldo + col) = w;
          } else if (!TRANS && !p.out_vec) {
            float* dst = out_f32 + (long long)row * p.ldo + col;
            dst[0] = fmaf(scale, v.x, dst[0]);
            dst[1] = fmaf(scale, v.y, dst[1]);
            dst[2] = fmaf(scale, v.z, dst[2]);
            dst[3] = fmaf(scale, v.w, dst[3]);
          } else if (!TRANS) {
            float4* dst = reinterpret_cast<float4*>(out_f32 + (long long)row * p.ldo + col);
            const float4 o = *dst;
            *dst = make_float4(fmaf(scale, v.x, o.x), fmaf(scale, v.y, o.y), fmaf(scale, v.z, o.z), fmaf(scale, v.w, o.w));
          } else {
            float* dst = out_f32 + (long long)col * p.ldo + row;
            const float o0 = dst[0], o1 = dst[p.ldo], o2 = dst[2 * p.ldo], o3 = dst[3 * p.ldo];
            dst[0] = fmaf(scale, v.x, o0);
            dst[p.ldo] = fmaf(scale, v.y, o1);
            dst[2 * p.ldo] = fmaf(scale, v.z, o2);
            dst[3 * p.ldo] = fmaf(scale, v.w, o3);
          }
        }
      }
      // nobody overwrites its partial tile, or leaves, while a peer may still read it
      __syncwarp();
      cluster_arrive();
      cluster_wait();
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
    tmem_dealloc(tmem_base, P::TMEM);
  }
}

template <int R, bool SEG, bool B_MN, bool MASK, bool TRANS>
static int launch(const Params& p, const CUtensorMap& tA, const CUtensorMap& tB, int tiles, int split, cudaStream_t st) {
  auto kern = lora_skinny_kernel<R, SEG, B_MN, MASK, TRANS>;
  static PerDeviceOnce configured;  // one per template instantiation
  if (ensure_max_dynamic_smem(configured, kern, Plan<R>::TOTAL) != cudaSuccess) return -10;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(tiles) * unsigned(split));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = Plan<R>::TOTAL;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(split);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p, tA, tB);
  if (e != cudaSuccess) {
    fprintf(stderr, "lf_lora_skinny: launch failed: %s\n", cudaGetErrorString(e));
    return -11;
  }
  return 0;
}

template <int R>
static int dispatch(const LfGemmArgs* a, const Params& p, const CUtensorMap& tA, const CUtensorMap& tB, int tiles,
                    int split, cudaStream_t st) {
  if (a->a_mn) {
    if (!a->out_transposed) return a->mask_a ? -5 : launch<R, true, true, false, false>(p, tA, tB, tiles, split, st);
    return a->mask_a ? launch<R, true, true, true, true>(p, tA, tB, tiles, split, st)
                     : launch<R, true, true, false, true>(p, tA, tB, tiles, split, st);
  }
  if (a->b_mn) return a->mask_a ? -5 : launch<R, false, true, false, false>(p, tA, tB, tiles, split, st);
  return a->mask_a ? launch<R, false, false, true, false>(p, tA, tB, tiles, split, st)
                   : launch<R, false, false, false, false>(p, tA, tB, tiles, split, st);
}

}  // namespace skinny
}  // namespace lf

// LfGemmArgs of the skinny products: N = bn = padded rank.  a_mn = 0: epi LF_EPI_BF16_ADAPTER_SCALE,
// A [M, K] K-major, adapters per 128-row tile.  a_mn = 1: epi LF_EPI_F32_ACCUM, `seg_tiles` holds
// num_seg_tiles rows int4 {adapter, first token, end token, 0} (adapter >= 0, non-empty; null with one
// row = adapter 0, tokens 0 to K), M = features.
// `split` = CTAs that share a tile's reduction (1, 2, 4 or 8).
extern "C" int lf_lora_skinny(const LfGemmArgs* a, int split) {
  using namespace lf;
  using namespace lf::skinny;
  if (a == nullptr || a->a == nullptr || a->b == nullptr || a->out == nullptr) return -1;
  if (a->N != a->bn || a->K2 != 0 || a->nacc != 1) return -2;
  if (split != 1 && split != 2 && split != 4 && split != 8) return -3;
  if (a->a_mn ? (a->epi != LF_EPI_F32_ACCUM || (a->seg_tiles == nullptr && a->num_seg_tiles != 1) || !a->b_mn)
              : (a->epi != LF_EPI_BF16_ADAPTER_SCALE || a->seg_tiles != nullptr))
    return -4;
  // 16-byte accesses to the output (columns of a row, or 8-byte pieces of it); fp32 rows that lie elsewhere are
  // gone through value by value
  const bool aligned = (reinterpret_cast<uintptr_t>(a->out) & 15) == 0;
  if (!a->a_mn && (!aligned || a->ldo % 8 != 0)) return -6;
  CUtensorMap tA, tB;
  int rc = make_tmap_2d_b16(&tA, a->a, a->a_rows, a->a_cols, a->a_ld, a->a_mn ? 64 : BM, 64, true);
  if (rc != 0) return -20 + rc;
  rc = make_tmap_2d_b16(&tB, a->b, a->b_rows, a->b_cols, a->b_ld, a->b_mn ? 64 : a->bn, 64, true);
  if (rc != 0) return -30 + rc;
  Params p;
  p.M = a->M;
  p.K = a->K;
  p.tiles_per_seg = (a->M + BM - 1) / BM;
  p.tile_adapter = a->tile_adapter;
  p.segs = reinterpret_cast<const int4*>(a->seg_tiles);
  p.b_adapter_rows = a->b_adapter_rows;
  p.out = a->out;
  p.ldo = a->ldo;
  p.out_adapter_stride = a->out_adapter_stride;
  p.out_vec = aligned && a->ldo % 4 == 0 && a->out_adapter_stride % 4 == 0;
  p.adapter_scale = a->adapter_scale;
  p.scale = a->scale;
  p.adapter_thresh16 = a->adapter_thresh16;
  p.adapter_inv_keep = a->adapter_inv_keep;
  p.thresh16 = a->thresh16;
  p.inv_keep = a->inv_keep;
  p.seed_lo = a->seed_lo;
  p.seed_hi = a->seed_hi;
  p.stream_id = a->stream_id;
  p.row_offset = a->row_offset;
  p.col_offset8 = a->col_offset >> 3;
  p.err = a->err;
  const int tiles = a->a_mn ? p.tiles_per_seg * a->num_seg_tiles : p.tiles_per_seg;
  if (tiles <= 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);
  switch (a->bn) {
    case 64: return dispatch<64>(a, p, tA, tB, tiles, split, st);
    case 128: return dispatch<128>(a, p, tA, tB, tiles, split, st);
    case 192: return dispatch<192>(a, p, tA, tB, tiles, split, st);
    case 256: return dispatch<256>(a, p, tA, tB, tiles, split, st);
    default: return -2;
  }
}
