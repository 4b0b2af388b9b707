// One call per direction of a LoRA linear layer: the launches of its kernels (lora_skinny.cu,
// umma_gemm_pair.cu, umma_gemm.cu) issued from native code, and the kernels that lay separate
// adapter matrices out as the rank-padded stacks those kernels read and take gradients apart again.
// A layer of 100 tokens spent 120 us on the GPU and 830 us in the Python that described its six
// launches and padded, stacked and cast its adapters with a dozen more.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "gemm_api.h"

namespace lf {
namespace stack {

struct List {
  LfLoraPiece piece[LF_LORA_PIECES];
};

// Pieces of one adapter: A [r, K] -> [R, K] and B [N, r] -> [N, R], zeros in the padding.  grid.y =
// adapter; a thread writes eight bf16 at a time.  Rows of A are copied 16 bytes at a time where the
// source is aligned; B's rows are a few elements long and are gathered.
__global__ void __launch_bounds__(256)
pack_kernel(const List list, __nv_bfloat16* __restrict__ a_out, __nv_bfloat16* __restrict__ b_out, int R, int K, int N) {
  const LfLoraPiece p = list.piece[blockIdx.y];
  const long long a_vec = (long long)R * K / 8, b_vec = (long long)N * R / 8;
  const __nv_bfloat16* a = static_cast<const __nv_bfloat16*>(p.a);
  const __nv_bfloat16* b = static_cast<const __nv_bfloat16*>(p.b);
  const bool aligned = ((reinterpret_cast<uintptr_t>(a) | (uintptr_t)(p.a_ld * 2)) & 15) == 0;
  uint4* ao = reinterpret_cast<uint4*>(a_out + (long long)blockIdx.y * R * K);
  uint4* bo = reinterpret_cast<uint4*>(b_out + (long long)blockIdx.y * N * R);
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < a_vec + b_vec; i += gridDim.x * 256ll) {
    __align__(16) __nv_bfloat16 v[8];
    uint4& v4 = *reinterpret_cast<uint4*>(v);
    v4 = make_uint4(0u, 0u, 0u, 0u);
    if (i < a_vec) {
      const int row = int(i / (K / 8)), col = int(i - (long long)row * (K / 8)) * 8;
      if (row < p.r) {
        const __nv_bfloat16* src = a + row * p.a_ld + col;
        if (aligned) {
          v4 = *reinterpret_cast<const uint4*>(src);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = src[j];
        }
      }
      ao[i] = v4;
    } else {
      const long long k = i - a_vec;
      const long long row = k / (R / 8);
      const int col = int(k - row * (R / 8)) * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (col + j < p.r) v[j] = b[row * p.b_ld + col + j];
      bo[k] = v4;
    }
  }
}

// The other way: fp32 gradient stacks -> contiguous bf16 gradients [r, K] and [N, r] (either may be
// missing).
__global__ void __launch_bounds__(256)
unpack_kernel(const List list, const float* __restrict__ da, const float* __restrict__ db, int R, int K, int N) {
  const LfLoraPiece p = list.piece[blockIdx.y];
  __nv_bfloat16* a = static_cast<__nv_bfloat16*>(const_cast<void*>(p.a));
  __nv_bfloat16* b = static_cast<__nv_bfloat16*>(const_cast<void*>(p.b));
  const long long na = a != nullptr ? (long long)p.r * K : 0, nb = b != nullptr ? (long long)N * p.r : 0;
  const float* sa = da + (long long)blockIdx.y * R * K;
  const float* sb = db + (long long)blockIdx.y * N * R;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < na + nb; i += gridDim.x * 256ll) {
    if (i < na) {
      a[i] = __float2bfloat16(sa[i]);   // the first r rows of the [R, K] stack
    } else {
      const long long k = i - na, row = k / p.r;
      b[k] = __float2bfloat16(sb[row * R + (k - row * p.r)]);
    }
  }
}

static unsigned blocks_for(long long work, int n) {
  const long long want = (work + 255) / 256, cap = (148ll * 8 + n - 1) / n;
  return unsigned(want < 1 ? 1 : (want < cap ? want : cap));
}

}  // namespace stack
}  // namespace lf

extern "C" {

int lf_lora_skinny(const LfGemmArgs* a, int split);
int lf_gemm_pair(const LfGemmArgs* a);

// pieces: n adapters; a_out bf16 [n, R, K], b_out bf16 [n, N, R] (16-byte aligned, K % 8 == 0, R % 8 == 0)
int lf_lora_pack(const LfLoraPiece* pieces, int n, void* a_out, void* b_out, int R, int K, int N, void* stream) {
  if (K % 8 != 0 || R % 8 != 0) return -1;
  for (int first = 0; first < n; first += LF_LORA_PIECES) {
    lf::stack::List list;
    const int m = n - first < LF_LORA_PIECES ? n - first : LF_LORA_PIECES;
    memcpy(list.piece, pieces + first, m * sizeof(LfLoraPiece));
    const long long work = ((long long)R * K + (long long)N * R) / 8;
    lf::stack::pack_kernel<<<dim3(lf::stack::blocks_for(work, m), m), 256, 0, (cudaStream_t)stream>>>(
        list, (__nv_bfloat16*)a_out + (long long)first * R * K, (__nv_bfloat16*)b_out + (long long)first * N * R, R, K, N);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_lora_unpack(const LfLoraPiece* pieces, int n, const float* da, const float* db, int R, int K, int N,
                   void* stream) {
  for (int first = 0; first < n; first += LF_LORA_PIECES) {
    lf::stack::List list;
    const int m = n - first < LF_LORA_PIECES ? n - first : LF_LORA_PIECES;
    memcpy(list.piece, pieces + first, m * sizeof(LfLoraPiece));
    long long work = 0;
    for (int i = 0; i < m; ++i) {
      const long long w = (list.piece[i].a ? (long long)list.piece[i].r * K : 0) +
                          (list.piece[i].b ? (long long)list.piece[i].r * N : 0);
      work = w > work ? w : work;
    }
    if (work == 0) continue;
    lf::stack::unpack_kernel<<<dim3(lf::stack::blocks_for(work, m), m), 256, 0, (cudaStream_t)stream>>>(
        list, da != nullptr ? da + (long long)first * R * K : nullptr, db != nullptr ? db + (long long)first * N * R : nullptr,
        R, K, N);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

static LfGemmArgs base_args(const LfLoraLinearArgs* l) {
  LfGemmArgs g;
  memset(&g, 0, sizeof(g));
  g.err = l->err;
  g.stream = l->stream;
  g.nacc = 1;
  g.scale = 1.f;
  g.inv_keep = 1.f;
  return g;
}
static void set_operand(const void*& p, int64_t& rows, int64_t& cols, int64_t& ld, const void* src, int64_t r, int64_t c,
                        int64_t l) {
  p = src;
  rows = r;
  cols = c;
  ld = l;
}
static void set_dropout(LfGemmArgs& g, const LfLoraLinearArgs* l) {
  g.adapter_thresh16 = l->adapter_thresh16;
  g.adapter_inv_keep = l->adapter_inv_keep;
  g.thresh16 = l->thresh16;
  g.inv_keep = l->inv_keep;
  g.seed_lo = l->seed_lo;
  g.seed_hi = l->seed_hi;
  g.stream_id = l->stream_id;
  g.row_offset = l->row_offset;
  g.col_offset = l->col_offset;
}
static int big_gemm(LfGemmArgs& g, const LfLoraLinearArgs* l) {
  g.scratch = l->scratch;
  g.scratch_bytes = l->scratch_bytes;
  if (l->pair && g.bn == 256) {
    const int rc = lf_gemm_pair(&g);
    if (rc != -5) return rc;
  }
  return lf_gemm(&g);
}

// S' = a * drop(X) A^T (unless the caller has it), Y = X W^T + S' B^T + bias.
int lf_lora_linear_fwd(const LfLoraLinearArgs* l) {
  if (l == nullptr) return -1;
  const int64_t M = l->M, K = l->K, N = l->N, R = l->R, n = l->n_adapters;
  if (!l->have_s) {
    LfGemmArgs g = base_args(l);
    set_operand(g.a, g.a_rows, g.a_cols, g.a_ld, l->x, M, K, l->x_ld);
    set_operand(g.b, g.b_rows, g.b_cols, g.b_ld, l->a_all, n * R, K, l->a_ld);
    g.tile_adapter = l->tile_adapter;
    g.adapter_scale = l->adapter_scale;
    g.scale = l->scale;
    g.out = l->s;
    g.ldo = l->s_ld;
    g.M = int(M);
    g.N = g.bn = g.b_adapter_rows = int(R);
    g.K = int(K);
    g.epi = LF_EPI_BF16_ADAPTER_SCALE;
    g.mask_a = l->dropout;
    set_dropout(g, l);
    const int rc = lf_lora_skinny(&g, l->split_s);
    if (rc != 0) return rc;
  }
  LfGemmArgs g = base_args(l);
  set_operand(g.a, g.a_rows, g.a_cols, g.a_ld, l->x, M, K, l->x_ld);
  set_operand(g.b, g.b_rows, g.b_cols, g.b_ld, l->w, N, K, l->w_ld);
  set_operand(g.a2, g.a2_rows, g.a2_cols, g.a2_ld, l->s, M, R, l->s_ld);
  set_operand(g.b2, g.b2_rows, g.b2_cols, g.b2_ld, l->b_all, n * N, R, l->b_ld);
  g.tile_adapter = l->tile_adapter;
  g.out = l->y;
  g.ldo = N;
  g.bias = l->bias;
  g.M = int(M);
  g.N = g.b2_adapter_rows = int(N);
  g.K = int(K);
  g.K2 = int(R);
  g.bn = N >= 256 ? 256 : 128;
  g.epi = LF_EPI_BF16;
  g.group_m = l->fwd_group_m;
  g.max_ctas = l->fwd_max_ctas;
  return big_gemm(g, l);
}

// dS = a * dY B, then (where asked for) dB += dY^T S', dA += dS^T drop(X) and
// dX = dY W + keep (.) (dS A) / (1 - p).
int lf_lora_linear_bwd(const LfLoraLinearArgs* l) {
  if (l == nullptr) return -1;
  const int64_t M = l->M, K = l->K, N = l->N, R = l->R, n = l->n_adapters;
  int rc;
  {
    LfGemmArgs g = base_args(l);
    set_operand(g.a, g.a_rows, g.a_cols, g.a_ld, l->dy, M, N, l->dy_ld);
    set_operand(g.b, g.b_rows, g.b_cols, g.b_ld, l->b_all, n * N, R, l->b_ld);
    g.tile_adapter = l->tile_adapter;
    g.adapter_scale = l->adapter_scale;
    g.scale = l->scale;
    g.out = l->ds;
    g.ldo = R;
    g.M = int(M);
    g.N = g.bn = int(R);
    g.K = g.b_adapter_rows = int(N);
    g.b_mn = 1;
    g.epi = LF_EPI_BF16_ADAPTER_SCALE;
    if ((rc = lf_lora_skinny(&g, l->split_ds)) != 0) return rc;
  }
  if (l->db != nullptr && l->num_segs > 0) {
    LfGemmArgs g = base_args(l);
    set_operand(g.a, g.a_rows, g.a_cols, g.a_ld, l->dy, M, N, l->dy_ld);
    set_operand(g.b, g.b_rows, g.b_cols, g.b_ld, l->s, M, R, l->s_ld);
    g.seg_tiles = l->seg_rows;
    g.num_seg_tiles = l->num_segs;
    g.out = l->db;
    g.ldo = R;
    g.out_adapter_stride = N * R;
    g.M = int(N);
    g.N = g.bn = int(R);
    g.K = int(M);
    g.a_mn = g.b_mn = 1;
    g.epi = LF_EPI_F32_ACCUM;
    if ((rc = lf_lora_skinny(&g, l->split_db)) != 0) return rc;
  }
  if (l->da != nullptr && l->num_segs > 0) {
    LfGemmArgs g = base_args(l);
    set_operand(g.a, g.a_rows, g.a_cols, g.a_ld, l->x, M, K, l->x_ld);
    set_operand(g.b, g.b_rows, g.b_cols, g.b_ld, l->ds, M, R, R);
    g.seg_tiles = l->seg_rows;
    g.num_seg_tiles = l->num_segs;
    g.out = l->da;
    g.ldo = K;
    g.out_transposed = 1;
    g.out_adapter_stride = R * K;
    g.M = int(K);
    g.N = g.bn = int(R);
    g.K = int(M);
    g.a_mn = g.b_mn = 1;
    g.epi = LF_EPI_F32_ACCUM;
    g.mask_a = l->dropout;
    set_dropout(g, l);
    if ((rc = lf_lora_skinny(&g, l->split_da)) != 0) return rc;
  }
  if (l->dx == nullptr) return 0;
  LfGemmArgs g = base_args(l);
  set_operand(g.a, g.a_rows, g.a_cols, g.a_ld, l->dy, M, N, l->dy_ld);
  set_operand(g.b, g.b_rows, g.b_cols, g.b_ld, l->w, N, K, l->w_ld);
  set_operand(g.a2, g.a2_rows, g.a2_cols, g.a2_ld, l->ds, M, R, R);
  set_operand(g.b2, g.b2_rows, g.b2_cols, g.b2_ld, l->a_all, n * R, K, l->a_ld);
  g.tile_adapter = l->tile_adapter;
  g.out = l->dx;
  g.ldo = K;
  g.M = int(M);
  g.N = int(K);
  g.K = int(N);
  g.K2 = g.b2_adapter_rows = int(R);
  g.b_mn = g.b2_mn = 1;
  g.group_m = l->dx_group_m;
  g.max_ctas = l->dx_max_ctas;
  if (l->dropout) {
    g.bn = K >= 256 ? l->dropmix_bn : 128;
    g.nacc = 2;
    g.epi = LF_EPI_BF16_DROPMIX;
    set_dropout(g, l);
  } else {
    g.bn = K >= 256 ? 256 : 128;
    g.epi = LF_EPI_BF16;
  }
  return big_gemm(g, l);
}

}  // extern "C"
