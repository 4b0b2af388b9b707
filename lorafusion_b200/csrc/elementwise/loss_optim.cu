// Cross-entropy over a chunk of logits (loss + in-place gradient) and the multi-tensor
// Adam step for LoRA adapters.
//
// Cross-entropy: the lm_head GEMM is run chunk by chunk over tokens so that the
// [tokens, vocab] logits never exist in full; this kernel turns one bf16 logits chunk into
// per-token losses and overwrites it with d(loss)/d(logits), which the next GEMM multiplies
// by the lm_head weight.  (The reference goes through HF's lm_head + torch cross-entropy,
// lorafusion/pipeline_parallel/pipe_module.py:218-221.)
//
// Adam: one launch updates every LoRA tensor of one adapter.  Tensors are described by a
// chunk table (offset, length) into parallel arenas: fp32 gradient, fp32 master weight,
// fp32 m, fp32 v and the bf16 working copy the GEMM kernels read.  The gradient arena is
// zeroed as it is consumed.  (The reference uses torch.optim.AdamW(fused=True) per adapter,
// benchmarks_paper/bench_multi_gpu.py:225-230.)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "../common/ptx.cuh"

namespace lf {

constexpr int CE_VECS = 4;   // 16-byte vectors in flight a thread

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum2(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// e^x of two packed bf16 logits relative to a maximum.
__device__ __forceinline__ unsigned long long exp_pair(uint32_t w, unsigned long long neg_m2, unsigned long long log2e2) {
  const float2 f = unpack_bf16x2(w);
  float a, b;
  unpack_f32x2(mul_f32x2(add_f32x2(f32x2(f.x, f.y), neg_m2), log2e2), a, b);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(b));
  return f32x2(a, b);
}

// One CTA per token.  Pass 1: online max / sum-exp.  Pass 2: write the gradient in place.  Two
// exponentials a logit keep the special-function units busy for 117 us of 2048 rows of 128256, next
// to 158 us of memory traffic, so the rest of the arithmetic is done two logits at a time, the label's
// column apart, and four vectors of a thread are in flight: 265 -> 233 us (either alone gave nothing,
// nor did keeping part of the row in shared memory instead of reading it twice).
// Rows of at most 4096 logits, one batch of vectors of 128 threads, get CTAs of that size: they wait for
// memory and for one another most of the time, and of the larger CTAs, whose registers leave room for
// three on an SM instead of four, too few are resident (2048 rows of 64, 1000, 4096: 5.6, 5.8, 8.7 us, and
// 14.3, 14.3, 17.5 us in CTAs of 512).
// labels < 0 are ignored (loss 0, gradient 0).  A label of V or more, which the embedding would clamp, has
// no column: the gradient is that of the log-sum-exp alone, the loss takes the last column's logit, and
// nothing outside the row's V columns is touched.  grad_scale multiplies the gradient
// (1 / number of valid tokens for a mean loss).
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
cross_entropy_kernel(__nv_bfloat16* __restrict__ logits, const int* __restrict__ labels,
                     float* __restrict__ loss_out, int V, long long ld, float grad_scale) {
  __shared__ float red_m[THREADS / 32];
  __shared__ float red_s[THREADS / 32];
  const long long row = blockIdx.x;
  __nv_bfloat16* lr = logits + row * ld;
  const int label = labels[row];
  const int nvec = V / 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (label < 0) {
    const uint4 z = make_uint4(0, 0, 0, 0);
    for (int c = threadIdx.x; c < nvec; c += THREADS) reinterpret_cast<uint4*>(lr)[c] = z;
    for (int c = nvec * 8 + threadIdx.x; c < V; c += THREADS) lr[c] = __float2bfloat16(0.f);
    if (threadIdx.x == 0) loss_out[row] = 0.f;
    return;
  }

  const unsigned long long log2e2 = f32x2(1.4426950408889634f, 1.4426950408889634f);
  // The maximum starts below every finite bf16, not at -inf: a logit of -inf (masked) then weighs
  // 2^-inf = 0, also in front of the first finite one of its thread, where -inf - -inf would be NaN.
  float m = -FLT_MAX, s = 0.f;
  for (int c0 = threadIdx.x; c0 < nvec; c0 += CE_VECS * THREADS) {
    uint4 raw[CE_VECS];
#pragma unroll
    for (int k = 0; k < CE_VECS; ++k)
      if (c0 + k * THREADS < nvec) raw[k] = reinterpret_cast<const uint4*>(lr)[c0 + k * THREADS];
#pragma unroll
    for (int k = 0; k < CE_VECS; ++k) {
      if (c0 + k * THREADS >= nvec) continue;
      const uint32_t w[4] = {raw[k].x, raw[k].y, raw[k].z, raw[k].w};
      // the maximum of bf16 values is one of them: taken on packed pairs
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(w);
      const __nv_bfloat162 m2 = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
      const float lm = fmaxf(__low2float(m2), __high2float(m2));
      if (lm > m) {
        s *= __expf(m - lm);
        m = lm;
      }
      const unsigned long long neg_m2 = f32x2(-m, -m);
      unsigned long long sum = 0ull;
#pragma unroll
      for (int j = 0; j < 4; ++j) sum = add_f32x2(sum, exp_pair(w[j], neg_m2, log2e2));
      float s0, s1;
      unpack_f32x2(sum, s0, s1);
      s += s0 + s1;
    }
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += THREADS) {
    const float f = __bfloat162float(lr[c]);
    if (f > m) {
      s *= __expf(m - f);
      m = f;
    }
    s += __expf(f - m);
  }
  // block reduce (max, then rescaled sums)
  float wm = warp_max(m);
  s = m == -FLT_MAX ? 0.f : s * __expf(m - wm);  // threads that saw no finite logit
  s = warp_sum2(s);
  if (lane == 0) {
    red_m[warp] = wm;
    red_s[warp] = s;
  }
  __syncthreads();
  float bm = red_m[0];
  for (int i = 1; i < THREADS / 32; ++i) bm = fmaxf(bm, red_m[i]);
  float bs = 0.f;
  for (int i = 0; i < THREADS / 32; ++i)
    bs += (red_m[i] == -FLT_MAX) ? 0.f : red_s[i] * __expf(red_m[i] - bm);
  const float lse = bm + __logf(bs);
  const float inv_sum = 1.f / bs, scale = inv_sum * grad_scale;
  const float label_logit = __bfloat162float(lr[min(label, V - 1)]);
  __syncthreads();  // everyone has read the label's logit before it is overwritten
  float* label_grad = red_m;   // kept there by thread 0: in a register it would be spilled over the second pass
  if (threadIdx.x == 0) {
    loss_out[row] = lse - label_logit;
    *label_grad = (__expf(label_logit - bm) * inv_sum - 1.f) * grad_scale;
  }

  const unsigned long long neg_bm2 = f32x2(-bm, -bm), scale2 = f32x2(scale, scale);
  for (int c0 = threadIdx.x; c0 < nvec; c0 += CE_VECS * THREADS) {
    uint4 raw[CE_VECS];
#pragma unroll
    for (int k = 0; k < CE_VECS; ++k)
      if (c0 + k * THREADS < nvec) raw[k] = reinterpret_cast<const uint4*>(lr)[c0 + k * THREADS];
#pragma unroll
    for (int k = 0; k < CE_VECS; ++k) {
      if (c0 + k * THREADS >= nvec) continue;
      uint32_t w[4] = {raw[k].x, raw[k].y, raw[k].z, raw[k].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float g0, g1;
        unpack_f32x2(mul_f32x2(exp_pair(w[j], neg_bm2, log2e2), scale2), g0, g1);
        w[j] = pack_bf16x2(g0, g1);
      }
      reinterpret_cast<uint4*>(lr)[c0 + k * THREADS] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += THREADS) {
    const float f = __bfloat162float(lr[c]);
    lr[c] = __float2bfloat16(__expf(f - bm) * scale);
  }
  __syncthreads();
  // the label's column, which the loops above treated like any other
  // (patching it into its vector on the way cost 7 % at V = 50257: one more comparison a vector)
  if (threadIdx.x == 0 && label < V) lr[label] = __float2bfloat16(*label_grad);
}

// ---------------------------------------------------------------------------------
// Adam / AdamW over a chunk table.
// ---------------------------------------------------------------------------------
// A chunk is a 2-D region of `rows` x `ld` elements starting at `offset` in every arena.
// Its gradient is always cleared; only columns [col0, col0 + cols) of each row are
// trainable (block-diagonal B matrices of merged projections keep their off-diagonal
// blocks at zero this way).  A flat tensor is rows = 1, ld = cols = length, col0 = 0.
// `grad` and `work` use the padded layout (`offset`); master / m / v hold the trainable
// elements only, densely: element (row, col) lives at state + row * cols + (col - col0).
struct AdamChunk {
  long long offset;
  long long rows;
  long long ld;
  long long col0;
  long long cols;
  long long state;
};

struct AdamHyper {
  float lr, beta1, beta2, eps, weight_decay;
  float bias_c1, bias_c2;  // 1 - beta1^t, 1 - beta2^t
  float grad_scale;        // multiplies the accumulated gradient before the update
};

__device__ __forceinline__ void adam_one(float g, float& w, float& mi, float& vi, const AdamHyper& h,
                                         float inv_c1, float inv_sqrt_c2) {
  mi = h.beta1 * mi + (1.f - h.beta1) * g;
  vi = h.beta2 * vi + (1.f - h.beta2) * g * g;
  w -= h.lr * h.weight_decay * w;
  w -= h.lr * (mi * inv_c1) / (sqrtf(vi) * inv_sqrt_c2 + h.eps);
}

// A work item {chunk, first element, element count} is what kAdamShares CTAs share: regions differ in
// size by two orders of magnitude (a 16 x 8192 A block next to a 57344 x 64 B block), so the host cuts
// them into equal pieces instead of giving every region the same number of CTAs.  Regions
// whose offsets and sizes are all multiples of four elements (every region the adapter arenas
// produce) go through 16-byte accesses with 32-bit index arithmetic; anything else takes the
// scalar path.
struct AdamWorkItem {
  int chunk;
  unsigned first, count;  // elements; multiples of 4 inside vectorisable regions
};

// Bound by latency unless every load of a thread is issued before its first use: an item is shared by
// kAdamShares neighbouring CTAs, and a thread loads gradient, weight and moments of its two pieces
// first (padding is not read at all).  The 86 MB of a two-layer 8B adapter take 34 us (2.5 TB/s); one
// CTA an item, whose threads walked 32 pieces one after the other, took 267 us, and sixteen CTAs an
// item with two pieces one after the other 152 us.
constexpr unsigned kAdamShares = 16;

__global__ void __launch_bounds__(256)
adam_chunks_kernel(const AdamChunk* __restrict__ chunks, const AdamWorkItem* __restrict__ items,
                   float* __restrict__ grad, float* __restrict__ master, float* __restrict__ m,
                   float* __restrict__ v, __nv_bfloat16* __restrict__ work, AdamHyper h) {
  const AdamWorkItem item = items[blockIdx.x / kAdamShares];
  const unsigned first = (blockIdx.x % kAdamShares) * 256u + threadIdx.x;   // of the shares, neighbours first
  const AdamChunk c = chunks[item.chunk];
  const float inv_c1 = 1.f / h.bias_c1;
  const float inv_sqrt_c2 = rsqrtf(h.bias_c2);
  const long long total = c.rows * c.ld;
  const bool vec = (((c.offset | c.ld | c.col0 | c.cols | c.state) & 3) == 0) && total < (1ll << 31) &&
                   ((item.first | item.count) & 3u) == 0;
  if (vec) {
    float4* g4p = reinterpret_cast<float4*>(grad + c.offset);
    const unsigned ld = unsigned(c.ld), col0 = unsigned(c.col0), cols = unsigned(c.cols);
    const unsigned end4 = (item.first + item.count) >> 2;
    constexpr int U = 2;   // pieces in flight: 32768-element items are done in one go
    for (unsigned i0 = (item.first >> 2) + first; i0 < end4; i0 += U * 256u * kAdamShares) {
      float4 g[U], w4[U], m4[U], v4[U];
      long long se[U];
      bool live[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const unsigned i4 = i0 + k * 256u * kAdamShares;
        live[k] = false;
        if (i4 < end4) {
          const unsigned e = i4 << 2;
          const unsigned row = e / ld;
          const unsigned col = e - row * ld;
          live[k] = cols != 0 && col >= col0 && col < col0 + cols;   // padding is cleared only
          se[k] = c.state + (long long)row * cols + (col - col0);
          if (live[k]) {
            g[k] = g4p[i4];
            w4[k] = *reinterpret_cast<const float4*>(master + se[k]);
            m4[k] = *reinterpret_cast<const float4*>(m + se[k]);
            v4[k] = *reinterpret_cast<const float4*>(v + se[k]);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const unsigned i4 = i0 + k * 256u * kAdamShares;
        if (i4 < end4) g4p[i4] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!live[k]) continue;
        adam_one(g[k].x * h.grad_scale, w4[k].x, m4[k].x, v4[k].x, h, inv_c1, inv_sqrt_c2);
        adam_one(g[k].y * h.grad_scale, w4[k].y, m4[k].y, v4[k].y, h, inv_c1, inv_sqrt_c2);
        adam_one(g[k].z * h.grad_scale, w4[k].z, m4[k].z, v4[k].z, h, inv_c1, inv_sqrt_c2);
        adam_one(g[k].w * h.grad_scale, w4[k].w, m4[k].w, v4[k].w, h, inv_c1, inv_sqrt_c2);
        *reinterpret_cast<float4*>(master + se[k]) = w4[k];
        *reinterpret_cast<float4*>(m + se[k]) = m4[k];
        *reinterpret_cast<float4*>(v + se[k]) = v4[k];
        *reinterpret_cast<uint2*>(work + c.offset + (i4 << 2)) =
            make_uint2(pack_bf16x2(w4[k].x, w4[k].y), pack_bf16x2(w4[k].z, w4[k].w));
      }
    }
    return;
  }
  // Anything else: the same, an element at a time (indices inside a region fit the items' 32 bits).  Sixteen
  // regions of 3000 x 30: 11 us; 26 with the elements of a thread one after the other, and 19 so in one
  // CTA an item.
  const unsigned ld = unsigned(c.ld), end = item.first + item.count;
  constexpr int U = 2;
  for (unsigned i0 = item.first + first; i0 < end; i0 += U * 256u * kAdamShares) {
    float g[U], w[U], mi[U], vi[U];
    long long se[U];
    bool live[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const unsigned i = i0 + k * 256u * kAdamShares;
      live[k] = false;
      if (i < end) {
        const unsigned row = i / ld;
        const long long col = (long long)(i - row * ld) - c.col0;
        live[k] = col >= 0 && col < c.cols;
        se[k] = c.state + row * c.cols + col;
        if (live[k]) {
          g[k] = grad[c.offset + i];
          w[k] = master[se[k]];
          mi[k] = m[se[k]];
          vi[k] = v[se[k]];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const unsigned i = i0 + k * 256u * kAdamShares;
      if (i < end) grad[c.offset + i] = 0.f;
      if (!live[k]) continue;
      adam_one(g[k] * h.grad_scale, w[k], mi[k], vi[k], h, inv_c1, inv_sqrt_c2);
      m[se[k]] = mi[k];
      v[se[k]] = vi[k];
      master[se[k]] = w[k];
      work[c.offset + i] = __float2bfloat16(w[k]);
    }
  }
}

}  // namespace lf

using namespace lf;

extern "C" {

int lf_cross_entropy(void* logits, const int* labels, float* loss, long long M, int V,
                     long long ld, float grad_scale, void* stream) {
  if (M == 0) return 0;
  if (ld % 8 != 0) return -1;
  if (V <= 128 * CE_VECS * 8)
    cross_entropy_kernel<128><<<(unsigned)M, 128, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)logits, labels, loss, V, ld,
                                                                             grad_scale);
  else
    cross_entropy_kernel<512><<<(unsigned)M, 512, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)logits, labels, loss, V, ld,
                                                                             grad_scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// chunks: device array of AdamChunk {int64 offset, rows, ld, col0, cols, state};
// items: device array of AdamWorkItem {int32 chunk, uint32 first, uint32 count} covering every
// element of every chunk exactly once (first and count multiples of 4 unless the chunk has odd
// offsets or sizes).
int lf_adam_chunks(const void* chunks, const void* items, int num_items, float* grad, float* master,
                   float* m, float* v, void* work, float lr, float beta1, float beta2, float eps,
                   float weight_decay, int step, float grad_scale, void* stream) {
  if (num_items <= 0) return 0;
  AdamHyper h;
  h.lr = lr;
  h.beta1 = beta1;
  h.beta2 = beta2;
  h.eps = eps;
  h.weight_decay = weight_decay;
  h.bias_c1 = 1.f - powf(beta1, (float)step);
  h.bias_c2 = 1.f - powf(beta2, (float)step);
  h.grad_scale = grad_scale;
  adam_chunks_kernel<<<num_items * kAdamShares, 256, 0, (cudaStream_t)stream>>>(
      (const AdamChunk*)chunks, (const AdamWorkItem*)items, grad, master, m, v, (__nv_bfloat16*)work, h);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
