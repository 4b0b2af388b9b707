// Memory-bound token-wise kernels of the decoder block: RMSNorm (+ fused residual add),
// rotary embedding applied in place to the packed QKV projection, SwiGLU on the merged
// gate|up projection, and the embedding gather.  The base model is frozen, so none of the
// backward kernels produces weight gradients.  They stand in for the Liger Triton kernels
// the reference patches into HF models (lorafusion/utils/module.py:40-69).
//
// All kernels use 16-byte vector accesses; feature sizes must be multiples of 8.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lf {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < THREADS / 32) ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}

struct alignas(16) BF8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  BF8 b = *reinterpret_cast<const BF8*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(b.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void unpack8(const uint4& raw, float (&f)[8]) {
  const BF8& b = reinterpret_cast<const BF8&>(raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(b.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  BF8 b;
#pragma unroll
  for (int i = 0; i < 4; ++i) b.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<BF8*>(p) = b;
}

// ---------------------------------------------------------------------------------
// RMSNorm forward:  h = x (+ res);  y = h * rsqrt(mean(h^2) + eps) * w
// One CTA per token row; the row stays in registers between the reduction and the write.
// ---------------------------------------------------------------------------------
constexpr int NORM_THREADS = 256;
constexpr int NORM_MAX_VEC = 8;  // supports H up to 256 * 8 * 8 = 16384

// NV = 16-byte vectors per thread (ceil(H / 8 / 256)); a template so that the row fits in
// as few registers as the hidden size needs (occupancy is what hides the DRAM latency here).
template <int NV>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ h_out, float* __restrict__ rstd_out, int H,
                   float eps) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * H;
  const int nvec = H / 8;
  float v[NV][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
    if (c < nvec) {
      load8(xr + c * 8, v[i]);
      if (res != nullptr) {
        float r[8];
        load8(res + row * H + c * 8, r);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] += r[j];
        // the residual stream is stored in bf16: normalise exactly what is stored
        BF8 b;
#pragma unroll
        for (int j = 0; j < 4; ++j) b.v[j] = __floats2bfloat162_rn(v[i][2 * j], v[i][2 * j + 1]);
        if (h_out != nullptr) *reinterpret_cast<BF8*>(h_out + row * H + c * 8) = b;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 t = __bfloat1622float2(b.v[j]);
          v[i][2 * j] = t.x;
          v[i][2 * j + 1] = t.y;
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += v[i][j] * v[i][j];
    }
  }
  ss = block_sum<NORM_THREADS>(ss, red);
  const float rstd = rsqrtf(ss / float(H) + eps);
  if (threadIdx.x == 0 && rstd_out != nullptr) rstd_out[row] = rstd;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
    if (c < nvec) {
      float wv[8], o[8];
      load8(w + c * 8, wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = v[i][j] * rstd * wv[j];
      store8(y + row * H + c * 8, o);
    }
  }
}

// RMSNorm backward (no weight grad):
//   g = dy * w;  dx = rstd * (g - xhat * mean(g * xhat))  (+ dres),  xhat = h * rstd
template <int NV>
__global__ void __launch_bounds__(NORM_THREADS, NV <= 1 ? 8 : (NV <= 2 ? 5 : (NV <= 4 ? 3 : 2)))
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ h,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx, int H) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const int nvec = H / 8;
  const float rstd = rstd_in[row];
  // The row is read once and waits for the dot product as the bf16 it came in, four registers per
  // vector.  (Kept as fp32 it cost 96-106 registers a thread and with them the resident CTAs that
  // hide the DRAM latency; read a second time it cost L2 bandwidth: 173 us for 16384 x 4096, 98 so.
  // 8192 rows of 10240, 12288, 16384: 163, 195, 261 us with the second read, 122, 139, 178 so.  Rows of
  // up to 2048 need room for eight CTAs: at five, 8192 x 64 took 10.7 us, 9.3 at eight.)
  uint4 gv[NV], hv[NV], rv[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
    if (c < nvec) {
      gv[i] = *reinterpret_cast<const uint4*>(dy + row * H + c * 8);
      hv[i] = *reinterpret_cast<const uint4*>(h + row * H + c * 8);
      if (dres != nullptr) rv[i] = *reinterpret_cast<const uint4*>(dres + row * H + c * 8);
    }
  }
  float dot = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
    if (c < nvec) {
      float g[8], xh[8], wv[8];
      unpack8(gv[i], g);
      unpack8(hv[i], xh);
      load8(w + c * 8, wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) dot += (g[j] * wv[j]) * (xh[j] * rstd);
    }
  }
  dot = block_sum<NORM_THREADS>(dot, red) / float(H);
#pragma unroll
  for (int i = 0; i < NV; ++i) {   // or the compiler keeps the fp32 values of the first loop instead
    asm volatile("" : "+r"(gv[i].x), "+r"(gv[i].y), "+r"(gv[i].z), "+r"(gv[i].w));
    asm volatile("" : "+r"(hv[i].x), "+r"(hv[i].y), "+r"(hv[i].z), "+r"(hv[i].w));
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
    if (c < nvec) {
      float g[8], xh[8], wv[8], o[8];
      unpack8(gv[i], g);
      unpack8(hv[i], xh);
      load8(w + c * 8, wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rstd * (g[j] * wv[j] - (xh[j] * rstd) * dot);
      if (dres != nullptr) {
        float r[8];
        unpack8(rv[i], r);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += r[j];
      }
      store8(dx + row * H + c * 8, o);
    }
  }
}

// ---------------------------------------------------------------------------------
// Rotary embedding, rotate-half convention, in place on the q and k parts of the packed
// QKV activation [M, (Hq + 2 Hkv) * D].  cos/sin come from a table [max_pos, D/2] gathered
// by position id.  `sign` = +1 forward, -1 backward (the transpose of a rotation).
// ---------------------------------------------------------------------------------
// One CTA per token, or several where there are few heads and many tokens; threadIdx.x = 16-byte vector
// of a half head, threadIdx.y = head, threadIdx.z = token.  A thread keeps its piece of the cos / sin row
// for all the heads it rotates, two at a time and as many as every other thread (lf_rope_inplace), and
// the first heads are on their way before the position that selects the row is known.  16384 tokens of 1,
// 40 and 72 heads of 128: 5.7, 66, 105 us; 6.7, 74, 126 with a flat index over all vectors, two
// 64-bit divisions and a cos / sin load each; 11, 75, 118 with one token a CTA and 32 heads at a time,
// where a quarter of the threads rotated two of 40 heads and the others one.
constexpr int ROPE_THREADS = 256;

__global__ void __launch_bounds__(ROPE_THREADS)
rope_inplace_kernel(__nv_bfloat16* __restrict__ qkv, const int* __restrict__ pos, const float* __restrict__ cos_t,
                    const float* __restrict__ sin_t, int M, int n_rot_heads, int D, int row_stride, float sign) {
  const int half = D / 2;
  const long long row = (long long)blockIdx.x * blockDim.z + threadIdx.z;
  if (row >= M) return;
  const int by = blockDim.y;
  for (int vi = threadIdx.x; vi < half / 8; vi += blockDim.x) {   // (once, up to head size 4096)
    __nv_bfloat16* base = qkv + row * row_stride + vi * 8;
    uint4 lo[2], hi[2];
    auto load = [&](int h0) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int head = h0 + k * by;
        if (head < n_rot_heads) {
          lo[k] = *reinterpret_cast<const uint4*>(base + head * D);
          hi[k] = *reinterpret_cast<const uint4*>(base + head * D + half);
        }
      }
    };
    load(threadIdx.y);
    const long long table = (long long)pos[row] * half + vi * 8;
    float c[8], s[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      c[j] = cos_t[table + j];
      s[j] = sign * sin_t[table + j];
    }
    for (int h0 = threadIdx.y; h0 < n_rot_heads; h0 += 2 * by) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int head = h0 + k * by;
        if (head < n_rot_heads) {
          float l[8], h[8], olo[8], ohi[8];
          unpack8(lo[k], l);
          unpack8(hi[k], h);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            olo[j] = l[j] * c[j] - h[j] * s[j];
            ohi[j] = h[j] * c[j] + l[j] * s[j];
          }
          store8(base + head * D, olo);
          store8(base + head * D + half, ohi);
        }
      }
      load(h0 + 2 * by);
    }
  }
}

// ---------------------------------------------------------------------------------
// SwiGLU on the merged projection gu[M, 2I] = [gate | up]:  out = silu(gate) * up
// ---------------------------------------------------------------------------------
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu,
                                  __nv_bfloat16* __restrict__ out, long long M, int I) {
  const int vec = I / 8;
  const long long total = M * vec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long row = idx / vec;
    const int c = int(idx % vec) * 8;
    float g[8], u[8], o[8];
    load8(gu + row * 2 * I + c, g);
    load8(gu + row * 2 * I + I + c, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    store8(out + row * I + c, o);
  }
}

// dgu[M, 2I] from dout[M, I] and the saved gu.  One CTA per piece of a row, the pieces of a row side by
// side: one small division a CTA and all loads of two vectors in flight a thread, 190 -> 172 us for
// 8192 x 14336 (a flat index over all vectors takes two 64-bit divisions each).  The forward kernel,
// which has a third fewer loads to wait for, is the faster one with the flat index: 243 against 286 for
// 16384 x 14336.
// Rows too short for a CTA share one (threadIdx.y = row): 8192 x 64 took 3.5 us with the flat index, 8.7
// with eight threads of a CTA at work, 4.2 so (8192 x 256: 5.6, 9.0, 5.0).
constexpr int SWIGLU_THREADS = 256;
constexpr int SWIGLU_VECS = 2;

__global__ void __launch_bounds__(SWIGLU_THREADS)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ gu,
                  __nv_bfloat16* __restrict__ dgu, long long M, int I, int pieces) {
  const int vec = I / 8, bx = blockDim.x;
  const long long m = (long long)(blockIdx.x / pieces) * blockDim.y + threadIdx.y;
  if (m >= M) return;
  const __nv_bfloat16* row = gu + m * 2 * I;
  const __nv_bfloat16* drow = dout + m * I;
  __nv_bfloat16* orow = dgu + m * 2 * I;
  const int c0 = blockIdx.x % pieces * (bx * SWIGLU_VECS) + threadIdx.x;
  uint4 gv[SWIGLU_VECS], uv[SWIGLU_VECS], dv[SWIGLU_VECS];
#pragma unroll
  for (int k = 0; k < SWIGLU_VECS; ++k) {
    const int c = c0 + k * bx;
    if (c < vec) {
      gv[k] = *reinterpret_cast<const uint4*>(row + c * 8);
      uv[k] = *reinterpret_cast<const uint4*>(row + I + c * 8);
      dv[k] = *reinterpret_cast<const uint4*>(drow + c * 8);
    }
  }
#pragma unroll
  for (int k = 0; k < SWIGLU_VECS; ++k) {
    const int c = c0 + k * bx;
    if (c < vec) {
      float g[8], u[8], d[8], dg[8], du[8];
      unpack8(gv[k], g);
      unpack8(uv[k], u);
      unpack8(dv[k], d);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float sig = 1.f / (1.f + __expf(-g[j]));
        const float silu = g[j] * sig;
        du[j] = d[j] * silu;
        dg[j] = d[j] * u[j] * (sig + silu * (1.f - sig));
      }
      store8(orow + c * 8, dg);
      store8(orow + I + c * 8, du);
    }
  }
}

// ---------------------------------------------------------------------------------
// Embedding gather: out[m, :] = table[ids[m], :]
// ---------------------------------------------------------------------------------
__global__ void embedding_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                                 __nv_bfloat16* __restrict__ out, long long M, int H, int vocab) {
  const int vec = H / 8;
  const long long total = M * vec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long row = idx / vec;
    const int c = int(idx % vec) * 8;
    int id = ids[row];
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    *reinterpret_cast<BF8*>(out + row * H + c) =
        *reinterpret_cast<const BF8*>(table + (long long)id * H + c);
  }
}

// out = a + b (bf16), used for residual adds that are not fused into a norm.
__global__ void add_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                           __nv_bfloat16* __restrict__ out, long long n8) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n8;
       idx += (long long)gridDim.x * blockDim.x) {
    float x[8], y[8];
    load8(a + idx * 8, x);
    load8(b + idx * 8, y);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] += y[j];
    store8(out + idx * 8, x);
  }
}

static inline int grid_for(long long total, int threads) {
  long long b = (total + threads - 1) / threads;
  const long long cap = 148LL * 16;
  return int(b < 1 ? 1 : (b > cap ? cap : b));
}


// How many of M short rows share a CTA: at most `most` (and 64), and so that two CTAs an SM remain.
static inline int rows_per_cta(long long M, int most) {
  int n = most < 64 ? most : 64;
  while (n > 1 && (M + n - 1) / n < 2 * 148) n /= 2;
  return n < 1 ? 1 : n;
}

}  // namespace lf

using namespace lf;

extern "C" {

int lf_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out,
                   float* rstd, long long M, int H, float eps, void* stream) {
  if (H % 8 != 0 || H > NORM_THREADS * NORM_MAX_VEC * 8) return -1;
  if (M == 0) return 0;
  const int nv = (H / 8 + NORM_THREADS - 1) / NORM_THREADS;
#define LF_NORM_FWD(NVV)                                                                        \
  rmsnorm_fwd_kernel<NVV><<<(unsigned)M, NORM_THREADS, 0, (cudaStream_t)stream>>>(               \
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w,              \
      (__nv_bfloat16*)y, (__nv_bfloat16*)h_out, rstd, H, eps)
  if (nv <= 1) LF_NORM_FWD(1);
  else if (nv == 2) LF_NORM_FWD(2);
  else if (nv == 3) LF_NORM_FWD(3);
  else if (nv == 4) LF_NORM_FWD(4);
  else LF_NORM_FWD(8);
#undef LF_NORM_FWD
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd,
                   const void* dres, void* dx, long long M, int H, void* stream) {
  if (H % 8 != 0 || H > NORM_THREADS * NORM_MAX_VEC * 8) return -1;
  if (M == 0) return 0;
  const int nv = (H / 8 + NORM_THREADS - 1) / NORM_THREADS;
#define LF_NORM_BWD(NVV)                                                                        \
  rmsnorm_bwd_kernel<NVV><<<(unsigned)M, NORM_THREADS, 0, (cudaStream_t)stream>>>(               \
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)h, (const __nv_bfloat16*)w, rstd,         \
      (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, H)
  if (nv <= 1) LF_NORM_BWD(1);
  else if (nv == 2) LF_NORM_BWD(2);
  else if (nv == 3) LF_NORM_BWD(3);
  else if (nv == 4) LF_NORM_BWD(4);
  else LF_NORM_BWD(8);
#undef LF_NORM_BWD
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_rope_inplace(void* qkv, const int* pos, const float* cos_t, const float* sin_t, int M,
                    int n_rot_heads, int D, int row_stride, int backward, void* stream) {
  if (D % 16 != 0 || row_stride % 8 != 0) return -1;
  if (M == 0 || n_rot_heads <= 0 || D <= 0) return 0;
  const int bx = D / 16 < ROPE_THREADS ? D / 16 : ROPE_THREADS;
  int by = ROPE_THREADS / bx;
  if (by < n_rot_heads) {   // an even number of heads a thread, the same for all but the last
    const int per = ((n_rot_heads + by - 1) / by + 1) / 2 * 2;
    by = (n_rot_heads + per - 1) / per;
  } else {
    by = n_rot_heads;
  }
  const int bz = rows_per_cta(M, 128 / (bx * by));   // (z has room for 64)
  rope_inplace_kernel<<<((unsigned)M + bz - 1) / bz, dim3(bx, by, bz), 0, (cudaStream_t)stream>>>(
      (__nv_bfloat16*)qkv, pos, cos_t, sin_t, M, n_rot_heads, D, row_stride, backward ? -1.f : 1.f);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_swiglu_fwd(const void* gu, void* out, long long M, int I, void* stream) {
  if (I % 8 != 0) return -1;
  if (M == 0 || I == 0) return 0;
  swiglu_fwd_kernel<<<grid_for(M * (I / 8), 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)gu, (__nv_bfloat16*)out, M, I);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_swiglu_bwd(const void* dout, const void* gu, void* dgu, long long M, int I, void* stream) {
  if (I % 8 != 0) return -1;
  if (M == 0 || I == 0) return 0;
  const int vec = I / 8, half = (vec + SWIGLU_VECS - 1) / SWIGLU_VECS;
  const int bx = half < SWIGLU_THREADS ? half : SWIGLU_THREADS, by = rows_per_cta(M, SWIGLU_THREADS / bx);
  const int pieces = (half + bx - 1) / bx;
  swiglu_bwd_kernel<<<(unsigned)((M + by - 1) / by * pieces), dim3(bx, by), 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)dout, (const __nv_bfloat16*)gu, (__nv_bfloat16*)dgu, M, I, pieces);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_embedding(const int* ids, const void* table, void* out, long long M, int H, int vocab,
                 void* stream) {
  if (H % 8 != 0) return -1;
  if (M == 0) return 0;
  embedding_kernel<<<grid_for(M * (H / 8), 256), 256, 0, (cudaStream_t)stream>>>(
      ids, (const __nv_bfloat16*)table, (__nv_bfloat16*)out, M, H, vocab);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_add(const void* a, const void* b, void* out, long long n, void* stream) {
  if (n % 8 != 0) return -1;
  if (n == 0) return 0;
  add_kernel<<<grid_for(n / 8, 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)a, (const __nv_bfloat16*)b, (__nv_bfloat16*)out, n / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
