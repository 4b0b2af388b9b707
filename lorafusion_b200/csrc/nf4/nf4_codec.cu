// NF4 (4-bit NormalFloat) block quantisation of frozen base weights and the standalone
// dequantiser.
//
// Format (compatible with the bitsandbytes layout the reference dequantises in
// lorafusion/ops/triton_ops/dequantize_nf4.py:16-161): the weight [N, K] is flattened
// row-major and cut into blocks of 64 elements (K % 64 == 0, so a block never crosses a
// row); each block stores absmax and 64 4-bit codes, two per byte with the EVEN element in
// the high nibble.  The absmax vector is itself quantised ("double quantisation"): after
// subtracting its mean (`offset`), groups of 256 absmax values share one fp32 scale and
// each value is an 8-bit index into a 256-entry code table.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lf {

__constant__ float kNf4Code[16] = {
    -1.0f,
    -0.6961928009986877f,
    -0.5250730514526367f,
    -0.39491748809814453f,
    -0.28444138169288635f,
    -0.18477343022823334f,
    -0.09105003625154495f,
    0.0f,
    0.07958029955625534f,
    0.16093020141124725f,
    0.24611230194568634f,
    0.33791524171829224f,
    0.44070982933044434f,
    0.5626170039176941f,
    0.7229568362236023f,
    1.0f,
};

// Encoding: the code of x in [-1, 1] is the number of midpoints between consecutive code values
// that lie below x.  Midpoints are at least 0.079 apart, so of the 33 bins of width 1/16 centred on
// -1, -15/16, ..., 1 none holds two: a bin stores how many midpoints lie below it and the next
// midpoint (its own, if it has one), and one comparison settles the code.  That is two conflict-free
// shared-memory reads and about nine instructions an element instead of fifteen comparisons and
// additions, which had made the kernel five times slower than its loads and stores
// (28672 x 4096: 378 us for 300 MB).
constexpr int kEncodeBins = 64;   // 33 in use; the rest catch NaN, which encodes as 0

struct EncodeTables {
  float mid[kEncodeBins];
  uint32_t below[kEncodeBins];
};

__device__ __forceinline__ void fill_encode_tables(EncodeTables& t) {
  for (int b = threadIdx.x; b < kEncodeBins; b += blockDim.x) {
    const float lower = float(b - 16) / 16.f - 1.f / 32.f;
    uint32_t n = 0;
    float next = 2.f;   // past every value: the last bins have no midpoint left
    if (b <= 32) for (int i = 14; i >= 0; --i) {
      const float mid = 0.5f * (kNf4Code[i] + kNf4Code[i + 1]);
      if (mid < lower) ++n;
      else next = mid;
    }
    t.mid[b] = next;
    t.below[b] = n;
  }
}

__device__ __forceinline__ uint32_t nf4_encode(float x, const EncodeTables& t) {
  // 16 x + 16 rounded to an integer in the low mantissa bits.  A value on the edge of two bins may
  // go to either: no midpoint lies there, so both give the same code.
  const uint32_t b = __float_as_uint(fmaf(x, 16.f, 8388608.f + 16.f)) & 63u;
  return t.below[b] + (x > t.mid[b] ? 1u : 0u);
}

// Eight threads cover one 64-element block, each quantises 8 consecutive elements; a thread takes
// kQuantVecs such pieces, one block-width of threads apart, with all loads issued first.
constexpr int kQuantThreads = 256;
constexpr int kQuantVecs = 4;

__global__ void __launch_bounds__(kQuantThreads)
nf4_quantize_kernel(const __nv_bfloat16* __restrict__ w, uint8_t* __restrict__ packed, float* __restrict__ absmax,
                    long long n_elems) {
  __shared__ EncodeTables tables;
  const long long t0 = (long long)blockIdx.x * kQuantThreads * kQuantVecs + threadIdx.x;
  uint4 raw[kQuantVecs];
#pragma unroll
  for (int k = 0; k < kQuantVecs; ++k) {
    const long long e0 = (t0 + k * kQuantThreads) * 8;
    raw[k] = e0 < n_elems ? *reinterpret_cast<const uint4*>(w + e0) : make_uint4(0u, 0u, 0u, 0u);
  }
  fill_encode_tables(tables);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kQuantVecs; ++k) {
    const long long t = t0 + k * kQuantThreads;
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[k]);
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 v = __bfloat1622float2(h[j]);
      f[2 * j] = v.x;
      f[2 * j + 1] = v.y;
    }
    float am = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) am = fmaxf(am, fabsf(f[j]));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 4));
    if (t * 8 >= n_elems) continue;   // whole blocks of 64 are in or out: the shuffles above are complete
    const float inv = am > 0.f ? 1.f / am : 0.f;
    uint32_t out = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t hi = nf4_encode(f[2 * j] * inv, tables);
      const uint32_t lo = nf4_encode(f[2 * j + 1] * inv, tables);
      out |= ((hi << 4) | lo) << (8 * j);
    }
    reinterpret_cast<uint32_t*>(packed)[t] = out;
    if ((t & 7) == 0) absmax[t >> 3] = am;
  }
}

// Second level of the quantisation: the absmax vector minus its mean, in groups of 256 that share
// one fp32 scale, as the nearest of 256 code values (`mids` = the 255 midpoints between them).
// The mean is summed in 64 bits: fixed shares per CTA, then the partial sums in order, so it does not
// depend on scheduling.
constexpr int kMeanParts = 148;

__global__ void __launch_bounds__(256)
nf4_absmax_sum_kernel(const float* __restrict__ absmax, long long n, double* __restrict__ partial) {
  __shared__ double red[8];
  double s = 0.0;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += 256ll * kMeanParts) s += double(absmax[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = red[0];
    for (int i = 1; i < 8; ++i) t += red[i];
    partial[blockIdx.x] = t;
  }
}

// One warp per group of 256.
__global__ void __launch_bounds__(256)
nf4_double_quantize_kernel(const float* __restrict__ absmax, long long n, const double* __restrict__ partial,
                           const float* __restrict__ mids, const float* __restrict__ code, uint8_t* __restrict__ q,
                           float* __restrict__ code_out, float* __restrict__ nested, float* __restrict__ offset) {
  __shared__ float s_mid[256];
  __shared__ float s_mean;
  const int lane = threadIdx.x & 31;
  s_mid[threadIdx.x] = threadIdx.x < 255 ? mids[threadIdx.x] : INFINITY;
  if (blockIdx.x == 0) code_out[threadIdx.x] = code[threadIdx.x];   // every weight has a table of its own
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (int i = lane; i < kMeanParts; i += 32) t += partial[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) {
      s_mean = float(t / double(n));
      if (blockIdx.x == 0) *offset = s_mean;
    }
  }
  __syncthreads();
  const float mean = s_mean;
  const long long group = blockIdx.x * 8ll + (threadIdx.x >> 5);
  if (group * 256 >= n) return;
  float c[8];
  float mx = 0.f;
  bool nan = false;   // an infinite weight: its group's scale is NaN, as |c|'s maximum is
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const long long i = group * 256 + k * 32 + lane;
    c[k] = i < n ? absmax[i] - mean : 0.f;
    nan |= isnan(c[k]);
    mx = fmaxf(mx, fabsf(c[k]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float scale = __any_sync(0xffffffffu, nan) ? NAN : fmaxf(mx, 1e-12f);
  if (lane == 0) nested[group] = scale;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const long long i = group * 256 + k * 32 + lane;
    if (i >= n) continue;
    const float x = __fdiv_rn(c[k], scale);
    int lo = 0;   // number of midpoints below x
#pragma unroll
    for (int step = 128; step > 0; step >>= 1)
      if (!(s_mid[lo + step - 1] >= x)) lo += step;
    q[i] = uint8_t(lo);
  }
}

// Expansion.  Persistent CTAs: a thread expands four 4-byte words (8 codes each) that lie one
// block-width apart, so that every load instruction of a warp reads 128 contiguous bytes and every
// store instruction writes 512, and the words, scale codes and group scales of its next piece are
// on their way meanwhile; the table of scale codes sits in shared memory.  One short-lived CTA per
// piece, with three dependent global loads before its first store, spent most of its life waiting.
// With fp32 block scales there is one load less to wait for, and short-lived CTAs, one a piece and eight on
// an SM, are the faster ones: 28672 x 8192 92 us against 114 (8192 x 8192: 29.2 against 33.6).
//   absmax_q == nullptr : `absmax` holds fp32 block scales
//   absmax_q != nullptr : scale = code256[absmax_q[b]] * nested[b / 256] + offset
constexpr int kDequantThreads = 256;
constexpr int kDequantWords = 4;
constexpr int kDequantCtas = 148 * 6;   // persistent ones, resident at once

template <bool NESTED>
__global__ void __launch_bounds__(kDequantThreads, NESTED ? 6 : 1)
nf4_dequantize_kernel(const uint32_t* __restrict__ packed, const float* __restrict__ absmax,
                      const uint8_t* __restrict__ absmax_q, const float* __restrict__ code256,
                      const float* __restrict__ nested, float offset, uint4* __restrict__ out, long long n_words) {
  __shared__ float lut[16];
  __shared__ float code[256];
  if (threadIdx.x < 16) lut[threadIdx.x] = kNf4Code[threadIdx.x];
  if (NESTED) code[threadIdx.x] = code256[threadIdx.x];
  __syncthreads();
  const long long step = (long long)gridDim.x * kDequantThreads * kDequantWords;
  uint32_t word[kDequantWords], sq[kDequantWords];
  float sc[kDequantWords];
  auto load = [&](long long w0) {
#pragma unroll
    for (int k = 0; k < kDequantWords; ++k) {
      const long long wi = w0 + k * kDequantThreads;
      if (wi < n_words) {
        word[k] = packed[wi];
        const long long blk = wi >> 3;   // 64 codes per scale block
        if (NESTED) {
          sq[k] = absmax_q[blk];
          sc[k] = nested[blk >> 8];
        } else {
          sc[k] = absmax[blk];
        }
      }
    }
  };
  long long w0 = (long long)blockIdx.x * kDequantThreads * kDequantWords + threadIdx.x;
  load(w0);
  do {
    uint32_t cur[kDequantWords];
    float scale[kDequantWords];
#pragma unroll
    for (int k = 0; k < kDequantWords; ++k) {
      cur[k] = word[k];
      scale[k] = NESTED ? code[sq[k] & 255u] * sc[k] + offset : sc[k];
    }
    if (NESTED) load(w0 + step);
#pragma unroll
    for (int k = 0; k < kDequantWords; ++k) {
      const long long wi = w0 + k * kDequantThreads;
      if (wi >= n_words) continue;
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t byte = (cur[k] >> (8 * j)) & 0xffu;
        // even element in the high nibble
        __nv_bfloat162 v = __floats2bfloat162_rn(lut[byte >> 4] * scale[k], lut[byte & 15u] * scale[k]);
        o[j] = *reinterpret_cast<uint32_t*>(&v);
      }
      out[wi] = make_uint4(o[0], o[1], o[2], o[3]);
    }
    w0 += step;
  } while (NESTED && w0 < n_words);
}

}  // namespace lf

using namespace lf;

extern "C" {

int lf_nf4_quantize(const void* w, void* packed, float* absmax, long long n_elems, void* stream) {
  if (n_elems % 64 != 0) return -1;
  if (n_elems == 0) return 0;
  const long long per_block = (long long)kQuantThreads * kQuantVecs * 8;
  const long long grid = (n_elems + per_block - 1) / per_block;
  nf4_quantize_kernel<<<(unsigned)grid, kQuantThreads, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)w, (uint8_t*)packed, absmax, n_elems);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// absmax: fp32 [n]; partial: double [148] scratch; mids: fp32 [255]; code: fp32 [256]; q: uint8 [n]; code_out:
// fp32 [256], a copy of code; nested: fp32 [ceil(n / 256)]; offset: fp32 [1], the mean that was subtracted.
int lf_nf4_double_quantize(const float* absmax, long long n, double* partial, const float* mids, const float* code,
                           void* q, float* code_out, float* nested, float* offset, void* stream) {
  if (n <= 0) return n == 0 ? 0 : -1;
  cudaStream_t st = (cudaStream_t)stream;
  nf4_absmax_sum_kernel<<<kMeanParts, 256, 0, st>>>(absmax, n, partial);
  const long long groups = (n + 255) / 256;
  nf4_double_quantize_kernel<<<(unsigned)((groups + 7) / 8), 256, 0, st>>>(absmax, n, partial, mids, code,
                                                                            (uint8_t*)q, code_out, nested, offset);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_nf4_dequantize(const void* packed, const float* absmax, const void* absmax_q,
                      const float* code256, const float* nested, float offset, void* out,
                      long long n_elems, void* stream) {
  if (n_elems % 64 != 0) return -1;
  if (n_elems == 0) return 0;
  const long long n_words = n_elems / 8;
  const long long per_block = (long long)kDequantThreads * kDequantWords;
  long long grid = (n_words + per_block - 1) / per_block;
  if (absmax_q != nullptr && grid > kDequantCtas) grid = kDequantCtas;
  cudaStream_t st = (cudaStream_t)stream;
  if (absmax_q != nullptr)
    nf4_dequantize_kernel<true><<<(unsigned)grid, kDequantThreads, 0, st>>>(
        (const uint32_t*)packed, absmax, (const uint8_t*)absmax_q, code256, nested, offset, (uint4*)out, n_words);
  else
    nf4_dequantize_kernel<false><<<(unsigned)grid, kDequantThreads, 0, st>>>(
        (const uint32_t*)packed, absmax, nullptr, nullptr, nullptr, 0.f, (uint4*)out, n_words);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
