// Counter-based dropout mask shared by every kernel that needs it (and by the CPU oracle
// in lorafusion_b200/ops/philox.py, which must produce identical bits).
//
// One Philox4x32-7 call is keyed by (seed_lo, seed_hi) and indexed by the counter
// (row, col / 8, stream, 0).  Its 128 output bits are read as eight 16-bit lanes; element
// (row, col) uses lane (col % 8): lane j = (out[j >> 1] >> (16 * (j & 1))) & 0xffff and is
// KEPT iff lane >= thresh16, where thresh16 = round(p * 65536).  Because the mask is a
// pure function of (seed, stream, row, col) it is never stored: forward, recompute and
// the backward kernels regenerate it.
#pragma once
#include <stdint.h>

namespace lf {

struct Philox4 {
  uint32_t x, y, z, w;
};

__host__ __device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return static_cast<uint32_t>((static_cast<uint64_t>(a) * b) >> 32);
#endif
}

template <int ROUNDS = 7>
__host__ __device__ __forceinline__ Philox4 philox4x32(uint32_t c0, uint32_t c1, uint32_t c2,
                                                        uint32_t c3, uint32_t k0, uint32_t k1) {
  constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  constexpr uint32_t W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const uint32_t hi0 = mulhi32(M0, c0), lo0 = M0 * c0;
    const uint32_t hi1 = mulhi32(M1, c2), lo1 = M1 * c2;
    const uint32_t n0 = hi1 ^ c1 ^ k0;
    const uint32_t n2 = hi0 ^ c3 ^ k1;
    c0 = n0;
    c1 = lo1;
    c2 = n2;
    c3 = lo0;
    k0 += W0;
    k1 += W1;
  }
  return Philox4{c0, c1, c2, c3};
}

// Bit j of the result is 1 iff element (row, 8 * col8 + j) is kept.
__host__ __device__ __forceinline__ uint32_t dropout_keep8(uint32_t row, uint32_t col8,
                                                           uint32_t stream, uint32_t seed_lo,
                                                           uint32_t seed_hi, uint32_t thresh16) {
  const Philox4 o = philox4x32<7>(row, col8, stream, 0u, seed_lo, seed_hi);
  const uint32_t w[4] = {o.x, o.y, o.z, o.w};
  uint32_t bits = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t lane = (w[j >> 1] >> (16 * (j & 1))) & 0xffffu;
    bits |= (lane >= thresh16 ? 1u : 0u) << j;
  }
  return bits;
}

// The same call with the work that depends on the row alone or on the column alone taken out.
// Written as (row, col8, stream, 0), the first round multiplies only the row, the second one row
// and column apart, and half of the third still sees the row alone: of the fourteen 32 x 32 -> 64
// multiplies three belong to the row and one to the column, so a caller that walks the columns of
// a row (or the rows of a column) pays ten, or nine, per call.  Same bits as philox4x32<7>.
struct PhiloxRow {
  uint32_t a, b, c, d;
};
struct PhiloxCol {
  uint32_t e, f;
};
struct Wide {
  uint32_t hi, lo;
};

// One 32 x 32 -> 64 multiply for both halves.
__host__ __device__ __forceinline__ Wide mul_wide(uint32_t a, uint32_t b) {
  uint64_t p;
#if defined(__CUDA_ARCH__)
  asm("mul.wide.u32 %0, %1, %2;" : "=l"(p) : "r"(a), "r"(b));
#else
  p = uint64_t(a) * b;
#endif
  return Wide{uint32_t(p >> 32), uint32_t(p)};
}

__host__ __device__ __forceinline__ PhiloxRow philox_row(uint32_t row, uint32_t stream, uint32_t k0, uint32_t k1) {
  constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
  const Wide x = mul_wide(M0, row);
  const Wide y = mul_wide(M1, x.hi ^ k1);
  const Wide z = mul_wide(M0, y.hi ^ (M1 * stream) ^ (k0 + W0));
  return PhiloxRow{x.lo ^ (k1 + W1), y.lo ^ (k0 + 2u * W0), z.hi ^ (k1 + 2u * W1), z.lo};
}
__host__ __device__ __forceinline__ PhiloxCol philox_col(uint32_t col8, uint32_t stream, uint32_t k0) {
  constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  const Wide x = mul_wide(M0, mulhi32(M1, stream) ^ col8 ^ k0);
  return PhiloxCol{x.hi, x.lo};
}
__host__ __device__ __forceinline__ Philox4 philox_rest(const PhiloxRow& r, const PhiloxCol& c, uint32_t k0,
                                                         uint32_t k1) {
  constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
  const Wide x = mul_wide(M1, c.e ^ r.a);
  uint32_t c0 = x.hi ^ r.b, c1 = x.lo, c2 = r.c ^ c.f, c3 = r.d;
#pragma unroll
  for (uint32_t i = 3; i < 7; ++i) {
    const Wide u = mul_wide(M0, c0), v = mul_wide(M1, c2);
    c0 = v.hi ^ c1 ^ (k0 + i * W0);
    c2 = u.hi ^ c3 ^ (k1 + i * W1);
    c1 = v.lo;
    c3 = u.lo;
  }
  return Philox4{c0, c1, c2, c3};
}

// Two 16-bit lanes at once: 0xffff in each half of the result whose lane reaches the threshold
// (`thresh2` holds it in both halves, so it must fit 16 bits).  The lanes without their top bits
// are compared by one subtraction that cannot borrow across them; the top bits then decide by
// majority, and the verdict in each top bit is spread over its half.
__host__ __device__ __forceinline__ uint32_t keep_lanes2(uint32_t w, uint32_t thresh2) {
  const uint32_t d = (w | 0x80008000u) - (thresh2 & 0x7fff7fffu);
  const uint32_t ge = (w & d) | ((w | d) & ~thresh2);
#if defined(__CUDA_ARCH__)
  uint32_t m;
  asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(m) : "r"(ge));
  return m;
#else
  return ((ge & 0x8000u) ? 0xffffu : 0u) | ((ge & 0x80000000u) ? 0xffff0000u : 0u);
#endif
}

}  // namespace lf
