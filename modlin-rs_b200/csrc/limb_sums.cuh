// Exact residues from sums of 8-bit limb products: T = sum_d 2^(8d) S_d, S_d the
// sum of the products of limbs i and j with i + j = d.
#pragma once
#include <cstdint>

#include "field.cuh"

namespace modlin {

__device__ __forceinline__ uint64_t mad_wide_u32(uint32_t a, uint32_t b, uint64_t c) {
  uint64_t d;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// x = sum_{d<15} 2^(8d) a[d][c] mod 2^61 - 1, lazily: x < 2^62 and congruent.
// The diagonal sums are a[d][c] <= 8 * 128 * 255^2 < 2^26 (K <= 128), and
// 2^(8(d+8)) = 8 * 2^(8d) (mod p), so V_d = a_d + 8 a_(d+8) <= 57 * 128 * 255^2
// < 2^29 (d < 7; V_7 = a_7). L = sum_{d<4} 2^(8d) V_d and H = sum_{d<4}
// 2^(8d) V_(d+4) are < 2^54, and 2^32 H = 2^32 (H mod 2^29) + (H >> 29) (mod p)
// since 2^61 = 1, so x = L + 2^32 (H mod 2^29) + (H >> 29) < 2^62.
__device__ __forceinline__ uint64_t m61_fold15(const uint32_t (&a)[15][4], int c) {
  uint32_t V[8];
#pragma unroll
  for (int d = 0; d < 7; ++d) V[d] = a[d][c] + 8u * a[d + 8][c];
  V[7] = a[7][c];
  const uint64_t L = mad_wide_u32(V[3], 1u << 24, mad_wide_u32(V[2], 1u << 16, mad_wide_u32(V[1], 1u << 8, V[0])));
  const uint64_t H = mad_wide_u32(V[7], 1u << 24, mad_wide_u32(V[6], 1u << 16, mad_wide_u32(V[5], 1u << 8, V[4])));
  return L + ((uint64_t)((uint32_t)H & 0x1FFFFFFFu) << 32) + (H >> 29);
}

// (cv - x) mod 2^61 - 1 for a canonical cv and any x < 2^62:
// y = cv + 4p - x lies in (0, 2^64), one fold leaves y1 <= p + 7, and one
// conditional subtraction makes it canonical.
__device__ __forceinline__ uint64_t m61_sub_lazy(uint64_t cv, uint64_t x) {
  const uint64_t y = cv + (4 * kM61) - x;
  const uint64_t y1 = (y & kM61) + (y >> 61);
  return y1 >= kM61 ? y1 - kM61 : y1;
}

// sum_d 2^(8d) a[d][c] mod p for 8 limbs and any p < 2^63 (r64 = 2^64 mod p).
__device__ __forceinline__ uint64_t finish_wide(const FpBarrett& f, const uint32_t (&a)[15][4], int c, uint64_t r64) {
  u128 lo = 0, hi = 0;
#pragma unroll
  for (int d = 0; d < 8; ++d) lo += (u128)a[d][c] << (8 * d);
#pragma unroll
  for (int d = 8; d < 15; ++d) hi += (u128)a[d][c] << (8 * (d - 8));
  return f.add(f.reduce(lo), f.mul(f.reduce(hi), r64));
}

// The reductions of a field policy: T as a canonical residue, c + T and d x - T
// (c, d, x canonical). a[d][c]: diagonal d of the lane's entry c.
template <class F, int LIMBS>
struct LimbRed;

template <>
struct LimbRed<FpM61, 8> {
  __device__ explicit LimbRed(const FpM61&) {}
  __device__ __forceinline__ FpM61 field() const { return FpM61(); }
  // 2^S x mod p for a canonical x.
  template <int S>
  __device__ __forceinline__ uint64_t shifted(uint64_t x) const {
    return ((x << S) & kM61) | (x >> (61 - S));
  }
  static __device__ __forceinline__ uint64_t last(uint64_t y) {
    const uint64_t x = FpM61::fold(y);
    return x >= kM61 ? x - kM61 : x;
  }
  // T in a form that fits 64 bits, and c - T from it.
  __device__ __forceinline__ uint64_t lazy(const uint32_t (&a)[15][4], int c) const { return m61_fold15(a, c); }
  __device__ __forceinline__ uint64_t minus(uint64_t v, uint64_t t) const { return m61_sub_lazy(v, t); }
  __device__ __forceinline__ uint64_t residue(const uint32_t (&a)[15][4], int c) const {
    return last(m61_fold15(a, c));
  }
  __device__ __forceinline__ uint64_t plus(uint64_t v, const uint32_t (&a)[15][4], int c) const {
    return last(v + m61_fold15(a, c));  // < 2^61 + 2^62
  }
  __device__ __forceinline__ uint64_t mul_sub(uint64_t d, uint64_t x, const uint32_t (&a)[15][4], int c) const {
    const u128 t = (u128)d * x;
    const uint64_t lo = (uint64_t)t, hi = (uint64_t)(t >> 64);
    return last((lo & kM61) + ((lo >> 61) | (hi << 3)) + 4 * kM61 - m61_fold15(a, c));  // in (0, 2^64)
  }
};

// p < 2^32, diagonals below 2^26 (K <= 128): T is below 2^43 for LIMBS <= 2; for
// LIMBS = 4 the diagonals from 2^32 on are weighted by 2^(8d) mod p instead,
// which keeps T below 2^60. One 64-bit reduction either way.
template <int LIMBS>
struct LimbRed<FpSmall, LIMBS> {
  FpSmall f;
  uint32_t w[3];  // 2^32, 2^40, 2^48 mod p
  uint64_t kp;    // a multiple of p in [2^60, 2^60 + p)
  __device__ explicit LimbRed(const FpSmall& g) : f(g) {
    const uint64_t p = f.modulus();
    kp = ((1ULL << 60) + p - 1) / p * p;
    w[0] = (uint32_t)f.reduce64(1ULL << 32);
    w[1] = (uint32_t)f.reduce64(1ULL << 40);
    w[2] = (uint32_t)f.reduce64(1ULL << 48);
  }
  __device__ __forceinline__ const FpSmall& field() const { return f; }
  template <int S>
  __device__ __forceinline__ uint64_t shifted(uint64_t x) const {
    return f.reduce64(x << S);  // x < 2^32, S <= 32
  }
  __device__ __forceinline__ uint64_t lazy(const uint32_t (&a)[2 * LIMBS - 1][4], int c) const { return sum(a, c); }
  __device__ __forceinline__ uint64_t minus(uint64_t v, uint64_t t) const { return f.reduce64(v + kp - t); }
  __device__ __forceinline__ uint64_t sum(const uint32_t (&a)[2 * LIMBS - 1][4], int c) const {
    uint64_t t = a[0][c];
#pragma unroll
    for (int d = 1; d < (LIMBS == 4 ? 4 : 2 * LIMBS - 1); ++d) t += (uint64_t)a[d][c] << (8 * d);
    if constexpr (LIMBS == 4) {
#pragma unroll
      for (int d = 4; d < 7; ++d) t = mad_wide_u32(a[d][c], w[d - 4], t);
    }
    return t;
  }
  __device__ __forceinline__ uint64_t residue(const uint32_t (&a)[2 * LIMBS - 1][4], int c) const {
    return f.reduce64(sum(a, c));
  }
  __device__ __forceinline__ uint64_t plus(uint64_t v, const uint32_t (&a)[2 * LIMBS - 1][4], int c) const {
    return f.reduce64(v + sum(a, c));
  }
  __device__ __forceinline__ uint64_t mul_sub(uint64_t d, uint64_t x, const uint32_t (&a)[2 * LIMBS - 1][4],
                                              int c) const {
    if (f.modulus() >= (1ULL << 31)) return f.sub(f.mul(d, x), residue(a, c));
    return f.reduce64((uint64_t)(uint32_t)d * (uint32_t)x + kp - sum(a, c));  // < 2^62 + 2^61
  }
};

template <>
struct LimbRed<FpBarrett, 8> {
  FpBarrett f;
  uint64_t r64;  // 2^64 mod p
  __device__ explicit LimbRed(const FpBarrett& g) : f(g), r64(g.reduce((u128)1 << 64)) {}
  __device__ __forceinline__ const FpBarrett& field() const { return f; }
  template <int S>
  __device__ __forceinline__ uint64_t shifted(uint64_t x) const {
    return f.reduce((u128)x << S);
  }
  __device__ __forceinline__ uint64_t residue(const uint32_t (&a)[15][4], int c) const {
    return finish_wide(f, a, c, r64);
  }
  __device__ __forceinline__ uint64_t plus(uint64_t v, const uint32_t (&a)[15][4], int c) const {
    return f.add(v, residue(a, c));
  }
  __device__ __forceinline__ uint64_t mul_sub(uint64_t d, uint64_t x, const uint32_t (&a)[15][4], int c) const {
    return f.sub(f.mul(d, x), residue(a, c));
  }
};

}  // namespace modlin
