// What the batched rank's kernels share: tile layout, sums, shared memory.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "block_inv.cuh"
#include "field.cuh"
#include "mma_limbs.cuh"
#include "rank_batch.cuh"

namespace modlin {

namespace {

constexpr int kP = 64;  // panel width
constexpr int kG = 8;   // rows per warp in flight during the in-panel elimination
constexpr int kStride = 80;                // bytes per row of a 64-deep limb plane
constexpr int kPlane = kP * kStride;       // one limb plane of a 64 x 64 tile
constexpr int kRegion = 8 * kPlane;        // 8 limb planes: 40 KiB

// Lazy accumulation of products of residues: u128 sums reduced once per
// safe_batch products in general; for p < 2^32 a product fits in 32 x 32 ->
// 64 bits, so the sums stay in a u64 and are reduced once per
// floor((2^64 - 1) / (p - 1)^2) products (at least 1; p < 2^31 gives >= 4).
// A reduced sum (< p) counts as one product.
template <class F>
struct Acc {
  using T = u128;
  __device__ static T prod(const F& f, uint64_t a, uint64_t b) { return f.prod(a, b); }
  __device__ static uint64_t reduce(const F& f, T x) { return f.reduce(x); }
  __device__ static uint64_t batch(const F& f) { return f.safe_batch(); }
};
template <>
struct Acc<FpSmall> {
  using T = uint64_t;
  __device__ static T prod(const FpSmall&, uint64_t a, uint64_t b) { return (uint64_t)(uint32_t)a * (uint32_t)b; }
  __device__ static uint64_t reduce(const FpSmall& f, T x) { return f.reduce64(x); }
  __device__ static uint64_t batch(const FpSmall& f) {
    const uint64_t q = f.modulus() - 1;
    return q <= 1 ? UINT64_MAX : UINT64_MAX / (q * q);
  }
};

// Regions of shared memory: `a` holds the block being inverted, then the left
// operand's planes, or LF on the panel path; `b` the inverse's scratch, then
// the right operand's planes, or Us; `a2` (one CTA an SM) the left operand's
// second buffer.
struct BatchSmem {
  alignas(16) uint8_t b[kRegion];
  alignas(16) uint8_t a[kRegion];
  uint64_t prow[kP];  // pivot row's panel segment
  int pcol[kP];
  int red[16];
  uint64_t inv;
  int found;
  long long job;
};
static_assert(sizeof(InvScratch<8>) <= kRegion && kP * kInvLd * 8 <= kRegion && kP * (kP + 1) * 8 <= kRegion, "");

// Diagonal sums of the 16 x 8 tile (row group rg, column group cg) of the
// 64 x 64 product of the planes at A and B.
template <int LIMBS>
__device__ __forceinline__ void block_tile(uint32_t (&acc)[2 * LIMBS - 1][4], const uint8_t* A, const uint8_t* B,
                                           int rg, int cg) {
  mml::tile_k32<LIMBS, 2, kStride>(acc, mml::saddr(A) + rg * 16 * kStride, kPlane, mml::saddr(B) + cg * 8 * kStride,
                                   kPlane);
}

}  // namespace

}  // namespace modlin
