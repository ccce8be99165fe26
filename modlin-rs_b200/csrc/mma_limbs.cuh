// Modular products of small tiles on the tensor cores from inside a CTA:
// residues as LIMBS planes of 8-bit limbs in shared memory, warp-level
// mma.sync (u8 x u8 -> s32) for all limb pairs, accumulated by diagonal.
//
// For tiles of one CTA (64 x 64 blocks, one matrix per SM) the warp-level
// instruction is the fitting one: its operands are registers, a result is
// there after the last instruction, and nothing is staged through tensor
// memory. Measured on B200: an m16n8k32 takes 8 cycles of an SM quarter
// (2048 multiply-adds an SM and cycle, a quarter of tcgen05's rate), so a
// multiply-add over 2^61 - 1 (64 limb products) is 32 an SM and cycle, against
// 5 on the integer pipes (a 32 x 32 -> 64 multiply-add is issued every 4 cycles).
//
// Plane layout: [limb][row][stride bytes], the K bytes of a row contiguous;
// the left operand has a row per output row, the right one a row per output
// column. Strides of 16 (K = 16) and 80 (K = 64) bytes keep ldmatrix free of
// bank conflicts.
#pragma once
#include <cstdint>
#include <type_traits>

#include "field.cuh"
#include "limb_sums.cuh"

namespace modlin {
namespace mml {

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldm_x4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void ldm_x2(uint32_t& r0, uint32_t& r1, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldm_x1(uint32_t& r0, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x1.shared.b16 {%0}, [%1];" : "=r"(r0) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma_k32(uint32_t (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_k16(uint32_t (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(b0));
}

// Diagonal sums of one warp's 16 x 8 output tile: A's rows 0 .. 15 and B's
// rows (output columns) 0 .. 7 at the given plane addresses. Lane (g, t) =
// (lane / 4, lane % 4) gets rows g, g + 8 and columns 2 t, 2 t + 1: entries
// (g, 2t), (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1).
template <int LIMBS, int KCHUNKS, int STRIDE>
__device__ __forceinline__ void tile_k32(uint32_t (&acc)[2 * LIMBS - 1][4], uint32_t A, uint32_t a_plane, uint32_t B,
                                         uint32_t b_plane) {
  const int lane = threadIdx.x & 31;
  const uint32_t la = A + (lane & 15) * STRIDE + (lane >> 4) * 16;
  const uint32_t lb = B + (lane & 7) * STRIDE + ((lane >> 3) & 1) * 16;
#pragma unroll
  for (int d = 0; d < 2 * LIMBS - 1; ++d)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[d][q] = 0;
#pragma unroll 1
  for (int kc = 0; kc < KCHUNKS; ++kc) {
    // Eight limbs in two halves of the left operand: 16 registers less.
    constexpr int kHalf = LIMBS > 4 ? LIMBS / 2 : LIMBS;
#pragma unroll 1
    for (int h = 0; h < LIMBS; h += kHalf) {
      uint32_t a[kHalf][4];
#pragma unroll
      for (int i = 0; i < kHalf; ++i) ldm_x4(a[i], la + (h + i) * a_plane + kc * 32);
      const auto half = [&](auto off) {
#pragma unroll
        for (int j = 0; j < LIMBS; ++j) {
          uint32_t b0, b1;
          ldm_x2(b0, b1, lb + j * b_plane + kc * 32);
#pragma unroll
          for (int i = 0; i < kHalf; ++i) mma_k32(acc[decltype(off)::value + i + j], a[i], b0, b1);
        }
      };
      if (h == 0)
        half(std::integral_constant<int, 0>{});
      else
        half(std::integral_constant<int, LIMBS - kHalf>{});
    }
  }
}

// The same with K = 16 (16-byte rows).
template <int LIMBS>
__device__ __forceinline__ void tile_k16(uint32_t (&acc)[2 * LIMBS - 1][4], uint32_t A, uint32_t a_plane, uint32_t B,
                                         uint32_t b_plane) {
  const int lane = threadIdx.x & 31;
  const uint32_t la = A + (lane & 15) * 16, lb = B + (lane & 7) * 16;
#pragma unroll
  for (int d = 0; d < 2 * LIMBS - 1; ++d)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[d][q] = 0;
  uint32_t a[LIMBS][2];
#pragma unroll
  for (int i = 0; i < LIMBS; ++i) ldm_x2(a[i][0], a[i][1], la + i * a_plane);
#pragma unroll
  for (int j = 0; j < LIMBS; ++j) {
    uint32_t b0;
    ldm_x1(b0, lb + j * b_plane);
#pragma unroll
    for (int i = 0; i < LIMBS; ++i) mma_k16(acc[i + j], a[i][0], a[i][1], b0);
  }
}

// Bytes i of four residues as one word per limb i.
template <int LIMBS>
__device__ __forceinline__ void limb_words(uint32_t (&w)[LIMBS], const uint64_t (&v)[4]) {
#pragma unroll
  for (int h = 0; h < (LIMBS > 4 ? 2 : 1); ++h) {
    const uint32_t x0 = (uint32_t)(v[0] >> (32 * h)), x1 = (uint32_t)(v[1] >> (32 * h)),
                   x2 = (uint32_t)(v[2] >> (32 * h)), x3 = (uint32_t)(v[3] >> (32 * h));
    const uint32_t p = __byte_perm(x0, x1, 0x5140), q = __byte_perm(x2, x3, 0x5140);
    w[4 * h] = __byte_perm(p, q, 0x5410);
    if constexpr (LIMBS > 1) w[4 * h + 1] = __byte_perm(p, q, 0x7632);
    if constexpr (LIMBS > 2) {
      const uint32_t r = __byte_perm(x0, x1, 0x7362), s = __byte_perm(x2, x3, 0x7362);
      w[4 * h + 2] = __byte_perm(r, s, 0x5410);
      w[4 * h + 3] = __byte_perm(r, s, 0x7632);
    }
  }
}
// The same, word i to dst[i * plane] (4-byte aligned).
template <int LIMBS, class I>
__device__ __forceinline__ void put_planes4(uint8_t* dst, I plane, const uint64_t (&v)[4]) {
  uint32_t w[LIMBS];
  limb_words<LIMBS>(w, v);
#pragma unroll
  for (int i = 0; i < LIMBS; ++i) *reinterpret_cast<uint32_t*>(dst + i * plane) = w[i];
}

// The limbs of one residue as single bytes.
template <int LIMBS, class I>
__device__ __forceinline__ void put_planes1(uint8_t* dst, I plane, uint64_t v) {
#pragma unroll
  for (int i = 0; i < LIMBS; ++i) dst[i * plane] = (uint8_t)(v >> (8 * i));
}

}  // namespace mml
}  // namespace modlin
